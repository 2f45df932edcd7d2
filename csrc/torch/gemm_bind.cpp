// Bindings of the tcgen05 GEMM family (gemm_sm100.cu).
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "flagcx.h"
#include "flagcx_ext.h"
#include "gemm_fp8_sm100.h"
#include "gemm_sm100.h"

namespace fcxt {

FcxDevComm devComm(uint64_t comm);                       // fused_ops.cpp
size_t heapOffset(uint64_t comm, const at::Tensor &t);   // fused_ops.cpp
at::Tensor colSum(const at::Tensor &a, const c10::optional<at::Tensor> &into);  // module.cpp

static void checkMat(const at::Tensor &t, const char *name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.dim() == 2 && t.stride(1) == 1, name, " must be a 2-D bf16 CUDA tensor with contiguous rows");
}

// c[M,N] = a[M,K] @ b[N,K]^T on the tcgen05 path.  err is an int32 device scalar that the kernel sets when a wait gives up.
static at::Tensor gemmNT(const at::Tensor &a, const at::Tensor &b, at::Tensor &err) {
  checkMat(a, "a");
  checkMat(b, "b");
  TORCH_CHECK(a.size(1) == b.size(1), "inner dimensions differ");
  c10::cuda::CUDAGuard g(a.device());
  auto c = at::empty({a.size(0), b.size(0)}, a.options());
  auto e = fcxGemmBf16(a.data_ptr(), b.data_ptr(), c.data_ptr(), (int)a.size(0), (int)b.size(0), (int)a.size(1), (int)a.stride(0),
                       (int)b.stride(0), (int)c.stride(0), err.data_ptr<int>(), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "tcgen05 GEMM launch failed: ", cudaGetErrorString(e));
  return c;
}

// General form on the tcgen05 path.  a_mn / b_mn say how an operand is stored: False = [M,K] / [N,K] (K contiguous),
// True = [K,M] / [K,N] (the operand is read transposed where it lies).  So, for y = x w^T with x [T,I], w [O,I]:
//   forward   y  = gemm(x,  w,  False, False, bias)      [T,O]
//   dgrad     dx = gemm(dy, w,  False, True)              [T,I]   (w is [K=O, N=I])
//   wgrad     dw = gemm(dy, x,  True,  True)              [O,I]   (dy is [K=T, M=O], x is [K=T, N=I])
// split_k = 0 lets the launcher cut K when the output has too few tiles to fill the GPU (wgrad: K = tokens).
static at::Tensor gemmEx(const at::Tensor &a, const at::Tensor &b, bool aMN, bool bMN, const c10::optional<at::Tensor> &bias, int64_t splitK,
                         at::Tensor &err, int64_t pair, const c10::optional<at::Tensor> &out, bool accumulate) {
  checkMat(a, "a");
  checkMat(b, "b");
  const int64_t M = aMN ? a.size(1) : a.size(0), Ka = aMN ? a.size(0) : a.size(1);
  const int64_t N = bMN ? b.size(1) : b.size(0), Kb = bMN ? b.size(0) : b.size(1);
  TORCH_CHECK(Ka == Kb, "inner dimensions differ: ", Ka, " vs ", Kb);
  const void *biasPtr = nullptr;
  if (bias.has_value() && bias->defined()) {
    TORCH_CHECK(bias->is_cuda() && bias->scalar_type() == at::kBFloat16 && bias->is_contiguous() && bias->numel() == N, "bias must be bf16 [N]");
    biasPtr = bias->data_ptr();
  }
  c10::cuda::CUDAGuard g(a.device());
  at::Tensor c;
  if (out.has_value() && out->defined()) {
    c = *out;
    TORCH_CHECK(c.is_cuda() && c.scalar_type() == at::kBFloat16 && c.dim() == 2 && c.size(0) == M && c.size(1) == N && c.stride(1) == 1,
                "out must be a bf16 [M, N] CUDA matrix with contiguous rows");
  } else {
    TORCH_CHECK(!accumulate, "accumulate needs out");
    c = at::empty({M, N}, a.options());
  }
  FcxGemmOpts o{};
  o.aMN = aMN ? 1 : 0; o.bMN = bMN ? 1 : 0; o.bias = biasPtr; o.splitK = (int)splitK; o.accumulate = accumulate ? 1 : 0; o.pair = (int)pair;
  auto e = fcxGemmBf16Opts(a.data_ptr(), b.data_ptr(), c.data_ptr(), (int)M, (int)N, (int)Ka, (int)a.stride(0), (int)b.stride(0),
                           (int)c.stride(0), &o, err.data_ptr<int>(), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "tcgen05 GEMM failed: ", cudaGetErrorString(e), ": ", fcxGemmLastDetail());
  return c;
}

// Forward of a linear layer in one call: (y [..., O], x as a contiguous [T, I] matrix, kept for the backward pass).
static std::tuple<at::Tensor, at::Tensor> linearFwd(const at::Tensor &x, const at::Tensor &w, const c10::optional<at::Tensor> &bias,
                                                    at::Tensor &err) {
  const at::Tensor x2 = (x.dim() == 2 ? x : x.reshape({-1, x.size(-1)})).contiguous();
  at::Tensor y = gemmEx(x2, w, false, false, bias, 0, err, -1, c10::nullopt, false);
  if (x.dim() != 2) {
    auto shape = x.sizes().vec();
    shape.back() = w.size(0);
    y = y.view(shape);
  }
  return {y, x2};
}

// Its backward in one call: dx = dy w, dw = dy^T x, db = column sums of dy, each as asked (undefined otherwise).  With dw_into
// / db_into the weight or bias gradient is added to that tensor (the parameter's .grad) and not returned.
static std::tuple<c10::optional<at::Tensor>, c10::optional<at::Tensor>, c10::optional<at::Tensor>> linearBwd(
    const at::Tensor &dy, const at::Tensor &x2, const at::Tensor &w, bool needX, bool needW, bool needB, at::Tensor &err,
    const c10::optional<at::Tensor> &dwInto, const c10::optional<at::Tensor> &dbInto) {
  const at::Tensor dy2 = (dy.dim() == 2 ? dy : dy.reshape({-1, dy.size(-1)})).contiguous();
  c10::optional<at::Tensor> dx, dw, db;
  const bool intoW = dwInto.has_value() && dwInto->defined(), intoB = dbInto.has_value() && dbInto->defined();
  bool done = false;
  if (needX && needW) {
    checkMat(dy2, "dy");
    checkMat(x2, "x");
    checkMat(w, "w");
    const int64_t T = dy2.size(0), O = dy2.size(1), I = w.size(1);
    TORCH_CHECK(w.size(0) == O && x2.size(0) == T && x2.size(1) == I, "dy, x and w disagree on a dimension");
    TORCH_CHECK(!intoW || (dwInto->is_cuda() && dwInto->scalar_type() == at::kBFloat16 && dwInto->is_contiguous() && dwInto->dim() == 2 &&
                           dwInto->size(0) == O && dwInto->size(1) == I),
                "dw_into must be a contiguous bf16 [O, I] CUDA matrix");
    c10::cuda::CUDAGuard g(dy2.device());
    at::Tensor outX = at::empty({T, I}, dy2.options()), outW = intoW ? *dwInto : at::empty({O, I}, dy2.options());
    auto e = fcxGemmBackwardBf16(dy2.data_ptr(), w.data_ptr(), x2.data_ptr(), outX.data_ptr(), outW.data_ptr(), (int)T, (int)I, (int)O,
                                 (int)dy2.stride(0), (int)w.stride(0), (int)x2.stride(0), intoW ? 1 : 0, err.data_ptr<int>(),
                                 at::cuda::getCurrentCUDAStream().stream());
    done = e == cudaSuccess;
    TORCH_CHECK(done || e == cudaErrorNotSupported, "tcgen05 GEMM launch failed: ", cudaGetErrorString(e));
    if (done) {
      dx = outX;
      if (!intoW) dw = outW;
    }
  }
  if (!done && needX) dx = gemmEx(dy2, w, false, true, c10::nullopt, 0, err, -1, c10::nullopt, false);
  if (!done && needW) {
    at::Tensor r = gemmEx(dy2, x2, true, true, c10::nullopt, 0, err, -1, dwInto, intoW);
    if (!intoW) dw = r;
  }
  if (needB) {
    at::Tensor r = colSum(dy2, dbInto);
    if (!intoB) db = r;
  }
  return {dx, dw, db};
}

// The linear layer as an autograd function of its own: forward and backward stay in native code, so that on small layers
// the interpreter is not what their time goes into.
class LinearFunction : public torch::autograd::Function<LinearFunction> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext *ctx, const at::Tensor &x, const at::Tensor &w, const c10::optional<at::Tensor> &bias,
                            at::Tensor err) {
    auto [y, x2] = linearFwd(x, w, bias, err);
    ctx->save_for_backward({x2, w});
    ctx->saved_data["err"] = err;
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["bias"] = bias.has_value() && bias->defined();
    return y;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext *ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    at::Tensor err = ctx->saved_data["err"].toTensor();
    const auto shape = ctx->saved_data["shape"].toIntVector();
    const bool bias = ctx->saved_data["bias"].toBool();
    auto [dx, dw, db] = linearBwd(grads[0], saved[0], saved[1], ctx->needs_input_grad(0), ctx->needs_input_grad(1),
                                  bias && ctx->needs_input_grad(2), err, c10::nullopt, c10::nullopt);
    if (dx.has_value() && shape.size() != 2) dx = dx->view(shape);
    return {dx.value_or(at::Tensor()), dw.value_or(at::Tensor()), db.value_or(at::Tensor()), at::Tensor()};
  }
};

static at::Tensor linearApply(const at::Tensor &x, const at::Tensor &w, const c10::optional<at::Tensor> &bias, const at::Tensor &err) {
  return LinearFunction::apply(x, w, bias, err);
}

// (pre, act) = (a w^T, gelu_tanh(a w^T + bias)) in one kernel: the CTA-pair GEMM writes both from its epilogue.  pre is what
// the backward pass of bias + GELU needs; a [M,K], w [N,K], bias [N] or None.
static std::tuple<at::Tensor, at::Tensor> gemmBiasGelu(const at::Tensor &a, const at::Tensor &w, const c10::optional<at::Tensor> &bias,
                                                       at::Tensor &err) {
  checkMat(a, "a");
  checkMat(w, "w");
  const int64_t M = a.size(0), K = a.size(1), N = w.size(0);
  TORCH_CHECK(w.size(1) == K, "inner dimensions differ: ", K, " vs ", w.size(1));
  const void *biasPtr = nullptr;
  if (bias.has_value() && bias->defined()) {
    TORCH_CHECK(bias->is_cuda() && bias->scalar_type() == at::kBFloat16 && bias->is_contiguous() && bias->numel() == N, "bias must be bf16 [N]");
    biasPtr = bias->data_ptr();
  }
  c10::cuda::CUDAGuard g(a.device());
  auto pre = at::empty({M, N}, a.options()), act = at::empty({M, N}, a.options());
  FcxGemmOpts o{};
  o.bias = biasPtr; o.splitK = 1; o.pair = 1; o.geluOut = act.data_ptr();
  auto e = fcxGemmBf16Opts(a.data_ptr(), w.data_ptr(), pre.data_ptr(), (int)M, (int)N, (int)K, (int)a.stride(0), (int)w.stride(0),
                           (int)pre.stride(0), &o, err.data_ptr<int>(), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "tcgen05 GEMM + GELU failed: ", cudaGetErrorString(e), ": ", fcxGemmLastDetail());
  return {pre, act};
}

// y[M,N] = all_gather(x_local)[M,K] @ w[N,K]^T.  gathered: heap tensor [M,K]; flags: heap int64 tensor [M/128];
// epoch: 1-based use count of this (gathered, flags) pair.
static at::Tensor agGemm(uint64_t comm, const at::Tensor &xLocal, at::Tensor &gathered, at::Tensor &flags, const at::Tensor &w,
                         int64_t epoch, int64_t commCtas, at::Tensor &err, bool exchange) {
  checkMat(xLocal, "x_local");
  checkMat(w, "w");
  TORCH_CHECK(xLocal.is_contiguous() && gathered.is_contiguous(), "x_local and gathered must be contiguous");
  c10::cuda::CUDAGuard g(xLocal.device());
  FcxDevComm dc = devComm(comm);
  const int M = (int)xLocal.size(0) * dc.nranks, K = (int)xLocal.size(1), N = (int)w.size(0);
  TORCH_CHECK(gathered.numel() >= (int64_t)M * K && flags.numel() >= M / 128, "workspace too small");
  auto y = at::empty({M, N}, xLocal.options());
  auto e = fcxAgGemmBf16(&dc, xLocal.data_ptr(), gathered.data_ptr(), heapOffset(comm, gathered), heapOffset(comm, flags), w.data_ptr(),
                         y.data_ptr(), M, N, K, (int)w.stride(0), (int)y.stride(0), (uint64_t)epoch, (int)commCtas, exchange, err.data_ptr<int>(),
                         at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "fused all-gather GEMM launch failed: ", cudaGetErrorString(e));
  return y;
}

// out[M/n,N] = reduce_scatter(a[M,K] @ w[N,K]^T).  stage: heap bf16 tensor [n, M/n, N]; counters: heap int64 tensor
// [M/n/128 * ceil(N/256)]; epoch: 1-based use count of this (stage, counters) pair.
static at::Tensor gemmRs(uint64_t comm, const at::Tensor &a, const at::Tensor &w, at::Tensor &stage, at::Tensor &counters, int64_t epoch,
                         at::Tensor &err, bool exchange) {
  checkMat(a, "a");
  checkMat(w, "w");
  c10::cuda::CUDAGuard g(a.device());
  FcxDevComm dc = devComm(comm);
  const int M = (int)a.size(0), K = (int)a.size(1), N = (int)w.size(0);
  TORCH_CHECK(M % (dc.nranks * 128) == 0, "rows must be a multiple of 128 x ranks");
  TORCH_CHECK(stage.numel() >= (int64_t)M * N && counters.numel() >= (M / dc.nranks / 128) * ((N + 255) / 256), "workspace too small");
  auto out = at::empty({M / dc.nranks, N}, a.options());
  auto e = fcxGemmRsBf16(&dc, a.data_ptr(), w.data_ptr(), out.data_ptr(), heapOffset(comm, stage), heapOffset(comm, counters), M, N, K,
                         (int)a.stride(0), (int)w.stride(0), (int)out.stride(0), (uint64_t)epoch, exchange, err.data_ptr<int>(),
                         at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "fused GEMM reduce-scatter launch failed: ", cudaGetErrorString(e));
  return out;
}

// bf16 [M,K] -> (e4m3 [M,K], fp32 scales [K/128, M])
static std::tuple<at::Tensor, at::Tensor> quantFp8Act(const at::Tensor &x) {
  checkMat(x, "x");
  TORCH_CHECK(x.size(1) % 128 == 0, "K must be a multiple of 128");
  c10::cuda::CUDAGuard g(x.device());
  auto q = at::empty({x.size(0), x.size(1)}, x.options().dtype(at::kFloat8_e4m3fn));
  auto sa = at::empty({x.size(1) / 128, x.size(0)}, x.options().dtype(at::kFloat));
  auto e = fcxQuantFp8Act(x.data_ptr(), q.data_ptr(), sa.data_ptr<float>(), (int)x.size(0), (int)x.size(1), (int)x.stride(0),
                          at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "fp8 quantisation launch failed: ", cudaGetErrorString(e));
  return {q, sa};
}

// bf16 [N,K] -> (e4m3 [N,K], fp32 scales [ceil(N/128), K/128])
static std::tuple<at::Tensor, at::Tensor> quantFp8Weight(const at::Tensor &w) {
  checkMat(w, "w");
  TORCH_CHECK(w.size(1) % 128 == 0, "K must be a multiple of 128");
  c10::cuda::CUDAGuard g(w.device());
  auto q = at::empty({w.size(0), w.size(1)}, w.options().dtype(at::kFloat8_e4m3fn));
  auto sb = at::empty({(w.size(0) + 127) / 128, w.size(1) / 128}, w.options().dtype(at::kFloat));
  auto e = fcxQuantFp8Weight(w.data_ptr(), q.data_ptr(), sb.data_ptr<float>(), (int)w.size(0), (int)w.size(1), (int)w.stride(0),
                             at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "fp8 quantisation launch failed: ", cudaGetErrorString(e));
  return {q, sb};
}

// bf16 c[M,N] = dequant(aq, sa) @ dequant(bq, sb)^T with the scales applied per 128-deep slice of K on the tcgen05 path
static at::Tensor gemmFp8NT(const at::Tensor &aq, const at::Tensor &sa, const at::Tensor &bq, const at::Tensor &sb, at::Tensor &err) {
  TORCH_CHECK(aq.is_cuda() && aq.scalar_type() == at::kFloat8_e4m3fn && aq.is_contiguous() && bq.scalar_type() == at::kFloat8_e4m3fn &&
                  bq.is_contiguous() && aq.dim() == 2 && bq.dim() == 2 && aq.size(1) == bq.size(1),
              "aq [M,K] and bq [N,K] must be contiguous e4m3 matrices");
  const int M = (int)aq.size(0), N = (int)bq.size(0), K = (int)aq.size(1);
  TORCH_CHECK(sa.scalar_type() == at::kFloat && sa.is_contiguous() && sa.numel() == (int64_t)(K / 128) * M, "sa must be fp32 [K/128, M]");
  TORCH_CHECK(sb.scalar_type() == at::kFloat && sb.is_contiguous() && sb.numel() == (int64_t)((N + 127) / 128) * (K / 128),
              "sb must be fp32 [ceil(N/128), K/128]");
  c10::cuda::CUDAGuard g(aq.device());
  auto c = at::empty({M, N}, aq.options().dtype(at::kBFloat16));
  auto e = fcxGemmFp8Blockwise(aq.data_ptr(), sa.data_ptr<float>(), bq.data_ptr(), sb.data_ptr<float>(), c.data_ptr(), M, N, K, (int)c.stride(0),
                               err.data_ptr<int>(), at::cuda::getCurrentCUDAStream().stream());
  TORCH_CHECK(e == cudaSuccess, "fp8 GEMM launch failed: ", cudaGetErrorString(e));
  return c;
}

void bindGemm(py::module &m) {
  m.def("quant_fp8_act", &quantFp8Act);
  m.def("quant_fp8_weight", &quantFp8Weight);
  m.def("gemm_fp8_nt", &gemmFp8NT, "block-scaled e4m3 GEMM (1x128 activation scales, 128x128 weight scales) on tcgen05");
  m.def("gemm_nt", &gemmNT, "bf16 a[M,K] @ b[N,K]^T on tcgen05");
  m.def("gemm", &gemmEx, py::arg("a"), py::arg("b"), py::arg("a_mn") = false, py::arg("b_mn") = false, py::arg("bias") = py::none(),
        py::arg("split_k") = 0, py::arg("err"), py::arg("pair") = -1, py::arg("out") = py::none(), py::arg("accumulate") = false,
        "out: write the result there; accumulate: add it to what out holds (a gradient that collects contributions). "
        "bf16 GEMM on tcgen05 with either operand read K-major or MN-major, optional bias row; pair: -1 kernel chosen by shape, "
        "0 one-CTA kernel (128 x 256 tiles), 1 CTA-pair kernel (cta_group::2, 256 x 256 tiles)");
  m.def("linear", &linearApply, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("err"), "differentiable x w^T + bias on tcgen05");
  m.def("linear_fwd", &linearFwd, py::arg("x"), py::arg("w"), py::arg("bias"), py::arg("err"));
  m.def("linear_bwd", &linearBwd, py::arg("dy"), py::arg("x2"), py::arg("w"), py::arg("need_x"), py::arg("need_w"), py::arg("need_b"),
        py::arg("err"), py::arg("dw_into") = py::none(), py::arg("db_into") = py::none());
  m.def("gemm_bias_gelu", &gemmBiasGelu, py::arg("a"), py::arg("w"), py::arg("bias"), py::arg("err"),
        "(a w^T, gelu_tanh(a w^T + bias)) from one CTA-pair GEMM launch");
  m.def("ag_gemm", &agGemm, py::arg("comm"), py::arg("x_local"), py::arg("gathered"), py::arg("flags"), py::arg("w"), py::arg("epoch"),
        py::arg("comm_ctas"), py::arg("err"), py::arg("exchange") = false,
        "exchange: take the exchanging kernel on a communicator of one rank too (it gets the plain GEMM otherwise)");
  m.def("gemm_rs", &gemmRs, py::arg("comm"), py::arg("a"), py::arg("w"), py::arg("stage"), py::arg("counters"), py::arg("epoch"), py::arg("err"),
        py::arg("exchange") = false);
}

}  // namespace fcxt
