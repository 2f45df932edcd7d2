"""GPU kernels at the sizes where a tile, a group or a slice ends, against float64 PyTorch."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nat():
    import flagcx_b200
    return flagcx_b200.native()


@pytest.fixture(scope="module")
def comm1():
    from flagcx_b200.wrapper import FLAGCXLibrary
    lib = FLAGCXLibrary()
    torch.zeros(1, device="cuda")
    comm = lib.flagcxCommInitRank(1, lib.flagcxGetUniqueId(), 0)
    yield comm
    torch.cuda.synchronize()
    lib.flagcxCommDestroy(comm)


def _bf(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).bfloat16()


def _close(got, ref, magnitude, k, roundings=1):
    """One rounding to bf16 (8 significant bits) is at most 2^-8 of a value; fp32 sums of k products may be off by k * 2^-24 of the products' absolute
    sum (twice that covers the tensor cores' own order and truncation)."""
    bound = roundings * 2.0 ** -8 * ref.abs() + k * 2.0 ** -23 * magnitude + 1e-30
    worst = ((got.double() - ref).abs() / bound).max()
    assert worst <= 1.0, float(worst)


@pytest.fixture(scope="module")
def ext(nat):
    lib = ctypes.CDLL(nat.__file__)
    lib.fcxGemmTileCost.restype = ctypes.c_double
    return lib


def _cdiv(a, b):
    return -(-a // b)


def _tiles(ext, m, n, k):
    """(CTA pairs or not, tiles, pieces of K) that a launch of its own uses for an [m, n] product of k terms."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    bn = ctypes.c_int(256)
    ext.fcxGemmTileCost(m, n, k, sms, ctypes.byref(bn))
    pair = bool(ext.fcxGemmPairSuits(m, n, k))
    units = _cdiv(m, 256) * _cdiv(n, 256) if pair else _cdiv(m, 128) * _cdiv(n, bn.value)
    return pair, units, ext.fcxGemmPieces(0, m, n, k, units, sms // 2 if pair else sms, sms)


def _close_in_pieces(got, a, b, pieces, before=None):
    """got = a^T b (+ before) with a [k, m] and b [k, n], K cut into `pieces`.  fp32 sums; every piece p_i is rounded to bf16
    (8 significant bits: unit roundoff 2^-8) and, where there are several or a value before, so is each of the partial
    totals it is added to, in any order: at most 2^-8 (sum |p_i| + pieces (|before| + sum |p_i|)), with the pieces' own
    sums taken in 64 bits."""
    k, per = a.shape[0], _cdiv(_cdiv(a.shape[0], 64), pieces) * 64
    assert _cdiv(k, per) == pieces
    parts = [a[i:i + per].double().t() @ b[i:i + per].double() for i in range(0, k, per)]
    ref, size = sum(parts), sum(p.abs() for p in parts)
    rounding = size
    if before is not None or pieces > 1:
        rounding = size + pieces * (size + (before.abs() if before is not None else 0))
    if before is not None:
        ref = ref + before
    bound = 1.02 * 2.0 ** -8 * rounding + k * 2.0 ** -23 * (a.double().abs().t() @ b.double().abs()) + 1e-30
    worst = float(((got.double() - ref).abs() / bound).max())
    assert worst <= 1.0, worst


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (64, 72, 256), (128, 192, 1024), (129, 1000, 136), (40, 3072, 1024), (384, 1000, 64)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True)])
def test_gemm_with_few_tiles(nat, M, N, K, a_mn, b_mn):
    """Sizes whose tiles would leave most SMs idle at 256 columns: the narrow tiles, in every operand orientation."""
    if (a_mn and M % 8) or N % 8:
        pytest.skip("MN-major operands need multiples of 8")
    torch.manual_seed(M + N + K)
    a, b, bias = _bf(M, K), _bf(N, K), _bf(N)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = nat.gemm(a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b, a_mn, b_mn, bias, 1, err, 0)
    assert int(err.item()) == 0
    ad, bd = a.double(), b.double()
    _close(got, ad @ bd.t() + bias.double(), ad.abs() @ bd.abs().t() + bias.double().abs(), K)


@pytest.mark.parametrize("M,N,K", [
    (1, 8, 128), (127, 72, 1152), (333, 1792, 1024), (129, 136, 2176),  # single CTAs, 64 columns
    (2056, 2176, 640),                                                  # ... or more
    (4104, 4360, 128), (4104, 4360, 640), (4352, 4096, 1152)])          # CTA pairs; K slices that end inside a group
def test_fp8_gemm_tiles(nat, M, N, K):
    torch.manual_seed(M + N)
    aq, sa = nat.quant_fp8_act(_bf(M, K))
    bq, sb = nat.quant_fp8_weight(_bf(N, K, scale=0.02))
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = nat.gemm_fp8_nt(aq, sa, bq, sb, err)
    assert int(err.item()) == 0
    ad = aq.double() * sa.double().t().repeat_interleave(128, 1)
    bd = bq.double() * sb.double().repeat_interleave(128, 0)[:N].repeat_interleave(128, 1)
    _close(got, ad @ bd.t(), ad.abs() @ bd.abs().t(), K)


@pytest.mark.parametrize("M,K,pad", [(1, 128, 0), (7, 384, 0), (333, 4096, 0), (4096, 1024, 0), (4097, 1152, 0), (65, 256, 4)])
def test_fp8_activation_quantisation(nat, M, K, pad):
    """Whole and ragged numbers of blocks, and rows that are only 8-byte aligned (pad 4)."""
    torch.manual_seed(M)
    x = _bf(M, K + pad, scale=3.0)[:, :K]
    x[0, :128] = 0  # a block of zeros has scale 1
    q, s = nat.quant_fp8_act(x)
    blocks = x.float().reshape(M, K // 128, 128)
    amax = blocks.abs().amax(-1)
    want = torch.where(amax > 0, amax / torch.full_like(amax, 448.0), torch.ones_like(amax))
    assert torch.equal(s.t(), want)
    ref = (blocks * (1 / want)[..., None]).clamp(-448, 448).to(torch.float8_e4m3fn)
    assert torch.equal(q.view(torch.uint8), ref.reshape(M, K).view(torch.uint8))


@pytest.mark.parametrize("L,cap,H,F", [(3, 384, 264, 200), (2, 256, 128, 8), (4, 2560, 512, 2056), (1, 128, 64, 128)])
def test_grouped_expert_gemms(nat, comm1, L, cap, H, F):
    """Row counts at and around the edges of the 128-row halves and 256-row tiles, an empty expert among them; F and H
    that end inside a tile; few tiles (128 columns) and many (256)."""
    torch.manual_seed(F)
    counts = ([0, 129, 384] if L == 3 else [1, 256] if L == 2 else [127, 2560, 257, 2049] if L == 4 else [128])
    rows = torch.tensor(counts, dtype=torch.int32, device="cuda")
    x = _bf(L * cap, H)
    w = [_bf(2 * F, H, scale=0.1) for _ in range(L)]
    wd = [_bf(H, F, scale=0.1) for _ in range(L)]
    h = torch.full((L * cap, F), 7.0, device="cuda", dtype=torch.bfloat16)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.moe_up(x, w, h, rows, err)
    # every row goes back to token (its own number), choice 0
    info = torch.zeros(L * cap, 4, dtype=torch.int32, device="cuda")
    info[:, 1] = torch.arange(L * cap, device="cuda")
    back = nat.heap_tensor(comm1.value, [L * cap, H], torch.bfloat16).fill_(5.0)
    done = nat.heap_tensor(comm1.value, [2], torch.int64).zero_()
    grid = nat.moe_down(comm1.value, h, wd, rows, info, back, done, 1, err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and int(done[0].item()) == grid
    for e, n in enumerate(counts):
        xs, hs = x[e * cap:e * cap + n].double(), h[e * cap:e * cap + n]
        gate, up = xs @ w[e][:F].double().t(), xs @ w[e][F:].double().t()
        ref = torch.nn.functional.silu(gate) * up
        # an error d in gate or up moves silu(gate) * up by at most 1.1 d |up| or |silu(gate)| d; __expf adds a few 2^-22
        dg = H * 2.0 ** -23 * (xs.abs() @ w[e].double().abs().t())
        slack = 1.1 * dg[:, :F] * up.abs() + torch.nn.functional.silu(gate).abs() * dg[:, F:] + 2.0 ** -18 * ref.abs()
        assert bool(((hs.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + slack + 1e-30).all()), e
        hd, wdd = hs.double(), wd[e].double()
        if n:
            _close(back[e * cap:e * cap + n], hd @ wdd.t(), hd.abs() @ wdd.abs().t(), F)
        assert bool((back[e * cap + n:(e + 1) * cap] == 5.0).all())  # rows past the count go nowhere
        assert bool((h[e * cap + (n + 31) // 32 * 32:(e + 1) * cap] == 7.0).all())


@pytest.mark.parametrize("entries,experts,H", [((1, 1), 2, 264), ((513, 2), 5, 1024), ((300, 4), 8, 2056), ((130, 3), 4, 128)])
@pytest.mark.parametrize("exchange", [False, True])
def test_dispatch_and_combine_edges(nat, comm1, entries, experts, H, exchange):
    """Token counts that end inside a warp's stretch of the numbering, 1, 2, 3 and 4 choices in the combine, and the dispatch
    both as one rank runs it and with the exchange of counts and arrivals of several ranks, this GPU being its own peer."""
    from flagcx_b200.parallel.ep import ExpertParallelContext, moe_reference
    T, K = entries
    F = 128
    torch.manual_seed(T)
    ep = ExpertParallelContext(comm1.value, 1, 0, T, H, F, K, dispatch_ctas=8, experts_per_rank=experts, capacity_factor=float(experts))
    ep.exchange = exchange
    idx = torch.stack([torch.randperm(experts, device="cuda")[:K] for _ in range(T)]).int().contiguous()
    w = torch.rand(T, K, device="cuda")
    up = [_bf(2 * F, H, scale=0.05) for _ in range(experts)]
    down = [_bf(H, F, scale=0.05) for _ in range(experts)]
    for _ in range(3):
        x = _bf(T, H)
        out = ep.forward(x, idx, w, up, down)
        torch.cuda.synchronize()
        ep.check()
        assert ep.recv_total.tolist() == [int((idx == e).sum().item()) for e in range(experts)]
        ref = moe_reference(x, idx, w, up, down)
        # bf16 roundings of the gate / up products (reference), of h, of y and of the result: four of 2^-9 in quadrature
        assert float((out.float() - ref).norm() / ref.norm()) < 4 * 2.0 ** -9
    # the calls alternate between two buffer sets: epochs 1 and 2 of the first, 1 of the second
    assert [int(f[0].item()) for f in ep.count_flags + ep.disp_done] == ([2, 1, 2, 1] if exchange else [0] * 4)
    if exchange:
        assert ep.count_mat[0].tolist() == [int((idx == e).sum().item()) for e in range(experts)]


@pytest.mark.parametrize("M,C", [(1, 256), (1185, 1024), (1184 * 4 + 3, 768), (9, 512), (1, 1280), (4099, 2048)])
@pytest.mark.parametrize("with_dres", [False, True])
def test_layernorm_backward_in_one_pass(nat, M, C, with_dres):
    """One row, one more row than warps on the GPU, and rows past the ring's depth; rows wider than 1024 take a second pass."""
    torch.manual_seed(M)
    x, dy, g, b = _bf(M, C), _bf(M, C), _bf(C) + 1, _bf(C)
    dres = _bf(M, C) if with_dres else None
    _, _, mean, rstd = nat.layernorm_fwd(x, None, g, b, 1e-5)
    dx, dg, db = nat.layernorm_bwd(dy, x, g, mean, rstd, dres)
    xd, dyd = x.double(), dy.double()
    xh = (xd - mean.double()[:, None]) * rstd.double()[:, None]
    gy = dyd * g.double()
    t = rstd.double()[:, None] * (gy - gy.mean(-1, keepdim=True) - xh * (gy * xh).mean(-1, keepdim=True))
    ref = t + dres.double() if with_dres else t
    mag = rstd.double()[:, None] * (gy.abs() + gy.abs().mean(-1, keepdim=True) + xh.abs() * (gy * xh).abs().mean(-1, keepdim=True))
    _close(dx, ref, mag + ref.abs(), 64)
    _close(dg, (dyd * xh).sum(0), (dyd * xh).abs().sum(0), max(8, M // 8))
    _close(db, dyd.sum(0), dyd.abs().sum(0), max(8, M // 8))
    into_g, into_b = _bf(C), _bf(C)
    before = into_g.clone(), into_b.clone()
    nat.layernorm_bwd(dy, x, g, mean, rstd, dres, into_g, into_b)
    _close(into_g, before[0].double() + (dyd * xh).sum(0), before[0].double().abs() + (dyd * xh).abs().sum(0), max(8, M // 8))
    _close(into_b, before[1].double() + dyd.sum(0), before[1].double().abs() + dyd.abs().sum(0), max(8, M // 8))


@pytest.mark.parametrize("M,C", [(1, 64), (97, 192), (255, 1024), (8200, 256)])
def test_bias_gelu_backward_sums_its_own_gradient(nat, M, C):
    torch.manual_seed(M)
    x, dy, b = _bf(M, C), _bf(M, C), _bf(C)
    dx, db = nat.bias_gelu_bwd(dy, x, b)
    xr = (x.double() + b.double()).requires_grad_()
    torch.nn.functional.gelu(xr, approximate="tanh").backward(dy.double())
    # tanh.approx is good to 2^-11; gelu' takes it once plainly and once in a square times |x| <= 5 or so
    assert float(((dx.double() - xr.grad).abs() - 2.0 ** -8 * xr.grad.abs()).max()) < 5 * 2.0 ** -9 * float(dy.abs().max())
    _close(db, dx.double().sum(0), dx.double().abs().sum(0), max(8, M // 8))
    into = _bf(C)
    before = into.clone()
    nat.bias_gelu_bwd(dy, x, b, into)
    _close(into, before.double() + dx.double().sum(0), before.double().abs() + dx.double().abs().sum(0), max(8, M // 8))


@pytest.mark.parametrize("M,C", [(1, 64), (511, 128), (512, 64), (1025, 192), (2047, 64), (4097, 448), (9000, 3584), (8192, 64), (5, 65600)])
def test_column_sums(nat, M, C):
    """One CTA and clusters of two to eight, rows that divide among them and rows that do not, both CTA sizes, very wide."""
    torch.manual_seed(M)
    a = _bf(M, C)
    _close(nat.col_sum(a), a.double().sum(0), a.double().abs().sum(0), max(8, M // 8))
    into = _bf(C)
    before = into.clone()
    nat.col_sum(a, into)
    _close(into, before.double() + a.double().sum(0), before.double().abs() + a.double().abs().sum(0), max(8, M // 8))


@pytest.mark.parametrize("shape,n_out,bias", [((40, 64), 192, True), ((2, 20, 64), 128, True), ((3, 8, 72), 64, False)])
def test_linear_in_one_call_each_way(nat, shape, n_out, bias):
    """Inputs of two and three dimensions, strided inputs and output gradients, and gradients that are not asked for."""
    from flagcx_b200.ops import linear
    torch.manual_seed(len(shape))
    base = _bf(*shape[:-1], 2 * shape[-1])
    x, w = base[..., :shape[-1]].detach().requires_grad_(), _bf(n_out, shape[-1]).requires_grad_()
    b = _bf(n_out).requires_grad_() if bias else None
    y = linear(x, w, b)
    assert y.shape == (*shape[:-1], n_out)
    dy = _bf(n_out, *shape[:-1]).movedim(0, -1)
    grads = torch.autograd.grad(y, [t for t in (x, w, b) if t is not None], dy, retain_graph=True)
    xd, wd, dyd = x.detach().double(), w.detach().double(), dy.double()
    x2, dy2 = xd.reshape(-1, shape[-1]), dyd.reshape(-1, n_out)
    yd = xd @ wd.t() + (b.detach().double() if bias else 0)
    _close(y.detach(), yd, xd.abs() @ wd.abs().t() + yd.abs(), shape[-1])
    _close(grads[0], dyd @ wd, dyd.abs() @ wd.abs(), n_out)
    _close(grads[1], dy2.t() @ x2, dy2.abs().t() @ x2.abs(), max(8, x2.shape[0]))
    if bias:
        _close(grads[2], dy2.sum(0), dy2.abs().sum(0), max(8, x2.shape[0]))
    only_w, = torch.autograd.grad(y, [w], dy)
    assert torch.equal(only_w, grads[1])


@pytest.mark.parametrize("rows,k,n", [(128, 64, 72), (640, 512, 264), (2048, 1024, 512)])
def test_tensor_parallel_halves_of_one_rank(nat, comm1, ext, rows, k, n):
    from flagcx_b200.parallel.tp import TensorParallelContext, column_parallel_linear, row_parallel_linear
    torch.manual_seed(rows)
    for half in (column_parallel_linear, row_parallel_linear):
        tp = TensorParallelContext(comm1.value, 1, 0, max_rows=rows, max_k=max(k, n), max_n=max(k, n), buffers=4)
        x, w, dy = _bf(rows, k).requires_grad_(), _bf(n, k).requires_grad_(), _bf(rows, n)
        y = half(x, w, tp)
        dx, dw = torch.autograd.grad(y, (x, w), dy)
        torch.cuda.synchronize()
        tp.check()
        xd, wd, dyd = x.detach().double(), w.detach().double(), dy.double()
        _close(y.detach(), xd @ wd.t(), xd.abs() @ wd.abs().t(), k)
        _close(dx, dyd @ wd, dyd.abs() @ wd.abs(), n)
        _close_in_pieces(dw, dy, x.detach(), _tiles(ext, n, k, rows)[2])


@pytest.mark.parametrize("T,I,O", [(8, 64, 64), (136, 264, 520), (128, 256, 1024), (776, 72, 200), (2328, 1000, 2944), (3000, 512, 2048),
                                   (8192, 1024, 1024), (64, 1024, 3072)])
@pytest.mark.parametrize("into", [False, True])
def test_input_and_weight_gradients_in_one_launch(nat, ext, T, I, O, into):
    """Both kernels (single CTAs, CTA pairs), sizes that they leave to two launches, cut and uncut sums over the tokens,
    and a weight gradient that is added to what is there.  The bounds are those of the pieces that the launch is cut into."""
    torch.manual_seed(T + I + O)
    dy, x, w = _bf(T, O), _bf(T, I), _bf(O, I)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    dw_into, db_into = (_bf(O, I), _bf(O)) if into and O % 64 == 0 else (None, None)
    before = [t.double() if t is not None else None for t in (dw_into, db_into)]
    dx, dw, db = nat.linear_bwd(dy, x, w, True, True, O % 64 == 0, err, dw_into, db_into)
    assert int(err.item()) == 0
    assert (dw is None) == (dw_into is not None)
    pair_x, units_x, alone_x = _tiles(ext, T, I, O)
    pair_w, units_w, alone_w = _tiles(ext, O, I, T)
    pieces_x, pieces_w = alone_x, alone_w
    if pair_x == pair_w:
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        cut_w, cut_x, swap, extra = (ctypes.c_int(0) for _ in range(4))
        if ext.fcxGemmDualPlan(units_w, _cdiv(T, 64), alone_w, units_x, _cdiv(O, 64), alone_x, sms // 2 if pair_x else sms,
                               *(ctypes.byref(v) for v in (cut_w, cut_x, swap, extra))):
            pieces_x, pieces_w = cut_x.value, cut_w.value
    _close_in_pieces(dx, dy.t(), w, pieces_x)
    _close_in_pieces(dw if dw is not None else dw_into, dy, x, pieces_w, before[0])
    if O % 64 == 0:
        dyd, b0 = dy.double(), before[1] if before[1] is not None else torch.zeros(O, dtype=torch.float64, device="cuda")
        _close(db if db is not None else db_into, dyd.sum(0) + b0, dyd.abs().sum(0) + b0.abs(), max(8, T // 8))
