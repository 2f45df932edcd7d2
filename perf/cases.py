"""The workloads this framework is timed on, through its public entry points, on one GPU.

Five kinds of work, each at the sizes its users run, the smallest included:

* ``train``   one optimisation step of the data-parallel engine on the GPT-2 decoder (forward, backward, AdamW, replayed
              as a CUDA graph): ``DataParallelTrainer.step``.
* ``linear``  a differentiable projection, forward and backward: ``flagcx_b200.ops.linear``.
* ``tp``      the two halves of a tensor-parallel block, forward and backward: ``column_parallel_linear`` (all-gather ->
              GEMM) and ``row_parallel_linear`` (GEMM -> reduce-scatter) on a one-rank communicator, with the shard
              shapes of eight ranks.
* ``fp8``     a block-scaled fp8 projection: activation quantisation and the e4m3 GEMM (weights quantised once).
* ``moe``     a mixture-of-experts layer, dispatch -> expert MLPs -> combine: ``ExpertParallelContext.forward``.
* ``coll``    a collective of n ranks.  One GPU holds all of them (``flagcxEmuCollective``: the kernels that run across
              GPUs, as one launch), with the kernel kind that the tuner picks for such a size: the low-latency form up to
              32 KiB, the zero-copy form above.
"""
import ctypes
import math
import os

import torch

# Every communicator of this process: room in the symmetric heap for the workspaces of several layers at once.
os.environ.setdefault("FLAGCX_HEAP_USER_BYTES", "8G")
os.environ.setdefault("FLAGCX_STAGE_BYTES", "64M")
os.environ.setdefault("FLAGCX_SOCKET_IFNAME", "lo")

import flagcx_b200  # noqa: E402
from flagcx_b200.models.gpt2 import GPT2, GPT2Config  # noqa: E402
from flagcx_b200.ops import linear  # noqa: E402
from flagcx_b200.parallel.ddp import DataParallelTrainer  # noqa: E402
from flagcx_b200.parallel.ep import ExpertParallelContext  # noqa: E402
from flagcx_b200.parallel.tp import TensorParallelContext, column_parallel_linear, row_parallel_linear  # noqa: E402
from flagcx_b200.wrapper import FLAGCXLibrary  # noqa: E402

LL_BYTES = 32 << 10  # largest message of the low-latency collective kernels
OPS = {"allreduce": 6, "allgather": 7, "reducescatter": 8, "alltoall": 9}  # flagcxCommOp_t
DTYPES = {"fp32": (torch.float32, 7), "bf16": (torch.bfloat16, 9)}         # and flagcxDataType_t


def listed():
    return [
        # the smallest model, a step of a few hundred launches of a few microseconds each: launch and latency bound
        {"name": "train_tiny", "kind": "train", "model": "tiny", "batch": 2, "seq": 64},
        # the headline benchmark: GPT-2-medium, micro-batch 8 x 1024
        {"name": "train_medium", "kind": "train", "model": "medium", "batch": 8, "seq": 1024},
        # the same model on a short last batch of ragged length
        {"name": "train_medium_ragged", "kind": "train", "model": "medium", "batch": 3, "seq": 776},
        # a projection on few tokens (the start of a sequence-length warm-up, a small micro-batch)
        {"name": "linear_small", "kind": "linear", "tokens": 64, "n_in": 1024, "n_out": 3072},
        # sizes that fill no tile: ragged tokens, widths that are no power of two
        {"name": "linear_ragged", "kind": "linear", "tokens": 2328, "n_in": 1000, "n_out": 2944},
        # Llama-3-8B feed-forward block on one of eight ranks (up + gate 2 x 1792, down 1792), 8192 tokens
        {"name": "tp_ffn", "kind": "tp", "tokens": 8192, "hidden": 4096, "col_out": 3584, "row_in": 1792},
        # block-scaled fp8: a full square projection, and a short ragged batch through a sharded one
        {"name": "fp8_large", "kind": "fp8", "tokens": 8192, "n_in": 4096, "n_out": 4096},
        {"name": "fp8_small", "kind": "fp8", "tokens": 333, "n_in": 4096, "n_out": 1792},
        # mixture of experts: a small layer on a short batch, and the Mixtral shape with all eight experts on this rank
        {"name": "moe_small", "kind": "moe", "tokens": 512, "hidden": 1024, "ffn": 2048, "experts": 4},
        {"name": "moe_mixtral", "kind": "moe", "tokens": 8192, "hidden": 4096, "ffn": 14336, "experts": 8},
        # a scalar-sized all-reduce (loss averages, norms) and a 25 MB gradient bucket, eight ranks
        {"name": "allreduce_4k", "kind": "coll", "op": "allreduce", "ranks": 8, "dtype": "fp32", "count": 1024},
        {"name": "allreduce_bucket", "kind": "coll", "op": "allreduce", "ranks": 8, "dtype": "bf16", "count": 13107200},
    ]


def _log(rng, lo, hi, multiple=1):
    """A size between lo and hi, even over its logarithm, rounded to a multiple."""
    return max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) // multiple * multiple)


def draw(rng):
    kind = rng.choice(["train", "linear", "linear", "tp", "fp8", "fp8", "moe", "moe", "coll", "coll"])
    if kind == "train":
        if rng.random() < 0.5:
            return {"kind": kind, "model": "tiny", "batch": _log(rng, 1, 64), "seq": rng.randrange(8, 65, 8)}
        return {"kind": kind, "model": "medium", "batch": rng.randint(1, 8), "seq": rng.randrange(64, 1025, 8)}
    if kind == "linear":
        return {"kind": kind, "tokens": _log(rng, 16, 8192, 8), "n_in": _log(rng, 512, 4096, 8), "n_out": _log(rng, 512, 4096, 64)}
    if kind == "tp":
        return {"kind": kind, "tokens": _log(rng, 256, 8192, 128), "hidden": _log(rng, 1024, 4096, 128), "col_out": _log(rng, 512, 3584, 128),
                "row_in": _log(rng, 512, 1792, 128)}
    if kind == "fp8":
        return {"kind": kind, "tokens": _log(rng, 16, 8192), "n_in": _log(rng, 512, 4096, 128), "n_out": _log(rng, 512, 4096, 8)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log(rng, 128, 4096), "hidden": _log(rng, 512, 4096, 256), "ffn": _log(rng, 1024, 7168, 128),
                "experts": rng.choice([2, 4, 8])}
    op, ranks, dtype = rng.choice(sorted(OPS)), rng.choice([2, 4, 8]), rng.choice(sorted(DTYPES))
    # an all-gather or all-to-all writes `ranks` times what a rank contributes: the same total as the largest all-reduce
    most = (25 << 20) // (4 if dtype == "fp32" else 2) // (1 if op == "allreduce" else ranks)
    return {"kind": "coll", "op": op, "ranks": ranks, "dtype": dtype, "count": _log(rng, 64, most)}


# ---------------------------------------------------------------------------------------------------------------------
# what a program has in hand before the call

_comm = None


def _communicator():
    """The process's one-rank communicator, made once as any program does."""
    global _comm
    if _comm is None:
        lib = FLAGCXLibrary()
        torch.zeros(1, device="cuda")
        _comm = (lib, lib.flagcxCommInitRank(1, lib.flagcxGetUniqueId(), 0))
    return _comm[1].value


def _randn(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()


class _Collective:
    """An n-rank group on this GPU and the ctypes arguments of one call."""

    def __init__(self, case, g):
        self.lib = FLAGCXLibrary()
        n, count = case["ranks"], case["count"]
        dtype, code = DTYPES[case["dtype"]]
        op = case["op"]
        send_n = count * (n if op in ("reducescatter", "alltoall") else 1)
        recv_n = count * (n if op in ("allgather", "alltoall") else 1)
        small = count * dtype.itemsize <= LL_BYTES
        prefix = {"allreduce": "ar", "reducescatter": "rs"}.get(op, "move")
        self.send = [(torch.rand(send_n, generator=g, device="cuda") * 2 - 1).to(dtype) for _ in range(n)]
        self.recv = [torch.empty(recv_n, dtype=dtype, device="cuda") for _ in range(n)]
        self.handle = ctypes.c_void_p()
        self.lib.call("flagcxEmuCreate", ctypes.byref(self.handle), n, 1 << 20)
        ptrs = ctypes.c_void_p * n
        kind, ctas = (prefix + "_ll", 1) if small else (prefix + "_zc", 16)
        self.args = (OPS[op], kind.encode(), ctas, ptrs(*[t.data_ptr() for t in self.send]), ptrs(*[t.data_ptr() for t in self.recv]),
                     count, code, code, ctypes.c_float(1.0), 0, 0, None)

    def __call__(self):
        self.lib.call("flagcxEmuCollective", self.handle, *self.args, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return self.recv

    def __del__(self):
        self.lib.call("flagcxEmuDestroy", self.handle)


class _Training:
    """A trainer that goes when the program drops it: its parameters' gradient hooks refer back to it, a cycle through
    autograd that the garbage collector does not see, and it holds several GB."""

    def __init__(self, model):
        torch.cuda.empty_cache()  # what an earlier trainer's graph and side streams have left in the allocator
        self.trainer = DataParallelTrainer(model)

    def __del__(self):
        for p in self.trainer.model.parameters():
            if p._post_accumulate_grad_hooks is not None:
                p._post_accumulate_grad_hooks.clear()
            p.grad = None
            p.data = p.data.new_empty(0)
        self.trainer.__dict__.clear()


def prepare(case, seed):
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    s = {"kind": kind}
    if kind == "train":
        torch.manual_seed(seed)
        cfg = GPT2Config.medium() if case["model"] == "medium" else GPT2Config.tiny()
        with torch.device("cuda"):
            model = GPT2(cfg)
        s["training"] = _Training(model)
        s["tokens"], s["targets"] = (torch.randint(0, cfg.vocab, (case["batch"], case["seq"]), generator=g, device="cuda") for _ in range(2))
        for _ in range(3):  # a loop in its steady state: the third step has captured the graph
            s["training"].trainer.step(s["tokens"], s["targets"])
    elif kind == "linear":
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        s["x"], s["dy"] = _randn(g, t, i), _randn(g, t, o)
        s["w"], s["bias"] = _randn(g, o, i, std=0.02), _randn(g, o, std=0.02)
        for k in ("x", "w", "bias"):
            s[k].requires_grad_(True)
    elif kind == "tp":
        t, h, c, r = case["tokens"], case["hidden"], case["col_out"], case["row_in"]
        s["tp"] = TensorParallelContext(_communicator(), 1, 0, max_rows=t, max_k=h, max_n=h, buffers=4)
        s["x"], s["dy"], s["w_col"] = _randn(g, t, h), _randn(g, t, c), _randn(g, c, h, std=0.02)
        s["a"], s["dz"], s["w_row"] = _randn(g, t, r), _randn(g, t, h), _randn(g, h, r, std=0.02)
        for k in ("x", "w_col", "a", "w_row"):
            s[k].requires_grad_(True)
    elif kind == "fp8":
        s["native"] = flagcx_b200.native()
        s["x"] = _randn(g, case["tokens"], case["n_in"])
        s["w"], s["scale"] = s["native"].quant_fp8_weight(_randn(g, case["n_out"], case["n_in"], std=0.02))
        s["err"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif kind == "moe":
        t, h, f, e = case["tokens"], case["hidden"], case["ffn"], case["experts"]
        # room for twice the balanced load: with few tokens the router's draw is uneven
        s["ep"] = ExpertParallelContext(_communicator(), 1, 0, t, h, f, 2, capacity_factor=2.0 if t < 4096 else 1.25, experts_per_rank=e)
        s["x"] = _randn(g, t, h)
        w, idx = torch.topk(torch.softmax(torch.randn(t, e, generator=g, device="cuda"), -1), 2, dim=-1)
        s["idx"], s["weights"] = idx.int().contiguous(), w.float().contiguous()
        s["up"] = [_randn(g, 2 * f, h, std=0.02) for _ in range(e)]
        s["down"] = [_randn(g, h, f, std=0.02) for _ in range(e)]
    elif kind == "coll":
        s["call"] = _Collective(case, g)
    else:
        raise ValueError(kind)
    return s


# ---------------------------------------------------------------------------------------------------------------------
# one pass

def run(s):
    kind = s["kind"]
    if kind == "train":
        trainer = s["training"].trainer
        loss = trainer.step(s["tokens"], s["targets"])
        return {"loss": loss, "master": trainer.master}
    if kind == "linear":
        y = linear(s["x"], s["w"], s["bias"])
        dx, dw, db = torch.autograd.grad(y, (s["x"], s["w"], s["bias"]), s["dy"])
        return {"y": y, "dx": dx, "dw": dw, "dbias": db}
    if kind == "tp":
        y = column_parallel_linear(s["x"], s["w_col"], s["tp"])
        z = row_parallel_linear(s["a"], s["w_row"], s["tp"])
        da, dw_row = torch.autograd.grad(z, (s["a"], s["w_row"]), s["dz"])
        dx, dw_col = torch.autograd.grad(y, (s["x"], s["w_col"]), s["dy"])
        return {"y": y, "z": z, "dx": dx, "dw_col": dw_col, "da": da, "dw_row": dw_row}
    if kind == "fp8":
        q, scale = s["native"].quant_fp8_act(s["x"])
        return s["native"].gemm_fp8_nt(q, scale, s["w"], s["scale"], s["err"])
    if kind == "moe":
        return s["ep"].forward(s["x"], s["idx"], s["weights"], s["up"], s["down"])
    return s["call"]()


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    kind = case["kind"]
    if kind == "train":
        cfg = GPT2Config.medium() if case["model"] == "medium" else GPT2Config.tiny()
        rows, c, f, layers, seq = case["batch"] * case["seq"], cfg.d_model, cfg.d_ff, cfg.n_layer, case["seq"]
        mats = layers * (4 * c * c + 2 * c * f) + cfg.vocab * c
        params = mats + cfg.seq_len * c + layers * (9 * c + f + 4 * c) + 2 * c
        attention = layers * case["batch"] * 3.5 * 2 * seq * seq * c  # causal: half the square, two products forward, five backward
        # fp32 master weights and both moments read and written, the bf16 weights written; everything between may stay on chip
        return {"bytes": params * (6 * 4 + 2) + 2 * rows * 8, "flops": 6.0 * rows * mats + attention}
    if kind == "linear":
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        return {"bytes": 2 * (2 * t * i + 2 * o * i + 2 * t * o + 2 * o), "flops": 6.0 * t * i * o}
    if kind == "tp":
        t, h, c, r = case["tokens"], case["hidden"], case["col_out"], case["row_in"]
        return {"bytes": 2 * 2 * (t * h + h * c + t * c + t * r + h * r + t * h), "flops": 6.0 * t * h * (c + r)}
    if kind == "fp8":
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        return {"bytes": 2 * t * i + o * i + 4 * (o // 128 + 1) * (i // 128) + 2 * t * o, "flops": 2.0 * t * i * o}
    if kind == "moe":
        t, h, f, e = case["tokens"], case["hidden"], case["ffn"], case["experts"]
        return {"bytes": 2 * (2 * t * h + 3 * e * h * f) + 16 * t, "flops": 2.0 * 2 * t * 3 * h * f}
    size = 4 if case["dtype"] == "fp32" else 2
    n, count, op = case["ranks"], case["count"], case["op"]
    values = n * count * ((n if op in ("reducescatter", "alltoall") else 1) + (n if op in ("allgather", "alltoall") else 1))
    adds = n * count * (n - 1) if op == "reducescatter" else count * (n - 1) if op == "allreduce" else 0
    return {"bytes": values * size, "flops": float(adds)}


def tolerance(case):
    """About four times what one pass differs from the same sums in 64 bits (train: from a second run of the same
    steps, whose split reductions add in another order; AdamW's first steps turn such noise in small gradients into
    whole learning-rate steps)."""
    kind = case["kind"]
    if kind == "coll":
        if case["op"] in ("allgather", "alltoall"):
            return "exact"
        return {"rel": 5e-7, "max": 2e-6} if case["dtype"] == "fp32" else {"rel": 7e-3, "max": 1.6e-2}
    return {"train": {"rel": 1e-2, "max": 0.4},       # seen: 0.0029 and 0.11
            "linear": {"rel": 1e-2, "max": 9e-2},     # seen: 0.0036 and 0.022 (split-K pieces added in bf16)
            "tp": {"rel": 7e-3, "max": 1.6e-2},       # seen: 0.0017 and 0.0039: one rounding to bf16
            "fp8": {"rel": 7e-3, "max": 1.6e-2},      # seen: the same, on the quantised operands
            "moe": {"rel": 1.5e-2, "max": 0.11}}[kind]  # seen: 0.0039 and 0.027 (bf16 between the products)


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits, from plain torch

def _fp8(x):
    return x.float().clamp(-448, 448).to(torch.float8_e4m3fn).double()


def _train_loss(case, seed):
    """The loss that the pass after `prepare` returns: four steps on the same batch, the first three of which update the
    fp32 master weights (AdamW) and with them the bf16 working weights."""
    cfg = GPT2Config.tiny()
    g = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = GPT2(cfg)  # for its random initial weights only
    tokens, targets = (torch.randint(0, cfg.vocab, (case["batch"], case["seq"]), generator=g, device="cuda") for _ in range(2))
    fn = torch.nn.functional
    work = {k: p.detach().bfloat16().double().requires_grad_(True) for k, p in model.named_parameters()}
    master = {k: p.detach().clone() for k, p in work.items()}
    m, v = ({k: torch.zeros_like(p) for k, p in master.items()} for _ in range(2))
    c, heads = cfg.d_model, cfg.n_head

    def forward(tok, tgt):
        n, t = tok.shape
        x = work["wte"][tok] + work["wpe"][:t]
        mask = torch.ones(t, t, dtype=torch.bool, device="cuda").triu(1)
        for i in range(cfg.n_layer):
            w = {k.split(".", 2)[2]: p for k, p in work.items() if k.startswith("blocks.%d." % i)}
            h = fn.layer_norm(x, (c,), w["ln1_w"], w["ln1_b"])
            q, k, val = (h @ w["qkv_w"].t() + w["qkv_b"]).view(n, t, 3, heads, c // heads).permute(2, 0, 3, 1, 4)
            att = torch.softmax((q @ k.transpose(-1, -2) / math.sqrt(c // heads)).masked_fill(mask, -math.inf), -1) @ val
            x = x + att.transpose(1, 2).reshape(n, t, c) @ w["proj_w"].t() + w["proj_b"]
            h = fn.layer_norm(x, (c,), w["ln2_w"], w["ln2_b"])
            x = x + fn.gelu(h @ w["fc_w"].t() + w["fc_b"], approximate="tanh") @ w["out_w"].t() + w["out_b"]
        logits = fn.layer_norm(x, (c,), work["lnf_w"], work["lnf_b"]) @ work["wte"][:cfg.vocab].t()
        return fn.cross_entropy(logits.view(-1, cfg.vocab), tgt.reshape(-1))

    for step in range(1, 5):
        total = 0.0
        for b in range(case["batch"]):  # one sequence at a time: the activations of a batch in 64 bits are large
            loss = forward(tokens[b:b + 1], targets[b:b + 1]) / case["batch"]
            if step < 4:
                loss.backward()
            total = total + loss.detach()
        if step == 4:
            return total
        with torch.no_grad():
            for k, p in work.items():
                m[k] = 0.9 * m[k] + 0.1 * p.grad
                v[k] = 0.95 * v[k] + 0.05 * p.grad ** 2
                master[k] -= 3e-4 * ((m[k] / (1 - 0.9 ** step)) / ((v[k] / (1 - 0.95 ** step)).sqrt() + 1e-8) + 0.1 * master[k])
                p.copy_(master[k].bfloat16())
                p.grad = None


def exact(case, seed):
    """The training step's weights have no such value: AdamW's first steps are learning-rate steps in the sign of each
    gradient, and the sign of the many gradients near zero is that of their rounding.  Its loss has one."""
    kind = case["kind"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "train":
        if case["model"] != "tiny":
            return None  # four steps of it in 64 bits take too long
        return {"loss": _train_loss(case, seed), "master": None}
    if kind == "linear":
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        x, dy = _randn(g, t, i).double(), _randn(g, t, o).double()
        w, bias = _randn(g, o, i, std=0.02).double(), _randn(g, o, std=0.02).double()
        return {"y": x @ w.t() + bias, "dx": dy @ w, "dw": dy.t() @ x, "dbias": dy.sum(0)}
    if kind == "tp":
        t, h, c, r = case["tokens"], case["hidden"], case["col_out"], case["row_in"]
        x, dy, w_col = _randn(g, t, h).double(), _randn(g, t, c).double(), _randn(g, c, h, std=0.02).double()
        a, dz, w_row = _randn(g, t, r).double(), _randn(g, t, h).double(), _randn(g, h, r, std=0.02).double()
        return {"y": x @ w_col.t(), "z": a @ w_row.t(), "dx": dy @ w_col, "dw_col": dy.t() @ x, "da": dz @ w_row, "dw_row": dz.t() @ a}
    if kind == "fp8":
        # the quantised operands are the entry point's own first result, so the scales are taken in 32 bits as it takes them
        t, i, o = case["tokens"], case["n_in"], case["n_out"]
        x, w = _randn(g, t, i).float().view(t, i // 128, 128), _randn(g, o, i, std=0.02).float()
        top = torch.full((), 448.0, device="cuda")  # torch multiplies by the reciprocal of a Python number: another last bit
        sx = x.abs().amax(-1, keepdim=True) / top
        w = torch.nn.functional.pad(w, (0, 0, 0, -o % 128)).view(-1, 128, i // 128, 128)
        sw = w.abs().amax((1, 3), keepdim=True) / top
        xq = _fp8(x * (1 / sx)) * sx.double()
        wq = _fp8(w * (1 / sw)) * sw.double()
        return xq.view(t, i) @ wq.reshape(-1, i)[:o].t()
    if kind == "moe":
        t, h, f, e = case["tokens"], case["hidden"], case["ffn"], case["experts"]
        x = _randn(g, t, h).double()
        weights, idx = torch.topk(torch.softmax(torch.randn(t, e, generator=g, device="cuda"), -1), 2, dim=-1)
        up = [_randn(g, 2 * f, h, std=0.02) for _ in range(e)]
        down = [_randn(g, h, f, std=0.02) for _ in range(e)]
        out = torch.zeros(t, h, dtype=torch.float64, device="cuda")
        for i in range(e):
            rows, choice = (idx == i).nonzero(as_tuple=True)
            gu = x[rows] @ up[i].double().t()
            y = (torch.nn.functional.silu(gu[:, :f]) * gu[:, f:]) @ down[i].double().t()
            out.index_add_(0, rows, weights[rows, choice].double()[:, None] * y)
        return out
    n, count, op = case["ranks"], case["count"], case["op"]
    dtype = DTYPES[case["dtype"]][0]
    send_n = count * (n if op in ("reducescatter", "alltoall") else 1)
    send = [(torch.rand(send_n, generator=g, device="cuda") * 2 - 1).to(dtype).double() for _ in range(n)]
    if op == "allreduce":
        total = sum(send)
        return [total.clone() for _ in range(n)]
    if op == "reducescatter":
        return list(sum(send).view(n, count).unbind(0))
    if op == "allgather":
        return [torch.cat(send) for _ in range(n)]
    return [torch.cat([s.view(n, count)[r] for s in send]) for r in range(n)]
