"""Expert-parallel MoE pieces on one GPU against fp32 PyTorch references:
the building blocks of one expert (device-row-count GEMM, SiLU-mul, the GEMM that
scatters its rows), and the whole fused layer on a one-rank communicator
(dispatch kernel, grouped expert GEMMs, combine kernel)."""
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
    uid = lib.flagcxGetUniqueId()
    comm = lib.flagcxCommInitRank(1, uid, 0)
    yield lib, comm
    torch.cuda.synchronize()
    lib.flagcxCommDestroy(comm)


@pytest.mark.parametrize("rows", [0, 1, 127, 128, 300, 512])
def test_gemm_with_device_row_count(nat, rows):
    torch.manual_seed(rows)
    a = (torch.randn(512, 256, device="cuda") * 0.5).bfloat16()
    b = (torch.randn(384, 256, device="cuda") * 0.5).bfloat16()
    c = torch.full((512, 384), 7.0, device="cuda", dtype=torch.bfloat16)
    m = torch.tensor([rows], dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    nat.gemm_dyn_m(a, b, c, m, err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = a.float() @ b.float().t()
    if rows:
        e = (c[:rows].float() - ref[:rows]).abs().max() / ref.abs().max()
        assert e < 2e-2
    assert bool((c[rows:] == 7.0).all())  # rows beyond the count stay untouched


@pytest.mark.parametrize("rows,cap,pad", [(0, 200, 0), (1, 40, 8), (129, 200, 0), (300, 300, 16)])
def test_gemm_that_scatters_its_rows(nat, comm1, rows, cap, pad):
    """One expert's output projection: buffers whose row count is no multiple of a tile, strided rows, top-2 places."""
    lib, comm = comm1
    torch.manual_seed(rows)
    K, N, T = 136, 200, 150
    a = (torch.randn(cap, K + pad, device="cuda") * 0.5).bfloat16()[:, :K]
    b = (torch.randn(N, K + pad, device="cuda") * 0.5).bfloat16()[:, :K]
    place = torch.randperm(2 * T, device="cuda")[:cap]  # (token, choice) of each row
    info = torch.zeros(cap, 4, dtype=torch.int32, device="cuda")
    info[:, 1], info[:, 2] = place // 2, place % 2
    back = nat.heap_tensor(comm.value, [2 * T, N], torch.bfloat16).fill_(5.0)
    done = nat.heap_tensor(comm.value, [2], torch.int64).zero_()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    m = torch.tensor([rows], dtype=torch.int32, device="cuda")
    grid = nat.gemm_rowmap(comm.value, a, b, m, info, back, done, 2, err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0 and int(done[0].item()) == grid
    want = torch.full((2 * T, N), 5.0, dtype=torch.float64, device="cuda")
    want[place[:rows]] = a[:rows].double() @ b.double().t()
    bound = 2.0 ** -8 * want.abs() + K * 2.0 ** -23 * K  # one rounding; products stay below one on average
    assert bool(((back.double() - want).abs() <= bound).all())


def test_silu_mul(nat):
    torch.manual_seed(3)
    gu = torch.randn(300, 2 * 512, device="cuda").bfloat16()
    h = torch.zeros(300, 512, device="cuda", dtype=torch.bfloat16)
    rows = torch.tensor([257], dtype=torch.int32, device="cuda")
    nat.silu_mul(gu, h, rows)
    torch.cuda.synchronize()
    ref = torch.nn.functional.silu(gu[:, :512].float()) * gu[:, 512:].float()
    assert ((h[:257].float() - ref[:257]).abs() / (ref[:257].abs() + 1.0)).max() < 2e-2
    assert bool((h[257:] == 0).all())
    nat.silu_mul(gu, h)
    torch.cuda.synchronize()
    assert ((h.float() - ref).abs() / (ref.abs() + 1.0)).max() < 2e-2


def test_fused_layer_on_one_rank(nat, comm1):
    from flagcx_b200.parallel.ep import ExpertParallelContext, moe_reference
    lib, comm = comm1
    T, H, F, K = 640, 512, 1024, 2
    ep = ExpertParallelContext(comm.value, 1, 0, T, H, F, K, dispatch_ctas=8)
    torch.manual_seed(4)
    w1 = (torch.randn(2 * F, H, device="cuda") * 0.05).bfloat16()
    w2 = (torch.randn(H, F, device="cuda") * 0.05).bfloat16()
    for rep in range(3):  # both buffer parities and a reused one
        x = torch.randn(T, H, device="cuda").bfloat16()
        idx = torch.zeros(T, K, dtype=torch.int32, device="cuda")
        idx[rep::7, 1] = -1  # a choice that is not dispatched
        wts = torch.rand(T, K, device="cuda")
        wts[idx < 0] = 0
        out = ep.forward(x, idx, wts, w1, w2)
        torch.cuda.synchronize()
        ep.check()
        assert int(ep.recv_total.item()) == int((idx == 0).sum().item())
        ref = moe_reference(x, idx, wts, [w1], [w2])
        e = (out.float() - ref).abs().max() / ref.abs().max()
        assert e < 3e-2, (rep, float(e))
        un = ep.unfused_forward(x, idx.clamp(min=0), wts, w1, w2)
        e = (un.float() - ref).abs().max() / ref.abs().max()
        assert e < 3e-2, ("unfused", rep, float(e))


def test_fused_layer_with_four_experts_on_one_rank(nat, comm1):
    """Several experts per rank: the dispatch kernel sorts the rows into one segment per local expert and every
    expert's GEMMs size themselves from their own device-resident row count."""
    from flagcx_b200.parallel.ep import ExpertParallelContext, moe_reference
    lib, comm = comm1
    T, H, F, K, L = 768, 512, 768, 2, 4
    ep = ExpertParallelContext(comm.value, 1, 0, T, H, F, K, dispatch_ctas=8, experts_per_rank=L, capacity_factor=1.5)
    torch.manual_seed(5)
    w1 = [(torch.randn(2 * F, H, device="cuda") * 0.05).bfloat16() for _ in range(L)]
    w2 = [(torch.randn(H, F, device="cuda") * 0.05).bfloat16() for _ in range(L)]
    for rep in range(3):
        x = torch.randn(T, H, device="cuda").bfloat16()
        first = torch.randint(0, L, (T,), device="cuda")
        idx = torch.stack([first, (first + 1 + torch.randint(0, L - 1, (T,), device="cuda")) % L], dim=1).int().contiguous()
        idx[rep::11, 1] = -1  # a choice that is not dispatched
        wts = torch.rand(T, K, device="cuda")
        wts[idx < 0] = 0
        out = ep.forward(x, idx, wts, w1, w2)
        torch.cuda.synchronize()
        ep.check()
        assert ep.recv_total.tolist() == [int((idx == e).sum().item()) for e in range(L)]
        ref = moe_reference(x, idx, wts, w1, w2)
        e = (out.float() - ref).abs().max() / ref.abs().max()
        assert e < 3e-2, (rep, float(e))


@pytest.mark.parametrize("T,H,F,L", [(512, 1024, 2048, 4), (777, 264, 520, 3)])
def test_fused_layer_repeats_exactly_and_rounds_gate_and_up_only_once(nat, comm1, T, H, F, L):
    """Call after call gives the same bits, with other inputs in between; and the result is no further from 64 bits than
    the layer whose gate and up products are rounded to bf16 before the activation, which the fused one does without."""
    from flagcx_b200.parallel.ep import ExpertParallelContext
    lib, comm = comm1
    K = 2
    ep = ExpertParallelContext(comm.value, 1, 0, T, H, F, K, experts_per_rank=L, capacity_factor=2.0)
    torch.manual_seed(T)
    up = [(torch.randn(2 * F, H, device="cuda") * 0.02).bfloat16() for _ in range(L)]
    down = [(torch.randn(H, F, device="cuda") * 0.02).bfloat16() for _ in range(L)]
    batches = []
    for _ in range(2):
        w, idx = torch.topk(torch.softmax(torch.randn(T, L, device="cuda"), -1), K, dim=-1)
        batches.append((torch.randn(T, H, device="cuda").bfloat16(), idx.int().contiguous(), w.contiguous()))
    first = [ep.forward(*b, up, down) for b in batches]
    for _ in range(3):
        for b, want in zip(batches, first):
            assert torch.equal(ep.forward(*b, up, down), want)
    ep.check()

    def layer(x, idx, w, rounded):
        r = (lambda t: t.bfloat16().double()) if rounded else (lambda t: t)
        out = torch.zeros(T, H, dtype=torch.float64, device="cuda")
        for e in range(L):
            rows, choice = (idx == e).nonzero(as_tuple=True)
            gu = r(x[rows].double() @ up[e].double().t())
            y = r(r(torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]) @ down[e].double().t())
            out.index_add_(0, rows, w[rows, choice].double()[:, None] * y)
        return r(out)

    for b, got in zip(batches, first):
        exact, rounded = layer(*b, False), layer(*b, True)
        assert float((got.double() - exact).norm()) < 0.9 * float((rounded - exact).norm())
