"""Token + position embedding: one kernel each way, against float64 sums."""
import pytest
import torch

from flagcx_b200.ops import embed, enable_direct_grad

pytestmark = pytest.mark.gpu


def _tokens(kind, B, T, V):
    if kind == "one":  # every position holds the same token: the whole CTA's work
        return torch.full((B, T), V - 1, dtype=torch.int64, device="cuda")
    tok = torch.randint(0, V, (B, T), device="cuda")
    if kind == "skew":  # a few tokens with many rows among many with one
        tok = torch.where(torch.rand(B, T, device="cuda") < 0.3, tok % 3, tok)
    return tok


@pytest.mark.parametrize("direct", [False, True])
@pytest.mark.parametrize("B,T,C,V,kind", [(1, 1, 256, 8, "random"), (2, 64, 256, 1000, "random"), (1, 129, 512, 3, "random"), (3, 776, 1024, 50304, "random"),
                                          (8, 1024, 1024, 50304, "skew"), (4, 100, 2048, 50, "skew"), (2, 300, 1024, 7, "one"), (1, 16384, 256, 997, "skew"),
                                          (17, 1024, 256, 997, "random"), (2, 64, 320, 1000, "random")])
def test_embedding_matches_float64(B, T, C, V, kind, direct):
    """The last two sizes are the library's (too many tokens, rows that are no whole vectors).  A gradient is one rounding to bf16
    of an fp32 sum of n rows and what was there: 2^-8 of it, and n 2^-24 of the rows' absolute sum; the library's own path rounds
    the sum, and the total with what was there, one after the other: three roundings of at most the absolute sum."""
    torch.manual_seed(B * 1000 + T)
    tok = _tokens(kind, B, T, V)
    wte, wpe = torch.randn(V, C, device="cuda").bfloat16().requires_grad_(True), torch.randn(T + 3, C, device="cuda").bfloat16().requires_grad_(True)
    before = [torch.zeros_like(wte), torch.zeros_like(wpe)]
    if direct:
        before = [torch.randn_like(wte), torch.randn_like(wpe)]
        for p, g in zip((wte, wpe), before):
            p.grad = g.clone()
            enable_direct_grad(p)
    x = embed(tok, wte, wpe)
    assert torch.equal(x, (wte.float()[tok] + wpe.float()[:T]).bfloat16())
    dx = torch.randn_like(x)
    x.backward(dx)
    rows = dx.double().view(B * T, C)
    sums = [torch.zeros(V, C, dtype=torch.float64, device="cuda").index_add_(0, tok.flatten(), r) for r in (rows, rows.abs())]
    sums += [torch.zeros(T + 3, C, dtype=torch.float64, device="cuda") for _ in range(2)]
    sums[2][:T], sums[3][:T] = rows.view(B, T, C).sum(0), rows.view(B, T, C).abs().sum(0)
    own = B * T <= 16384 and C % 256 == 0
    for p, b, total, size, n in ((wte, before[0], sums[0], sums[1], B * T), (wpe, before[1], sums[2], sums[3], B)):
        ref = b.double() + total
        size = size + b.double().abs()
        bound = 2.0 ** -8 * (ref.abs() if own else 3 * size) + (n + 1) * 2.0 ** -24 * size + 1e-30
        assert ((p.grad.double() - ref).abs() <= bound).all()
    if kind != "random":
        again = wte.grad.clone()
        wte.grad = before[0].clone() if direct else None
        wpe.grad = before[1].clone() if direct else None
        embed(tok, wte, wpe).backward(dx)
        assert not own or torch.equal(again, wte.grad)  # sums in position order: the same twice


def test_positions_without_a_row_are_refused():
    with pytest.raises(RuntimeError):
        embed(torch.zeros(1, 9, dtype=torch.int64, device="cuda"), torch.zeros(4, 256, device="cuda").bfloat16(), torch.zeros(8, 256, device="cuda").bfloat16())
