"""Gradients of the embedding when one token holds a good part of all positions, as padding does: its rows are summed by two CTAs."""
import pytest
import torch

from flagcx_b200.ops import embed, enable_direct_grad

pytestmark = pytest.mark.gpu


def _tokens(M, V, shares):
    tok = torch.randint(len(shares), V, (M,), device="cuda")
    where = torch.rand(M, device="cuda")
    for k, share in enumerate(shares):
        lo = sum(shares[:k])
        tok = torch.where((where >= lo) & (where < lo + share), torch.full_like(tok, k), tok)
    return tok


# around the 2048 rows and the quarter of the positions from which two CTAs share a token; the most such tokens; all positions
@pytest.mark.parametrize("B,T,C,shares", [(1, 2048, 256, [1.0]), (1, 2049, 256, [1.0]), (3, 776, 1024, [0.95]), (4, 1024, 512, [0.55, 0.3]), (5, 1637, 256, [0.27, 0.26]),
                                          (8, 1024, 1024, [0.32, 0.32, 0.32]), (8, 1024, 256, [0.26, 0.24]), (2, 1200, 2048, [0.97]), (1, 16384, 256, [0.5])])
def test_gradients_match_float64(B, T, C, shares):
    """One rounding to bf16 of an fp32 sum of n rows and what was there."""
    torch.manual_seed(B * T)
    V = 300
    tok = _tokens(B * T, V, shares).view(B, T)
    wte, wpe = torch.randn(V, C, device="cuda").bfloat16().requires_grad_(True), torch.randn(T, C, device="cuda").bfloat16().requires_grad_(True)
    before = [torch.randn_like(wte), torch.randn_like(wpe)]
    dx = torch.randn(B, T, C, device="cuda").bfloat16()
    got = []
    for _ in range(2):
        for p, g in zip((wte, wpe), before):
            p.grad = g.clone()
            enable_direct_grad(p)
        embed(tok, wte, wpe).backward(dx)
        got.append(wte.grad.clone())
    assert torch.equal(*got)  # the same order of sums every time
    rows = dx.double().view(B * T, C)
    total, size = (torch.zeros(V, C, dtype=torch.float64, device="cuda").index_add_(0, tok.flatten(), r) for r in (rows, rows.abs()))
    ref, size = before[0].double() + total, size + before[0].double().abs()
    assert ((wte.grad.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (B * T + 1) * 2.0 ** -24 * size + 1e-30).all()
    ref, size = before[1].double() + rows.view(B, T, C).sum(0), rows.view(B, T, C).abs().sum(0) + before[1].double().abs()
    assert ((wpe.grad.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + (B + 1) * 2.0 ** -24 * size + 1e-30).all()


def test_padding_alone_is_not_slower_than_the_library():
    """16 x 1024 positions of one token, 2048 columns: 570 us through the library's embedding, 790 where one CTA sums all rows, 390 so."""
    B, T, C, V = 16, 1024, 2048, 32000
    tok = torch.zeros(B, T, dtype=torch.int64, device="cuda")
    wte, wpe = torch.randn(V, C, device="cuda").bfloat16().requires_grad_(True), torch.randn(T, C, device="cuda").bfloat16().requires_grad_(True)
    dx = torch.randn(B, T, C, device="cuda").bfloat16()

    def library():
        return torch.nn.functional.embedding(tok, wte) + wpe[:T]

    def best(fn):
        times = []
        for _ in range(12):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            fn().backward(dx)
            end.record()
            end.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)

    wte.grad, wpe.grad = torch.zeros_like(wte), torch.zeros_like(wpe)
    slow = best(library)
    for p in (wte, wpe):
        enable_direct_grad(p)
    assert best(lambda: embed(tok, wte, wpe)) < slow
