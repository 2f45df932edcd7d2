"""``ops.embed`` under second derivatives and function transforms: what the library's embedding gives for the same call."""
import pytest
import torch

from flagcx_b200.ops import embed

pytestmark = pytest.mark.gpu

B, T, C, V = 2, 24, 256, 50  # a size that the embedding kernels take


def _inputs():
    g = torch.Generator(device="cuda").manual_seed(5)
    tok = torch.randint(0, V, (B, T), generator=g, device="cuda")
    wte, wpe = (torch.randn(n, C, generator=g, device="cuda").bfloat16() for n in (V, T + 2))
    return tok, wte, wpe, torch.randn(B, T, C, generator=g, device="cuda").bfloat16()


def _library(tok, wte, wpe):
    return torch.nn.functional.embedding(tok, wte) + wpe[:tok.shape[1]]


@pytest.mark.parametrize("asked", [(0,), (1,), (0, 1)])
def test_gradients_have_a_graph_under_create_graph(asked):
    tok, wte, wpe, dx = _inputs()
    tables = wte.requires_grad_(), wpe.requires_grad_()
    got = []
    for fn in (embed, _library):
        g = dx.clone().requires_grad_()
        grads = torch.autograd.grad(fn(tok, *tables), [tables[i] for i in asked], g, create_graph=True)
        ones = [torch.full_like(t, 0.5) for t in grads]
        got.append([*grads, *torch.autograd.grad(grads, (g,), ones)])
    for a, b in zip(*got, strict=True):
        assert torch.equal(a, b)


def test_transforms():
    tok, wte, wpe, dx = _inputs()

    def results(f):
        out = [torch.func.grad(lambda w: (f(tok, w, wpe) * dx).float().sum())(wte), torch.func.vmap(lambda p: f(tok, wte, p))(torch.stack([wpe, 2 * wpe])),
               *torch.func.jvp(lambda p: f(tok, wte, p), (wpe,), (torch.ones_like(wpe),))]
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(wte, torch.ones_like(wte))
            out.append(torch.autograd.forward_ad.unpack_dual(f(tok, dual, wpe)).tangent)
        out.append(torch.jit.trace(f, (tok, wte, wpe), check_trace=False)(tok.flip(0), wte, wpe))
        return out

    for a, b in zip(results(embed), results(_library), strict=True):
        assert torch.equal(a, b)
