"""``ops.linear`` as a part of autograd: hooks on saved tensors, checkpointing, streams, threads, and what it refuses."""
import threading

import pytest
import torch

from flagcx_b200.ops import linear

pytestmark = pytest.mark.gpu

# products whose K is not cut, so that results repeat to the bit: T, I, O
T, I, O = 264, 320, 448


def _inputs(seed, lead=(T,)):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    return r(*lead, I).requires_grad_(), r(O, I).requires_grad_(), r(O).requires_grad_(), r(*lead, O)


def _grads(x, w, b, dy):
    y = linear(x, w, b)
    return [y.detach(), *torch.autograd.grad(y, (x, w, b), dy)]


def _same(got, want):
    assert all(torch.equal(g, w) for g, w in zip(got, want, strict=True))


@pytest.mark.parametrize("lead", [(T,), (3, 88)])
def test_hooks_on_saved_tensors_see_the_input_and_the_weight(lead):
    x, w, b, dy = _inputs(1, lead)
    want = _grads(x, w, b, dy)
    packed = []

    def pack(t):
        packed.append(t.numel())
        return t.cpu()

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        y = linear(x, w, b)
        assert sorted(packed) == sorted([x.numel(), w.numel()])
        _same([y.detach(), *torch.autograd.grad(y, (x, w, b), dy)], want)


@pytest.mark.parametrize("reentrant", [False, True])
def test_activation_checkpointing(reentrant):
    from torch.utils.checkpoint import checkpoint
    x, w, b, dy = _inputs(2)
    want = _grads(x, w, b, dy)
    y = checkpoint(linear, x, w, b, use_reentrant=reentrant)
    if reentrant:
        y.backward(dy)
        _same([y.detach(), x.grad, w.grad, b.grad], want)
    else:
        _same([y.detach(), *torch.autograd.grad(y, (x, w, b), dy)], want)


def test_a_weight_changed_between_forward_and_backward_is_noticed():
    x, w, b, dy = _inputs(3)
    y = linear(x, w, b)
    with torch.no_grad():
        w.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, (x,), dy)


def test_two_streams_at_a_time():
    """Forward and backward on two side streams at once, many times over, against the same calls one after the other."""
    sets = [_inputs(10 + i) for i in range(2)]
    want = [_grads(*s) for s in sets]
    streams = [torch.cuda.Stream() for _ in sets]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(_grads(*sets[i]))
    torch.cuda.synchronize()
    for i in range(2):
        for g in got[i]:
            _same(g, want[i])


def test_threads_with_a_stream_each():
    """The launchers' host code from four threads at once."""
    sets = [_inputs(20 + i) for i in range(4)]
    want = [_grads(*s) for s in sets]
    torch.cuda.synchronize()
    got, errors = [[] for _ in sets], []

    def work(i):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                for _ in range(10):
                    got[i].append(_grads(*sets[i]))
            stream.synchronize()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(sets))]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert not errors, errors
    for i in range(len(sets)):
        assert len(got[i]) == 10
        for g in got[i]:
            _same(g, want[i])


def test_transforms_that_it_does_not_support_are_refused():
    x, w, b, dy = _inputs(4)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x.detach(), torch.ones_like(x))
        with pytest.raises((RuntimeError, NotImplementedError)):
            linear(dual, w, b)
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda t: linear(t, w, b).float().sum())(x.detach())
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda t: linear(t, w, b))(torch.stack([x.detach(), x.detach()]))
    # a second derivative is refused, not silently zero
    dyg = dy.clone().requires_grad_()
    dx, = torch.autograd.grad(linear(x, w, b), (x,), dyg, create_graph=True)
    with pytest.raises(RuntimeError):
        torch.autograd.grad(dx.float().sum(), (dyg,))
