"""Zero-copy kinds on emulated ranks at every alignment of their pieces: 32-byte accesses, 16-byte ones, and pieces that start inside
a 16-byte block.  Moved bytes are equal; sums are taken in rank order in fp32 and rounded once, so they are equal too."""
import pytest
import torch

from flagcx_b200.wrapper import FLAGCXLibrary
from tests.test_emu_collectives import Emu

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(native_lib):
    return FLAGCXLibrary(native_lib)


def _buffers(n, elems, dtype, shift, seed):
    """n buffers of `elems` elements that start `shift` elements into an allocation, with guard elements on both sides."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    whole = [torch.randn(shift + elems + 64, generator=g, device="cuda").to(dtype) for _ in range(n)]
    return whole, [w[shift:shift + elems] for w in whole]


def _in_order(xs):
    total = xs[0].float()
    for x in xs[1:]:
        total = total + x.float()
    return total.to(xs[0].dtype)


# pieces shorter than a block, around one and two blocks, a warp's worth of blocks, and more than one turn of every loop
@pytest.mark.parametrize("n,nctas", [(2, 1), (2, 16), (4, 3), (8, 16), (3, 4)])
@pytest.mark.parametrize("count", [1, 5, 8, 15, 16, 31, 33, 64, 519, 4096, 100003, 400000])
@pytest.mark.parametrize("dtype,send_shift,recv_shift", [(torch.bfloat16, 0, 0), (torch.bfloat16, 3, 0), (torch.bfloat16, 8, 5), (torch.float32, 0, 0),
                                                         (torch.float32, 1, 4)])
def test_pieces_of_any_alignment(lib, n, nctas, count, dtype, send_shift, recv_shift):
    emu = Emu(lib, n)
    try:
        for op, kind, send_n, recv_n in (("allgather", "move_zc", count, n * count), ("a2a", "move_zc", n * count, n * count),
                                         ("reducescatter", "rs_zc", n * count, count), ("allreduce", "ar_zc", count, count)):
            _, xs = _buffers(n, send_n, dtype, send_shift, seed=count)
            whole, ys = _buffers(n, recv_n, dtype, recv_shift, seed=7)
            guard = [w.clone() for w in whole]
            emu.coll(op, kind, nctas, xs, ys, count, dtype)
            for r in range(n):
                if op == "allgather":
                    want = torch.cat(xs)
                elif op == "a2a":
                    want = torch.cat([x[r * count:(r + 1) * count] for x in xs])
                elif op == "reducescatter":
                    want = _in_order([x[r * count:(r + 1) * count] for x in xs])
                else:
                    want = _in_order(xs)
                assert torch.equal(ys[r], want), (op, r)
                assert torch.equal(whole[r][:recv_shift], guard[r][:recv_shift]) and torch.equal(whole[r][recv_shift + recv_n:], guard[r][recv_shift + recv_n:]), op
    finally:
        emu.close()
