"""Zero-copy reductions of buffers that are 16- but not 32-byte aligned on either side, and of shifted ones at the edges of a warp's 31
units: sums in rank order in fp32, rounded once, equal to the bit; nothing beside the result is written."""
import pytest
import torch

from flagcx_b200.wrapper import FLAGCXLibrary
from tests.test_emu_collectives import Emu
from tests.test_zero_copy_alignment import _buffers, _in_order

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(native_lib):
    return FLAGCXLibrary(native_lib)


# shifts in elements, bf16: 8 is 16 bytes, 16 is 32; the others start inside a 16-byte block
@pytest.mark.parametrize("send_shift,recv_shift", [(8, 0), (0, 8), (8, 8), (16, 24), (3, 0), (5, 8), (15, 16)])
@pytest.mark.parametrize("n,nctas", [(2, 1), (4, 1), (8, 2)])
def test_reductions(lib, n, nctas, send_shift, recv_shift):
    dtype, thread_units = torch.bfloat16, 8 * 512 * nctas  # elements of one 16-byte unit per thread
    emu = Emu(lib, n)
    try:
        for count in (thread_units - 8, 2 * thread_units - 8, 2 * thread_units, 2 * thread_units + 1, 2 * thread_units + 8 * 31 + 3, 3 * thread_units - 7,
                      31 * 16 * 8 * nctas * 4 + 16, 9 * thread_units + 8 * 33 + 5):
            for op, kind, send_n in (("reducescatter", "rs_zc", n * count), ("allreduce", "ar_zc", count), ("reduce", "reduce_zc", count)):
                _, xs = _buffers(n, send_n, dtype, send_shift, seed=count)
                whole, ys = _buffers(n, count, dtype, recv_shift, seed=7)
                want = [w.clone() for w in whole]
                for r in range(n):
                    if op == "reduce" and r != 1:
                        continue
                    want[r][recv_shift:recv_shift + count] = _in_order([x[r * count:(r + 1) * count] for x in xs] if op == "reducescatter" else xs)
                emu.coll(op, kind, nctas, xs, ys, count, dtype, root=1)
                for r in range(n):
                    assert torch.equal(whole[r], want[r]), (op, count, r)
    finally:
        emu.close()


@pytest.mark.parametrize("n", [2, 4, 8])
@pytest.mark.parametrize("shift", [0, 4, 8])
def test_in_place(lib, n, shift):
    dtype, count = torch.float32, 20 * 512 * 4 + 13
    emu = Emu(lib, n)
    try:
        whole, xs = _buffers(n, count, dtype, shift, seed=3)
        want = [w.clone() for w in whole]
        total = _in_order(xs)
        for w in want:
            w[shift:shift + count] = total
        emu.coll("allreduce", "ar_zc", 2, xs, xs, count, dtype)
        for w, v in zip(whole, want):
            assert torch.equal(w, v)
    finally:
        emu.close()
