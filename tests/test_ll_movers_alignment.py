"""Low-latency movers on emulated ranks with pieces that start at any byte: 8-, 4-, 2- and 1-byte accesses and the ragged end."""
import pytest
import torch

from flagcx_b200.wrapper import FLAGCXLibrary
from tests.test_emu_collectives import Emu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 5, 8])
@pytest.mark.parametrize("dtype", [torch.uint8, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("count,shift", [(1, 0), (7, 1), (8, 0), (9, 3), (1000, 0), (1001, 0), (4093, 2), (8191, 1)])
def test_pieces_of_any_alignment(native_lib, n, dtype, count, shift):
    emu = Emu(FLAGCXLibrary(native_lib), n)
    g = torch.Generator(device="cuda").manual_seed(count)
    try:
        for op, send_n, recv_n in (("allgather", count, n * count), ("a2a", n * count, n * count), ("bcast", count, count)):
            whole = [torch.randint(0, 100, (shift + send_n,), generator=g, device="cuda").to(dtype) for _ in range(n)]
            xs = [w[shift:] for w in whole]
            out = [torch.full((shift + recv_n + 16,), 101, device="cuda").to(dtype) for _ in range(n)]
            ys = [o[shift:shift + recv_n] for o in out]
            emu.coll(op, "move_ll", 1, xs, ys, count, dtype, root=n - 1)
            for r in range(n):
                if op == "allgather":
                    want = torch.cat(xs)
                elif op == "a2a":
                    want = torch.cat([x[r * count:(r + 1) * count] for x in xs])
                else:
                    want = xs[n - 1]
                assert torch.equal(ys[r], want), (op, r)
                assert (out[r][:shift] == 101).all() and (out[r][shift + recv_n:] == 101).all(), op
    finally:
        emu.close()
