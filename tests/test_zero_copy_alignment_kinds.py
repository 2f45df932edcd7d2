"""Zero-copy kinds with one root and all-to-all-v at every alignment of their pieces, with CTAs that divide by the ranks (a piece has
CTAs of its own) and that do not; and the reductions' operations, with infinities and NaN, in wide, shifted and single units."""
import pytest
import torch

from flagcx_b200.wrapper import FLAGCXLibrary
from tests.test_emu_collectives import Emu
from tests.test_zero_copy_alignment import _buffers, _in_order

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(native_lib):
    return FLAGCXLibrary(native_lib)


def _unchanged_around(whole, before, shift, elems):
    return torch.equal(whole[:shift], before[:shift]) and torch.equal(whole[shift + elems:], before[shift + elems:])


@pytest.mark.parametrize("n,nctas", [(2, 1), (2, 16), (4, 3), (8, 16), (3, 4), (3, 6)])
@pytest.mark.parametrize("count", [1, 8, 15, 31, 64, 519, 100003])
@pytest.mark.parametrize("dtype,send_shift,recv_shift", [(torch.bfloat16, 0, 0), (torch.bfloat16, 3, 0), (torch.bfloat16, 8, 5), (torch.float32, 1, 4)])
def test_rooted_kinds_of_any_alignment(lib, n, nctas, count, dtype, send_shift, recv_shift):
    emu = Emu(lib, n)
    try:
        for op, kind, send_n, recv_n in (("bcast", "move_zc", count, count), ("gather", "move_zc", count, n * count),
                                         ("scatter", "move_zc", n * count, count), ("reduce", "reduce_zc", count, count)):
            for root in (0, n - 1):
                _, xs = _buffers(n, send_n, dtype, send_shift, seed=count + root)
                whole, ys = _buffers(n, recv_n, dtype, recv_shift, seed=7)
                before = [w.clone() for w in whole]
                emu.coll(op, kind, nctas, xs, ys, count, dtype, root=root)
                for r in range(n):
                    if op == "bcast":
                        want = xs[root]
                    elif op == "scatter":
                        want = xs[root][r * count:(r + 1) * count]
                    elif r != root:
                        want = before[r][recv_shift:recv_shift + recv_n]  # only the root's buffer is written
                    else:
                        want = torch.cat(xs) if op == "gather" else _in_order(xs)
                    assert torch.equal(ys[r], want), (op, root, r)
                    assert _unchanged_around(whole[r], before[r], recv_shift, recv_n), (op, root, r)
    finally:
        emu.close()


@pytest.mark.parametrize("n,nctas", [(2, 2), (4, 3), (8, 16)])
@pytest.mark.parametrize("unit", [1, 17, 4001])
@pytest.mark.parametrize("shift", [0, 1, 8])
def test_alltoallv_of_any_alignment(lib, n, nctas, unit, shift):
    """Counts that differ by pair, some of them none, with a gap of one element between the received pieces."""
    dtype = torch.bfloat16
    emu = Emu(lib, n)
    try:
        sc = [[unit * ((r + 2 * p) % 3) + (p & 1) for p in range(n)] for r in range(n)]
        sd = [[sum(sc[r][:p]) for p in range(n)] for r in range(n)]
        rc = [[sc[p][r] for p in range(n)] for r in range(n)]
        rd = [[sum(rc[r][:p]) + p for p in range(n)] for r in range(n)]
        send_n, recv_n = max(sum(c) for c in sc) + 1, max(sum(c) for c in rc) + n
        _, xs = _buffers(n, send_n, dtype, shift, seed=unit)
        whole, ys = _buffers(n, recv_n, dtype, shift, seed=7)
        want = [w.clone() for w in whole]
        for r in range(n):
            for p in range(n):
                at = shift + rd[r][p]
                want[r][at:at + rc[r][p]] = xs[p][sd[p][r]:sd[p][r] + sc[p][r]]
        emu.coll("a2av", "move_zc", nctas, xs, ys, 0, dtype, tables=[v for r in range(n) for t in (sc, sd, rc, rd) for v in t[r]])
        for r in range(n):
            assert torch.equal(whole[r], want[r]), r
    finally:
        emu.close()


def _want(xs, red):
    acc = xs[0].float()
    for x in xs[1:]:
        x = x.float()
        acc = acc + x if red in (0, 4) else torch.where(acc > x, acc, x) if red == 2 else torch.where(acc < x, acc, x)
    if red == 4:
        acc = acc / torch.full_like(acc, len(xs))  # by a Python number, torch on the GPU multiplies by its reciprocal
    return acc.to(xs[0].dtype)


# units of the general path, 32-byte pieces, and (shift) units that lie in two 16-byte blocks
@pytest.mark.parametrize("n,nctas,count", [(2, 1, 9000), (4, 2, 30011), (8, 1, 20003), (3, 2, 9001), (8, 16, 519)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shift", [0, 1])
def test_operations_and_special_values(lib, n, nctas, count, dtype, shift):
    emu = Emu(lib, n)
    try:
        for red in (0, 2, 3, 4):  # sum, max, min, average
            for op, kind, send_n in (("reducescatter", "rs_zc", n * count), ("allreduce", "ar_zc", count)):
                _, xs = _buffers(n, send_n, dtype, shift, seed=red)
                for r, x in enumerate(xs):
                    x[r::97] = float("inf")
                    x[r + 5::101] = -float("inf")
                    x[3 * r::103] = float("nan")
                    x[7::107] = torch.finfo(dtype).min
                _, ys = _buffers(n, count, dtype, 0, seed=7)
                emu.coll(op, kind, nctas, xs, ys, count, dtype, red=red)
                for r in range(n):
                    want = _want([x[r * count:(r + 1) * count] for x in xs] if op == "reducescatter" else xs, red)
                    assert torch.equal(ys[r].isnan(), want.isnan()), (op, red, r)
                    assert torch.equal(ys[r].nan_to_num(1.0, 2.0, 3.0), want.nan_to_num(1.0, 2.0, 3.0)), (op, red, r)
    finally:
        emu.close()
