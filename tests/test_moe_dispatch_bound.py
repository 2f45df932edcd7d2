"""How many CTAs the dispatch of one rank takes: never more than the caller's ``dispatch_ctas``."""
import ctypes

import pytest
import torch

import flagcx_b200


def _plan(entries, ctas, sms=148):
    lib = ctypes.CDLL(flagcx_b200.native().__file__)
    threads = ctypes.c_int()
    return lib.fcxMoeDispatchPlan(ctypes.c_int64(entries), ctas, sms, ctypes.byref(threads)), threads.value


def test_plan_keeps_to_the_callers_bound():
    for entries in (0, 1, 16, 17, 1000, 1024, 8192, 8193, 16384, 65536, 65537, 148 * 1024, 148 * 1024 + 1, 1 << 20, (1 << 31) - 1):
        for ctas in (0, 1, 8, 64, 148, 1000):
            grid, threads = _plan(entries, ctas)
            assert 0 <= grid <= max(1, min(ctas, 148)) and threads in (512, 1024)
            assert grid == 0 or grid * 1024 >= entries  # what a CTA's shared memory holds


def test_counting_does_not_grow_with_the_square_of_the_entries():
    """Every CTA reads all entries before its own stretch: more of them than were timed go to the cooperative kernel."""
    assert _plan(148 * 1024, 148)[0] == 148 and _plan(148 * 1024 + 1, 148)[0] == 0
    assert _plan(1 << 20, 1000)[0] == 0 and _plan(65537, 64)[0] == 0 and _plan(8193, 8)[0] == 0


def test_timed_choices():
    assert _plan(1024, 64) == (64, 512) and _plan(4096, 64) == (64, 512) and _plan(16384, 148) == (148, 512)
    assert _plan(16384, 64) == (64, 1024) and _plan(32768, 148) == (148, 1024)


class _KernelNode(ctypes.Structure):  # cudaKernelNodeParams
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p)]


def _kernel_grids(graph):
    rt = ctypes.CDLL("libcudart.so.12")
    handle, n = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t()
    assert rt.cudaGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    grids = []
    for node in nodes:
        kind, p = ctypes.c_int(), _KernelNode()
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        if kind.value == 0:
            assert rt.cudaGraphKernelNodeGetParams(ctypes.c_void_p(node), ctypes.byref(p)) == 0
            grids.append(p.grid[0] * p.grid[1] * p.grid[2])
    return grids


@pytest.fixture(scope="module")
def comm1():
    from flagcx_b200.wrapper import FLAGCXLibrary
    lib = FLAGCXLibrary()
    torch.zeros(1, device="cuda")
    comm = lib.flagcxCommInitRank(1, lib.flagcxGetUniqueId(), 0)
    yield comm
    torch.cuda.synchronize()
    lib.flagcxCommDestroy(comm)


@pytest.mark.gpu
@pytest.mark.parametrize("T,K,ctas", [(64, 2, 8), (3000, 2, 8), (3000, 2, 64), (9000, 2, 16), (9000, 2, 1000), (75000, 2, 148)])
def test_launch_keeps_to_the_callers_bound_and_moves_the_same_rows(comm1, T, K, ctas):
    """The launch as a captured graph has it, and its rows against those of the exchange that one rank has with itself."""
    from flagcx_b200.parallel.ep import ExpertParallelContext
    H, L = 1032 if T < 10000 else 8, 5
    torch.manual_seed(T)
    x = torch.randn(T, H, device="cuda").bfloat16()
    idx = torch.randint(-1, L + 1, (T, K), device="cuda", dtype=torch.int32)
    got = []
    for exchange in (True, False):
        ep = ExpertParallelContext(comm1.value, 1, 0, T, H, 64, K, capacity_factor=2.0, dispatch_ctas=ctas, experts_per_rank=L)
        ep.recv[0].zero_()
        ep.info[0].fill_(-7)

        def dispatch():
            ep.nat.moe_dispatch(ep.comm, x, idx, ep.count_mat[0], ep.count_flags[0], ep.recv[0], ep.info[0], ep.disp_done[0], 1, ep.slot,
                                ep.local_counts, ep.recv_total, ep.err, ep.dispatch_ctas, L, exchange)

        dispatch()
        torch.cuda.synchronize()
        valid = (idx >= 0) & (idx < L)
        got.append([t.clone() for t in (ep.recv[0], ep.info[0], ep.recv_total, ep.local_counts, ep.err)] + [ep.slot.view(T, K)[valid].clone()])
        if not exchange:
            graph = torch.cuda.CUDAGraph(keep_graph=True)
            with torch.cuda.graph(graph):
                dispatch()
            grids = _kernel_grids(graph)
            assert len(grids) == 1 and 1 <= grids[0] <= max(L, min(ctas, torch.cuda.get_device_properties(0).multi_processor_count))
        del ep
    for a, b in zip(*got, strict=True):
        assert torch.equal(a, b)
