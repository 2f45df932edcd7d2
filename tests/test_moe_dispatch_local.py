"""The dispatch of one rank without an exchange against the cooperative kernel that exchanges with itself."""
import pytest
import torch

from flagcx_b200.parallel.ep import ExpertParallelContext

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def comm1():
    from flagcx_b200.wrapper import FLAGCXLibrary
    lib = FLAGCXLibrary()
    torch.zeros(1, device="cuda")
    comm = lib.flagcxCommInitRank(1, lib.flagcxGetUniqueId(), 0)
    yield comm
    torch.cuda.synchronize()
    lib.flagcxCommDestroy(comm)


# tokens: one entry, stretches that end inside a warp's 32, more entries than two CTAs per SM have warps, a byte's worth of
# entries per thread; hidden sizes under, at and over a warp's 256 vectors
@pytest.mark.parametrize("T,K,H,L,capacity", [(1, 1, 64, 1, 1.0), (33, 2, 264, 3, 3.0), (517, 2, 1024, 4, 2.0), (5000, 3, 2048, 9, 2.0),
                                              (4097, 2, 2056, 17, 2.0), (70001, 1, 8, 64, 1.5), (3000, 2, 512, 8, 0.5)])
def test_same_rows_as_with_the_exchange(comm1, T, K, H, L, capacity):
    torch.manual_seed(T)
    x = torch.randn(T, H, device="cuda").bfloat16()
    idx = torch.randint(-1, L + 1, (T, K), device="cuda", dtype=torch.int32)  # some choices are not dispatched
    got = []
    for exchange in (True, False):
        ep = ExpertParallelContext(comm1.value, 1, 0, T, H, 64, K, capacity_factor=capacity, dispatch_ctas=64, experts_per_rank=L)
        ep.exchange = exchange
        ep.recv[0].zero_()
        ep.info[0].fill_(-7)
        ep.nat.moe_dispatch(ep.comm, x, idx, ep.count_mat[0], ep.count_flags[0], ep.recv[0], ep.info[0], ep.disp_done[0], 1, ep.slot,
                            ep.local_counts, ep.recv_total, ep.err, 64, L, ep.exchange)
        torch.cuda.synchronize()
        valid = (idx >= 0) & (idx < L)
        got.append([t.clone() for t in (ep.recv[0], ep.info[0], ep.recv_total, ep.local_counts, ep.err)] + [ep.slot.view(T, K)[valid].clone()])
        del ep
    for a, b in zip(*got):
        assert torch.equal(a, b)
