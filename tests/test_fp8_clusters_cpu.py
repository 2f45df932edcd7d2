"""Which tile the block-scaled fp8 GEMM takes and how many CTAs share it: only as many clusters as are on the chip at once."""
import ctypes

import pytest

import flagcx_b200

SMS, PAIRS, QUADS = 148, 74, 33  # of the B200 that was timed


@pytest.fixture(scope="module")
def lib():
    return ctypes.CDLL(flagcx_b200.native().__file__)


def _plan(lib, m, n, k, sms=SMS, pairs=PAIRS, quads=QUADS):
    cut = ctypes.c_int()
    return lib.fcxGemmFp8PlanFor(m, n, k, sms, pairs, quads, ctypes.byref(cut)), cut.value


def _tiles(m, n, width):
    return -(-m // 128) * -(-n // width)


def test_every_cluster_is_on_the_chip_at_once(lib):
    for pairs, quads in ((74, 33), (74, 37), (70, 32), (74, 0), (0, 0)):
        for m in (1, 100, 129, 333, 1000):
            for n in range(64, 4801, 64):
                for nk in (8, 11, 12, 13, 16, 32, 64):
                    tile, cut = _plan(lib, m, n, nk * 128, pairs=pairs, quads=quads)
                    assert cut == 1 or nk >= 12
                    assert cut == 1 or _tiles(m, n, tile) <= {2: pairs, 4: quads}[cut], (m, n, nk, tile, cut)


def test_the_plan_of_a_launch_keeps_to_it_too(lib):
    """SMs of one GPC only make a cluster: eight GPCs of whole pairs of SMs hold between 33 and 37 clusters of four."""
    cut = ctypes.c_int()
    tile = lib.fcxGemmFp8Plan(100, 64 * 37, 4096, SMS, ctypes.byref(cut))
    assert (tile, cut.value) == (64, 2)
    tile = lib.fcxGemmFp8Plan(100, 64 * 33, 4096, SMS, ctypes.byref(cut))
    assert (tile, cut.value) == (64, 4)


# m, n, k -> the fastest as timed (us at tile, cut = 64, 1 / 64, 2 / 64, 4 / 128, 2 / 128, 4 where they apply), around the rule's lines
@pytest.mark.parametrize("m,n,k,want", [
    (100, 64 * 33, 4096, (64, 4)),   # 11.5 / 8.0 / 6.8
    (100, 64 * 34, 4096, (64, 2)),   # 11.5 / 8.0 / 12.1
    (100, 64 * 37, 8192, (128, 4)),  # 20.4 / 12.2 / 16.5 / - / 10.9
    (100, 64 * 74, 2048, (64, 2)),   # 7.2 / 6.3
    (100, 128 * 74, 4096, (128, 2)),  # whole 12.9, cut 10.5
    (16, 512, 4096, (64, 4)),        # 11.3 / 8.0 / 6.6 / 9.5 / 8.0
    (16, 512, 1024, (64, 1)),        # 4.7 / 5.2 / 5.3
    (333, 1792, 4096, (128, 2)),     # 12.5 / - / - / 10.5
])
def test_timed_choices(lib, m, n, k, want):
    assert _plan(lib, m, n, k) == want


def test_short_sums_stay_whole(lib):
    assert _plan(lib, 16, 512, 11 * 128)[1] == 1 and _plan(lib, 16, 512, 16 * 128)[1] > 1


# us on CTA pairs / in 128 columns: many waves of a short sum are the gaps between tiles
@pytest.mark.parametrize("m,n,k", [(8192, 4096, 128),   # 15.7 / 24.2
                                   (5612, 3904, 256),   # 14.5 / 20.0
                                   (3589, 3384, 512),   # 14.4 / 16.0
                                   (8192, 1024, 128)])  # 7.1 / 8.2
def test_many_short_sums_run_on_pairs(lib, m, n, k):
    assert _plan(lib, m, n, k) == (0, 1)
