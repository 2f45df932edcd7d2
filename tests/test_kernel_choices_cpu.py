"""Host-side rules that pick a kernel or a tile, checked without a GPU: every rule gives a legal answer over its whole
range, and picks the variant that each side of its line was measured for."""
import ctypes
import math
import random

import pytest


@pytest.fixture(scope="module")
def ext():
    import flagcx_b200
    lib = ctypes.CDLL(flagcx_b200.native().__file__)
    lib.fcxGemmTileCost.restype = ctypes.c_double
    lib.fcxGemmTileCost.argtypes = [ctypes.c_int] * 4 + [ctypes.POINTER(ctypes.c_int)]
    lib.fcxGemmPairCost.restype = ctypes.c_double
    lib.fcxGemmFp8Tile.restype = ctypes.c_int
    lib.fcxMoeTileColumns.restype = ctypes.c_int
    lib.fcxGemmDualPlan.restype = lib.fcxGemmUnitsCovered.restype = ctypes.c_int
    return lib


def _width(ext, m, n, k):
    bn = ctypes.c_int(0)
    cost = ext.fcxGemmTileCost(m, n, k, 148, ctypes.byref(bn))
    assert cost > 0
    return bn.value


def test_gemm_tile_width(ext):
    for m in (1, 64, 128, 129, 1000, 8192):
        for n in (8, 64, 72, 256, 1000, 4096):
            for k in (8, 64, 1000, 8192):
                assert _width(ext, m, n, k) in (64, 128, 256)
    assert _width(ext, 8192, 4096, 4096) == 256  # enough tiles for every SM
    assert _width(ext, 64, 3072, 1024) == 64     # 12 tiles of 256 columns: 12 of 148 SMs


def test_uncut_sums_get_the_kernel_that_is_fastest_uncut(ext):
    """A launch that keeps K whole (one-rank tensor parallel, all-gather GEMM, the plain NT form) is priced without a cut: what
    it gets is within the rule's own margin (the pair kernel has to win by 15 %) of the cheapest kernel and tile."""
    ext.fcxGemmTileCostCut.restype = ctypes.c_double
    ext.fcxGemmPairSuitsCut.restype = ctypes.c_int
    few_rows = [(512, 1024, 4096), (256, 1024, 4096), (256, 2048, 2048), (256, 4096, 4096), (512, 2048, 4096), (1024, 1024, 4096), (384, 2048, 2048)]
    rest = [(m, n, k) for m in (64, 128, 640, 2328, 8192) for n in (64, 200, 1792, 4096) for k in (64, 1000, 4096)]
    for m, n, k in few_rows + rest:
        def uncut(rows, cols, slots, clocks):
            return -(-(-(-m // rows) * -(-n // cols)) // slots) * -(-k // 64) * clocks
        costs = {64: uncut(128, 64, 148, 384), 128: uncut(128, 128, 148, 512), 256: uncut(128, 256, 148, 768), "pair": uncut(256, 256, 74, 512)}
        bn = ctypes.c_int(0)
        tile = ext.fcxGemmTileCostCut(m, n, k, 148, 1, ctypes.byref(bn))
        assert tile == costs[bn.value]
        chosen = "pair" if ext.fcxGemmPairSuitsCut(m, n, k, 1) else bn.value
        least = min(costs.values()) if m >= 129 else min(v for c, v in costs.items() if c != "pair")
        assert costs[chosen] <= least / 0.85 + 1e-6, ((m, n, k), chosen, costs)


def test_no_choice_of_kernel_cuts_a_sum_finer(ext):
    """Every piece of K is one more rounding to bf16.  Whatever kernel and tile a size gets, it is cut into no more pieces than
    by the simple rule: CTA pairs for rows that fill their 256-row blocks to 7 %, else single CTAs of 256 columns."""
    rng = random.Random(5)
    sizes = [(288, 3392, 3832), (1072, 2368, 3592), (2376, 1280, 2960), (312, 3416, 3520), (640, 2112, 4048)]
    def size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi)))) // 8 * 8
    sizes += [(size(16, 8200), size(512, 4100), size(512, 8200)) for _ in range(20000)]
    for m, n, k in sizes:
        n_k, m1, m2 = -(-k // 64), -(-m // 128), -(-m // 256)
        if m >= 129 and m2 * 256 <= 1.07 * m and n >= 192:
            simple = ext.fcxGemmPickSplitK(0, m2 * -(-n // 256), 74, n_k, n)
        else:
            simple = ext.fcxGemmPickSplitK(0, m1 * -(-n // 256), 148, n_k, n)
        if ext.fcxGemmPairSuits(m, n, k):
            pieces = ext.fcxGemmPieces(0, m, n, k, m2 * -(-n // 256), 74, 148)
        else:
            pieces = ext.fcxGemmPieces(0, m, n, k, m1 * -(-n // _width(ext, m, n, k)), 148, 148)
        assert 1 <= pieces <= simple, (m, n, k, pieces, simple)
        assert (pieces - 1) * -(-n_k // pieces) < n_k  # the last piece is not empty
    assert ext.fcxGemmPieces(5, 288, 3392, 3832, 28, 74, 148) == 5  # a caller's own count stands


def test_fp8_tile(ext):
    for m in (1, 128, 129, 333, 8192):
        for n in (8, 64, 136, 1792, 4096):
            assert ext.fcxGemmFp8Tile(m, n, 148) in (0, 64, 128)
    # the fastest of the three at sizes on both sides of each line, as timed
    fastest = {(8192, 4096): 0, (8192, 1024): 0, (4096, 4096): 0, (2048, 4096): 0, (1024, 4096): 0, (3000, 2000): 128, (512, 4096): 128,
               (1024, 1024): 64, (333, 1792): 64, (128, 4096): 64, (64, 1024): 64}
    for (m, n), tile in fastest.items():
        assert ext.fcxGemmFp8Tile(m, n, 148) == tile, (m, n)


def test_moe_tile(ext):
    """Narrow tiles only where they were measured to be faster: as many waves, or a few more for short gate / up sums."""
    for blocks in (0, 1, 5, 74, 500):
        for cols in (8, 128, 1024, 28672):
            for k in (8, 512, 1024, 14336):
                for up in (0, 1):
                    assert ext.fcxMoeTileColumns(blocks, cols, k, up, 74) in (128, 256)
    for up in (0, 1):
        assert ext.fcxMoeTileColumns(68, 28672, 4096, up, 74) == 256
        assert ext.fcxMoeTileColumns(6, 1024, 2048, up, 74) == 128  # 24 wide or 48 narrow tiles on 74 pairs: one wave
    three_for_two = (6, 4096)  # 96 wide tiles, 192 narrow ones
    assert [ext.fcxMoeTileColumns(*three_for_two, k, 1, 74) for k in (512, 1024, 1280, 2048, 3328)] == [128, 128, 256, 256, 256]
    assert [ext.fcxMoeTileColumns(*three_for_two, k, 0, 74) for k in (512, 1024, 5632)] == [256] * 3
    five_for_three = (11, 4096)  # 176 and 352
    assert [ext.fcxMoeTileColumns(*five_for_three, k, 1, 74) for k in (512, 1024, 2560)] == [128, 256, 256]


def test_two_products_in_one_launch_cover_every_unit_once(ext):
    longest, s0, s1, swap, extra = (ctypes.c_int(0) for _ in range(5))
    for n in (1, 2, 73, 74, 148):
        for n0 in (1, 5, 48, 74, 75, 200):
            for n1 in (0, 1, 16, 74, 128, 500):
                for ex in (0, 1, 3, 8, 200):
                    workers = min(n, n0 + n1)
                    assert ext.fcxGemmUnitsCovered(workers, n0, n1, ex, 1, 1, ctypes.byref(longest)) == 1, (n, n0, n1, ex)
    # GPT-2-medium's backward GEMMs at 8192 tokens, (I, O): the launch ends within a short unit or so of a perfect split
    for i, o in ((1024, 3072), (1024, 1024), (1024, 4096), (4096, 1024)):
        uw, ux, kw, kx = (o // 256) * (i // 256), 32 * (i // 256), 128, o // 64
        alone = [ext.fcxGemmPickSplitK(0, u, 74, k, i) for u, k in ((uw, kw), (ux, kx))]
        ext.fcxGemmDualPlan(uw, kw, alone[0], ux, kx, alone[1], 74, *(ctypes.byref(v) for v in (s0, s1, swap, extra)))
        assert 1 <= s0.value <= alone[0] and 1 <= s1.value <= alone[1]
        units, lens = [uw * s0.value, ux * s1.value], [-(-kw // s0.value), -(-kx // s1.value)]
        if swap.value:
            units, lens = units[::-1], lens[::-1]
        assert ext.fcxGemmUnitsCovered(74, units[0], units[1], extra.value, lens[0], lens[1], ctypes.byref(longest)) == 1
        share = (uw * kw + ux * kx) / 74
        assert longest.value <= share + 1.5 * lens[1], (i, o, longest.value, share)
