"""Block-scaled fp8 GEMM with the sum over K shared by the CTAs of a cluster."""
import ctypes

import pytest
import torch

import flagcx_b200


def _plan(m, n, k, sms=148):
    lib = ctypes.CDLL(flagcx_b200.native().__file__)
    cut = ctypes.c_int()
    return lib.fcxGemmFp8Plan(m, n, k, sms, ctypes.byref(cut)), cut.value


def test_plan_leaves_no_stretch_empty_and_one_wave():
    cdiv = lambda a, b: -(-a // b)  # noqa: E731
    seen = set()
    for m in (1, 16, 129, 333, 1024, 8192):
        for n in (8, 72, 512, 1792, 4096):
            for nk in list(range(1, 40)) + [64, 224]:
                tile, cut = _plan(m, n, nk * 128)
                seen.add((tile, cut))
                assert tile in (0, 64, 128) and cut in (1, 2, 4)
                if cut > 1:
                    assert tile and (cut - 1) * cdiv(nk, cut) < nk and cdiv(m, 128) * cdiv(n, tile) * cut <= 148
    assert {(0, 1), (64, 1), (64, 2), (64, 4), (128, 2)} <= seen
    assert _plan(333, 1792, 4096) == (128, 2) and _plan(16, 512, 4096) == (64, 4) and _plan(16, 512, 1024) == (64, 1)


@pytest.mark.gpu
@pytest.mark.parametrize("m,n,k,cut", [(1, 8, 1536, 4), (16, 512, 4096, 4), (100, 4096, 4096, 2), (129, 1000, 1664, 4), (333, 1792, 4096, 2),
                                       (640, 1032, 4352, 2), (128, 2048, 2048, 4)])
def test_cut_sums_match_float64(m, n, k, cut):
    """One rounding to bf16 of an fp32 sum of k products (the slices' and the stretches' sums in any order)."""
    nat = flagcx_b200.native()
    assert _plan(m, n, k)[1] == cut
    g = torch.Generator(device="cuda").manual_seed(m + n)
    x, w = torch.randn(m, k, generator=g, device="cuda").bfloat16(), torch.randn(n, k, generator=g, device="cuda").bfloat16()
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    q, sa = nat.quant_fp8_act(x)
    wq, sb = nat.quant_fp8_weight(w)
    y = nat.gemm_fp8_nt(q, sa, wq, sb, err)
    a = q.double().view(m, k // 128, 128) * sa.t().double()[:, :, None]
    b = wq.double().view(n, k // 128, 128) * sb.double().repeat_interleave(128, 0)[:n, :, None]
    a, b = a.reshape(m, k), b.reshape(n, k)
    ref = a @ b.t()
    bound = 2.0 ** -8 * ref.abs() + k * 2.0 ** -23 * (a.abs() @ b.abs().t()) + 1e-30
    assert ((y.double() - ref).abs() <= bound).all() and int(err) == 0
    assert torch.equal(y, nat.gemm_fp8_nt(q, sa, wq, sb, err))
