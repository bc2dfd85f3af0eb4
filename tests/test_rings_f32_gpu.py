"""FP32 ring transforms (mixed-precision plans) at the ring lengths where the code changes -- every first
radix, both work-length launches (up to 16384-point convolutions), rings much shorter than the band limit,
transforms that leave part of a CTA idle -- against the FP64 plan, and the weighted round trip against its
parts.

Tolerance 2e-5 (max-norm): the aliases of one Fourier index are at most 150 FP32 terms added one by one
(150 2^-24 = 9e-6); the Legendre sums (2^-22 per product) and 14 FFT stages of 2^-24 stay below 1e-6 each.
"""
import math

import pytest

TOL = 2e-5


@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax,batch", [(1, 40, 2), (3, 40, 3), (7, 100, 1), (8, 300, 9), (48, 143, 5),
                                              (96, 287, 2), (512, 20, 10), (600, 50, 1), (1024, 20, 1), (2048, 20, 1)])
@pytest.mark.parametrize("spin", [0, 2])
def test_ring_lengths_vs_fp64(nside, lmax, batch, spin):
    import torch
    from polyspec_b200.sht import SHTPlan
    try:
        ref = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    except Exception:
        ref = None  # FP64 work arrays of 16384 points do not fit: adjointness instead
    mx = SHTPlan(nside, lmax, spins=(0, spin), prec="mixed", autotune=False)
    g = torch.Generator(device="cuda").manual_seed(nside + lmax + spin)
    nc = () if spin == 0 else (2,)
    alm = torch.randn((batch,) + nc + (mx.nalm,), dtype=torch.complex128, device="cuda", generator=g)
    alm[..., :lmax + 1] = alm[..., :lmax + 1].real.to(torch.complex128)  # m = 0
    mp = torch.randn((batch,) + nc + (mx.npix,), dtype=torch.float64, device="cuda", generator=g)
    x, y = mx.synthesis(alm, spin), mx.adjoint(mp, spin)
    assert mx.error_flag() == 0
    if ref is not None:
        for got, want in ((x, ref.synthesis(alm, spin)), (y, ref.adjoint(mp, spin))):
            assert float((got - want).abs().max() / want.abs().max()) < TOL
    else:
        w = torch.full((mx.nalm,), 2.0, dtype=torch.float64, device="cuda")
        w[:lmax + 1] = 1.0
        a, b = float((x * mp).sum()), float(((y * alm.conj()).real * w).sum())
        assert abs(a - b) < TOL * math.sqrt(float((x * x).sum()) * float((mp * mp).sum()))
    if mx.has_table(spin) and spin == 0:
        wt = torch.rand((1, mx.npix), dtype=torch.float64, device="cuda", generator=g)
        rt = mx.weighted_roundtrip(alm[:, None].contiguous(), wt)[:, 0]
        want = mx.adjoint(x * wt, 0)
        assert float((rt - want).abs().max() / want.abs().max()) < TOL
