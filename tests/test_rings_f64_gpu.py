"""FP64 ring transforms against the FP64 oracle at the ring lengths where the code changes: every first
radix and both work-length launches (equators of 4 Nside pixels, power of two or not, up to 8192-point
convolutions), rings much shorter than the band limit (aliases shared by threads or summed in loops) and
transforms that leave part of a CTA idle.

Tolerance 1e-11 (max-norm): the Legendre sums dominate (at most 300 terms and steps, amplification below
100, rounding 2^-53); a transform of 8192 points adds 13 stages of 2^-53.
"""
import numpy as np
import pytest

from oracle import sht as osht

TOL = 1e-11


@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax,batch", [(1, 40, 2), (3, 40, 3), (7, 100, 1), (8, 300, 1), (48, 143, 5),
                                              (96, 287, 2), (512, 20, 1), (600, 50, 1), (1000, 20, 2), (1024, 20, 1)])
@pytest.mark.parametrize("spin", [0, 2])
def test_ring_lengths_vs_oracle(nside, lmax, batch, spin):
    import torch
    from polyspec_b200.sht import SHTPlan
    rng = np.random.default_rng(nside + lmax)
    nc = 1 if spin == 0 else 2
    l, m = osht.getlm(lmax)
    alm = rng.normal(size=(batch, nc, len(l))) + 1j * rng.normal(size=(batch, nc, len(l)))
    alm[..., m == 0] = alm[..., m == 0].real
    alm[..., l < spin] = 0
    plan = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    ref = osht.synthesis(alm, lmax, spin, nside)
    out = plan.synthesis(torch.from_numpy(alm if spin else alm[:, 0]).cuda(), spin).cpu().numpy()
    assert np.abs(out.reshape(ref.shape) - ref).max() / np.abs(ref).max() < TOL
    mp = rng.normal(size=ref.shape)
    ref = osht.adjoint_synthesis(mp, lmax, spin, nside)
    got = plan.adjoint(torch.from_numpy(mp if spin else mp[:, 0]).cuda(), spin).cpu().numpy()
    assert np.abs(got.reshape(ref.shape) - ref).max() / np.abs(ref).max() < TOL
