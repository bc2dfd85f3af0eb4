"""FP64 Legendre stage against the FP64 oracle where its kernels switch shape: rings per thread and
warps per CTA by the number of rings and (m, map) pairs, several passes over l (Rh above one CTA's
rings), l chunks and their remainders, maps per CTA and their remainders, lmax below the spin, orders
whose seeds underflow near the poles; and non-finite inputs, which reach every output.

Tolerance 1e-11 (max-norm): at most 1000 recurrence steps and as many terms per sum, each rounded to
2^-53, with an amplification of the recurrence below 100.
"""
import numpy as np
import pytest

from oracle import sht as osht

TOL = 1e-11


def relerr(x, ref):
    return np.abs(x - ref).max() / max(np.abs(ref).max(), 1e-300)


@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax,batch", [(1, 1, 1), (2, 3, 2), (16, 31, 1), (16, 32, 4), (32, 33, 5), (33, 64, 1),
                                              (64, 95, 2), (128, 129, 7), (129, 65, 1), (130, 300, 1), (256, 767, 1),
                                              (300, 63, 3), (512, 96, 1), (512, 40, 40), (1024, 33, 1)])
@pytest.mark.parametrize("spin", [0, 1, 2, 3])
def test_kernel_shapes_vs_oracle(nside, lmax, batch, spin):
    import torch
    from polyspec_b200.sht import SHTPlan
    rng = np.random.default_rng(100 * nside + lmax + spin)
    nc = 1 if spin == 0 else 2
    l, m = osht.getlm(lmax)
    alm = rng.normal(size=(batch, nc, len(l))) + 1j * rng.normal(size=(batch, nc, len(l)))
    alm[..., m == 0] = alm[..., m == 0].real
    plan = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    a_t = torch.from_numpy(alm if spin else alm[:, 0]).cuda()
    out = plan.synthesis(a_t, spin).cpu().numpy().reshape(batch, nc, -1)
    alm[..., l < spin] = 0  # they have no harmonic
    assert relerr(out, osht.synthesis(alm, lmax, spin, nside)) < TOL
    mp = rng.normal(size=(batch, nc, 12 * nside * nside))
    got = plan.adjoint(torch.from_numpy(mp if spin else mp[:, 0]).cuda(), spin, scale=0.5).cpu().numpy()
    assert relerr(got.reshape(batch, nc, -1), 0.5 * osht.adjoint_synthesis(mp, lmax, spin, nside)) < TOL


@pytest.mark.gpu
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_non_finite_inputs_reach_every_output(spin, value):
    """A high (l, m) coefficient and a polar pixel: most rings never see that order above rounding."""
    import torch
    from polyspec_b200.sht import SHTPlan
    nside, lmax = 256, 700
    plan = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    nc = 1 if spin == 0 else 2
    alm = torch.zeros((1, nc, plan.nalm), dtype=torch.complex128, device="cuda")
    alm[0, 0, -1] = complex(value, 0.0)
    out = plan.synthesis(alm if spin else alm[:, 0], spin)
    assert not bool(torch.isfinite(out).any())
    mp = torch.zeros((1, nc, plan.npix), dtype=torch.float64, device="cuda")
    mp[0, 0, 0] = value
    got = plan.adjoint(mp if spin else mp[:, 0], spin)
    assert not bool(torch.isfinite(torch.view_as_real(got)).all(-1).any())
