"""Batched FP64 Legendre stage (FP64 MMA, several maps per tile) against the same maps transformed one by
one: groups of every width and remainder, l chunks and their remainders, lmax below the spin, several
passes over the rings; maps 20 decades apart do not touch each other, and a map that is not finite
leaves the others alone.

Tolerance 1e-12 (max-norm of each map): both sides sum at most 600 products of the same values, in
different orders, each rounded to 2^-53.
"""
import numpy as np
import pytest

TOL = 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax,batch", [(1, 2, 4), (8, 15, 5), (16, 16, 12), (32, 47, 13), (64, 32, 2),
                                              (100, 299, 6), (128, 129, 9), (256, 600, 3), (512, 33, 25)])
@pytest.mark.parametrize("spin", [0, 1, 2])
def test_batch_equals_single_maps(nside, lmax, batch, spin):
    import torch
    from polyspec_b200.sht import SHTPlan
    plan = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    g = torch.Generator(device="cuda").manual_seed(nside + batch + spin)
    nc = () if spin == 0 else (2,)
    scale = torch.logspace(-10, 10, batch, dtype=torch.float64, device="cuda").reshape((batch,) + (1,) * (len(nc) + 1))
    alm = scale * torch.randn((batch,) + nc + (plan.nalm,), dtype=torch.complex128, device="cuda", generator=g)
    mp = scale * torch.randn((batch,) + nc + (plan.npix,), dtype=torch.float64, device="cuda", generator=g)
    for x, call in ((alm, plan.synthesis), (mp, plan.adjoint)):
        got = call(x, spin)
        for b in range(batch):
            ref = call(x[b:b + 1], spin)[0]
            assert float((got[b] - ref).abs().max() / ref.abs().max()) < TOL, (call.__name__, b)
        bad = x.clone()
        bad[1].reshape(-1)[-1] = float("nan")
        out = call(bad, spin)
        out = torch.view_as_real(out) if out.is_complex() else out
        fine = torch.isfinite(out).reshape(batch, -1)
        assert not bool(fine[1].any()) and bool(fine[torch.arange(batch) != 1].all()), call.__name__
