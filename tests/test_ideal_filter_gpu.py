"""The ideal filter of a batch of maps against the filter of each map, at the full band limit (per-(l, m) product kernel)
and below it, and transforms into a given tensor.

Tolerance 1e-12 (max-norm): both sides are FP64 transforms of the same maps, whose sums of a few hundred products are
ordered differently, and the same three products per coefficient.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax,batch", [(4, 7, 1), (16, 40, 3), (32, 95, 7)])
@pytest.mark.parametrize("low", [False, True])
@pytest.mark.parametrize("pol", [False, True])
def test_batched_equals_single(nside, lmax, batch, low, pol):
    from polyspec_b200 import PolySpec, Weightings
    from polyspec_b200 import workloads as W
    cl = W.fiducial_cl(3 * nside - 1, True)
    cl = dict(cl) if pol else {'TT': cl['TT']}
    nf = 3 if pol else 1
    beam = [W.gaussian_beam(3 * nside - 1, 300.)] * nf
    base = PolySpec(nside, cl, beam=beam if pol else beam[0], pol=pol, lmax=lmax)
    wts = Weightings(base, np.ones((nf, 12 * nside ** 2)), cl, noise_cov=W.white_noise_cov(nside)[:nf])
    g = torch.Generator(device="cuda").manual_seed(nside)
    maps = torch.randn((batch, nf, 12 * nside ** 2), dtype=torch.float64, device="cuda", generator=g)
    top = lmax - 2 if low else lmax
    got = wts.batched_applySinv_ideal(maps, lmax=top)
    for b in range(batch):
        ref = wts.applySinv_ideal(maps[b], lmax=top)
        assert got[b].shape == ref.shape
        assert float((got[b] - ref).abs().max() / ref.abs().max()) < 1e-12
    assert tuple(wts.batched_applySinv_ideal(maps[:0], lmax=top).shape) == (0,) + tuple(got.shape[1:])


def test_adjoint_into():
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(8, 20, spins=(0, 2), autotune=False)
    g = torch.Generator(device="cuda").manual_seed(1)
    m = torch.randn((5, 2, P.npix), dtype=torch.float64, device="cuda", generator=g)
    buf = torch.zeros((7, 2, P.nalm), dtype=torch.complex128, device="cuda")
    assert P.adjoint(m, 2, 0.5, out=buf[1:6]).data_ptr() == buf[1].data_ptr()
    assert torch.equal(buf[1:6], P.adjoint(m, 2, 0.5)) and not buf[0].any() and not buf[6].any()
    for bad in (buf[:5, :1], buf[:5].real, buf.transpose(0, 1)[:, :5].transpose(0, 1).contiguous().conj(), buf[:4]):
        with pytest.raises(ValueError):
            P.adjoint(m, 2, out=bad)
