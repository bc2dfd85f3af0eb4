"""Scalar alm to (+s, -s) complex maps and back (ps_synthesis_pm, ps_adjoint_pm) against the (G, C) and (Q, U)
transforms and the recombinations they replace; map counts at the edges of the matrix tiles, ring counts at those of a
warp and a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("nside,lmax", [(4, 7), (16, 37), (64, 100), (96, 127)])
@pytest.mark.parametrize("spin", [1, 2, 3])
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 8, 9, 13])
def test_pairs_match_general_transforms(prec, nside, lmax, spin, batch):
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(nside, lmax, spins=(spin,), prec=prec, autotune=False)
    g = torch.Generator(device="cuda").manual_seed(nside + batch)
    a = torch.randn((batch, P.nalm), dtype=torch.complex128, device="cuda", generator=g)
    qu = P.synthesis(torch.stack([-a, torch.zeros_like(a)], 1), spin)
    plus, minus = P.synthesis_pm(a, spin)
    v = torch.randn((2, batch, P.npix), dtype=torch.complex128, device="cuda", generator=g)
    gc = P.adjoint(torch.stack([(v[0] + v[1]).real / 2, (v[0] - v[1]).imag / 2], 1), spin, 0.5)
    lp, lm = P.adjoint_pm(v[0], v[1], spin, 0.5)
    ref_p, ref_m = -(gc[:, 0] + 1j * gc[:, 1]), -(-1) ** spin * (gc[:, 0] - 1j * gc[:, 1])
    # mixed: the same kernels on the same numbers.  FP64: sums of about lmax rounded terms in another order
    tol = 0.0 if prec == "mixed" else 1e-14 * lmax
    scale = qu.abs().max()
    assert (torch.complex(qu[:, 0], qu[:, 1]) - plus).abs().max() <= tol * scale
    assert torch.equal(minus, plus.conj().resolve_conj())
    assert (ref_p - lp).abs().max() == 0 and (ref_m - lm).abs().max() == 0


@pytest.mark.parametrize("batch", [1, 5])
def test_nonfinite_alm_reaches_every_ring(batch):
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(16, 40, spins=(2,), autotune=False)
    a = torch.ones((batch, P.nalm), dtype=torch.complex128, device="cuda")
    for i in (0, 1, 30):  # l = 0 and 1 do not enter a spin-2 map but for their infinities
        b = a.clone()
        b[-1, i] = float("nan")
        plus, minus = P.synthesis_pm(b, 2)
        assert torch.isnan(plus[-1].real).all() and torch.isnan(minus[-1].imag).all()
        assert batch == 1 or torch.isfinite(plus[:-1].real).all()


def test_shapes_are_checked():
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(8, 10, spins=(1,), autotune=False)
    v = torch.zeros((2, P.npix), dtype=torch.complex128, device="cuda")
    with pytest.raises(ValueError):
        P.adjoint_pm(v[0], v[1], 1)
    with pytest.raises(ValueError):
        P.adjoint_pm(v, v[:1], 1)
    with pytest.raises(ValueError):
        P.synthesis_pm(torch.zeros(P.nalm, dtype=torch.complex128, device="cuda"), 1)
