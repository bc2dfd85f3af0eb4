"""Beams of other types than float64: the per-(l, m) beam on the device is float64 (or complex), the CG step's kernels
refuse operands of another type, shape or layout, and the filters give what the same beam gives in float64.

Tolerances: operands and operations of the real types are the same to the last bit.  The complex beam takes the CG step
through other sums: three steps of it agree to 1e-10 like those of the native and the batched CG; the ideal filter
differs by the order of three products (1e-12).
"""
import types

import numpy as np
import pytest
import torch


@pytest.mark.parametrize("dtype", [np.float32, np.float16, np.int64, np.float64])
def test_device_beam_is_float64(dtype):
    from polyspec_b200 import PolySpec
    beam = np.asarray([[3, 2, 1, 1, 1, 1]], dtype=dtype)
    base = types.SimpleNamespace(lmax=2, l_arr=np.asarray([0, 1, 2, 1, 2, 2]), beam_lm=beam, device="cpu",
                                 _dev_cache={})
    t = PolySpec.dev(base, 'beam_lm')
    assert t.dtype == torch.float64 and np.array_equal(t.numpy(), beam)


def test_step_refuses_other_operands():
    from polyspec_b200 import lmops
    n = 6
    vec = lambda: torch.zeros((3, n), dtype=torch.complex128)  # noqa: E731
    mat, beam, w = torch.zeros((3, 3, n)).double(), torch.zeros((3, n)).double(), torch.zeros(n).double()
    sc = lmops.StepScalars(1.0, "cpu")
    for bad in (beam.float(), beam.long(), vec(), beam[:, :4], torch.zeros((n, 3)).double().t()):
        with pytest.raises(ValueError):
            sc.apply(mat, bad, w, vec(), vec())
        with pytest.raises(ValueError):
            sc.direction(bad, vec(), vec(), vec())
    for bad in (vec().to(torch.complex64), vec()[:, :5], vec().conj(), torch.zeros((n, 3)).cdouble().t()):
        with pytest.raises(ValueError):
            sc.update(mat, w, vec(), vec(), bad, vec(), vec())
        with pytest.raises(ValueError):
            sc.next_rz(w, vec(), bad)
    with pytest.raises(ValueError):
        sc.update(mat.float(), w, vec(), vec(), vec(), vec(), vec())
    with pytest.raises(ValueError):
        sc.next_rz(w.float(), vec(), vec())


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["float32", "int", "complex", "default"])
@pytest.mark.parametrize("pol", [True, False])
def test_filters(kind, pol):
    from polyspec_b200 import PolySpec, Weightings
    from polyspec_b200 import workloads as W
    nside, lmax = 16, 32
    cl, cltot, beam, mask, noise, _ = W.cg_fisher_setup(nside, lmax, n_holes=10)
    nf = 3 if pol else 1
    beam = np.asarray(beam)[:nf]
    beam = {"float32": beam.astype(np.float32), "int": np.ones(beam.shape, dtype=np.int64),
            "complex": beam.astype(np.complex128), "default": np.ones(beam.shape)}[kind]
    tot = dict(cltot) if pol else {'TT': cltot['TT']}
    if kind == "default":  # the beam of ones takes the spectrum's type
        tot = {k: v.astype(np.float32) for k, v in tot.items()}
    cl = dict(cl) if pol else {'TT': cl['TT']}
    maps = torch.randn((2, nf, 12 * nside ** 2), dtype=torch.float64, device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(3))
    out = []
    for b in (beam, beam.real.astype(np.float64)):
        args = [] if kind == "default" and b is beam else list(b) if pol else b[0]
        base = PolySpec(nside, dict(tot), beam=args, pol=pol, lmax=lmax)
        wts = Weightings(base, mask[:nf], dict(cl), noise_cov=noise[:nf])
        out.append([wts.applySinv_optimal(maps[0], preconditioner="harmonic", nstep=3, thresh=0.0),
                    wts.applySinv_optimal(maps[0], preconditioner="pseudo_inverse", nstep=3, thresh=0.0),
                    wts.batched_applySinv_ideal(maps)])
    for got, want, tol in zip(out[0], out[1], (1e-10, 1e-10, 1e-12)):
        assert float((got - want).abs().max() / want.abs().max()) <= (tol if kind == "complex" else 0.0)
