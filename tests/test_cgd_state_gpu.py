"""State of the single-map CG: a finished solve holds its vectors and no more, and vectors and rz that a program sets
between steps (a restart, another start vector) are the ones the next step uses.

Tolerance 1e-12 (max-norm): one step of the same FP64 products and sums in another order.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solver(nside, lmax, preconditioner="harmonic"):
    from polyspec_b200 import PolySpec, Weightings
    from polyspec_b200 import workloads as W
    from polyspec_b200.weighting import CGD
    cl, cltot, beam, mask, noise, _ = W.cg_fisher_setup(nside, lmax, n_holes=10)
    base = PolySpec(nside, dict(cltot), beam=list(beam), pol=True, lmax=lmax)
    wts = Weightings(base, mask, dict(cl), noise_cov=noise)
    d = torch.randn((3, base.Npix), dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(1))
    return wts, d, lambda: CGD(wts, d, preconditioner=preconditioner)


def test_finished_solve_holds_its_vectors():
    wts, d, make = _solver(32, 95)
    make().run(nstep=1, thresh=0.0)  # tables of the base and the plan's workspace are there afterwards
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    cg = make()
    cg.run(nstep=3, thresh=0.0)
    vec = (cg.x.numel() * cg.x.element_size() + 511) // 512 * 512
    assert torch.cuda.memory_allocated() - before <= 3 * vec  # x, r, p


def _step(cg, x, r, p, rz):
    """One step in torch: (x, r, p, rz) after it."""
    q = cg._apply_A(p)
    alpha = rz / cg.dot(p, q)
    x, r = x + alpha * p, r - alpha * q
    z = cg._apply_M(r)
    rz1 = cg.dot(r, z)
    return x, r, z + rz1 / rz * p, rz1


@pytest.mark.parametrize("preconditioner", ["harmonic", "pseudo_inverse"])
@pytest.mark.parametrize("what", ["nothing", "direction", "scaled", "all", "layout", "aliased", "after run"])
def test_state_set_between_steps(preconditioner, what):
    _, _, make = _solver(16, 32, preconditioner)
    cg = make()
    if what == "after run":
        cg.run(nstep=2, thresh=0.0)
    else:
        cg.step()
        cg.step()
    if what == "direction":  # restart
        cg.p = cg._apply_M(cg.r)
        cg.rz = cg.dot(cg.r, cg.p)
    elif what == "scaled":
        cg.p *= 2.0
    elif what == "all":
        cg.x, cg.r = cg.x * 0.5, cg.r * 2.0
        cg.p = cg._apply_M(cg.r)
        cg.rz = cg.dot(cg.r, cg.p)
    elif what == "layout":
        cg.x, cg.r = cg.x.t().contiguous().t(), cg.r.conj().resolve_conj().conj()
        cg.p = cg.p.t().contiguous().t()
    elif what == "aliased":
        cg.p = cg.r
        cg.rz = cg.dot(cg.r, cg.r)
    want = _step(cg, cg.x.clone(), cg.r.clone(), cg.p.clone(), cg.rz)
    cg.step()
    for got, ref in zip((cg.x, cg.r, cg.p), want):
        assert float((got - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
    assert abs(cg.rz - want[3]) <= 1e-12 * abs(want[3])
