"""A CG step whose p^T A p or r^T z is zero has no alpha or beta: the vectors stay as they were, to the bit, and the solve
goes on from them; CGD raises ZeroDivisionError with its last iterate intact."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,n", [(1, 1), (3, 257), (3, 256 * 1024 + 3)])
@pytest.mark.parametrize("harmonic", [True, False])
@pytest.mark.parametrize("zero", ["pq", "rz"])
def test_vectors_stay(nf, n, harmonic, zero):
    from polyspec_b200 import lmops
    g = torch.Generator(device="cuda").manual_seed(n)
    vec = lambda: torch.randn((nf, n), dtype=torch.complex128, device="cuda", generator=g)  # noqa: E731
    S = torch.eye(nf, dtype=torch.float64, device="cuda")[:, :, None].expand(nf, nf, n).contiguous()
    beam, w = torch.ones((nf, n)).double().cuda(), torch.ones(n).double().cuda()
    x, r, z, beam_p = vec(), vec(), vec(), vec()
    p = vec() if zero == "rz" else torch.zeros_like(x)
    sc = lmops.StepScalars(0.0 if zero == "rz" else 1.0, p.device)

    def step():
        y = torch.zeros_like(p)
        sc.apply(S, beam, w, p, y)
        if harmonic:
            sc.update(S, w, p, y, x, r, z)
        else:
            sc.update(None, w, p, y, x, r, None)
            sc.next_rz(w, r, z)
        sc.direction(beam, z, p, beam_p)
    before = [t.clone() for t in (x, r, z, p, beam_p)]
    step()
    assert all(torch.equal(a, b) for a, b in zip(before, (x, r, z, p, beam_p)))
    rz, pq = sc.rz_pq()
    assert (pq == 0.0 and rz == 1.0) if zero == "pq" else (rz == 0.0 and pq > 0.0)
    p.copy_(vec())
    sc.t[0] = 1.0
    alpha_p = p / float(p.abs().square().sum())
    x0 = x + alpha_p
    step()  # with both set it is a step again; the sum's tree is some 30 terms deep
    assert float((x - x0).abs().max()) <= 1e-14 * float(alpha_p.abs().max()) + 4e-16 * float(x0.abs().max())
    assert torch.equal(beam_p, p) and not torch.equal(beam_p, before[4])


@pytest.mark.parametrize("preconditioner", ["harmonic", "pseudo_inverse"])
def test_solver_keeps_its_iterate(preconditioner):
    from polyspec_b200 import PolySpec, Weightings
    from polyspec_b200 import workloads as W
    from polyspec_b200.weighting import CGD
    nside, lmax = 16, 32
    cl, cltot, beam, mask, noise, _ = W.cg_fisher_setup(nside, lmax, n_holes=10)
    base = PolySpec(nside, dict(cltot), beam=list(beam), pol=True, lmax=lmax)
    wts = Weightings(base, mask, dict(cl), noise_cov=noise)
    d = torch.randn((3, base.Npix), dtype=torch.float64, device="cuda",
                    generator=torch.Generator(device="cuda").manual_seed(1))
    x0 = torch.einsum('abi,bi->ai', wts.d_x0op, base.to_lm(d))
    b = CGD(wts, d, preconditioner=preconditioner)._apply_A(x0)
    cg = CGD(wts, [], x0=x0, test_b=b, preconditioner=preconditioner)  # solved from the start: r = z = p = 0
    assert cg.rz == 0 and not cg.p.any()
    for _ in range(2):
        with pytest.raises(ZeroDivisionError):
            cg.step()
        assert torch.equal(cg.get_wiener_lm(), x0) and not cg.r.any() and not cg.p.any() and cg.i == 0
