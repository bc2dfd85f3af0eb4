"""The single-system CG step (ps_cgd_*) against the same operations in torch; lengths below, at and above a block and
beyond the largest grid, twice in a row on one workspace (the arrival counter has to return to zero)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf", [1, 3])
@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 5000, 256 * 1024 + 3])
@pytest.mark.parametrize("harmonic", [True, False])
def test_step(nf, n, harmonic):
    from polyspec_b200 import lmops
    g = torch.Generator(device="cuda").manual_seed(n)
    vec = lambda: torch.randn((nf, n), dtype=torch.complex128, device="cuda", generator=g)  # noqa: E731
    mat = lambda: torch.randn((nf, nf, n), dtype=torch.float64, device="cuda", generator=g)  # noqa: E731
    S, Sig = mat(), mat()
    beam, w = mat()[0], mat()[0, 0].abs()
    p, x, r = vec(), vec(), vec()
    rz = 0.7
    sc = lmops.StepScalars(rz, p.device)
    mul = lambda M, v: torch.einsum('abi,bi->ai', M.to(v.dtype), v)  # noqa: E731

    def dot(a, b):  # and what rounding may leave of the sum: its tree is some 30 terms deep
        t = (a * b.conj()).real * w
        return float(t.sum()), 1e-14 * float(((a.abs() * b.abs()) * w).sum())
    beam_p = torch.empty_like(p)
    for _ in range(2):
        y = vec()
        q = beam * y + mul(S, p)
        sc.apply(S, beam, w, p, y)
        assert (y - q).abs().max() <= 1e-14 * float(q.abs().max() + nf * S.abs().max() * p.abs().max())
        pq, tol = dot(p, y)
        assert abs(sc.rz_pq()[1] - pq) <= tol
        alpha = rz / sc.rz_pq()[1]
        x1, r1 = x + alpha * p, r - alpha * y
        z = torch.empty_like(r)
        if harmonic:
            sc.update(Sig, w, p, y, x, r, z)
            assert (z - mul(Sig, r)).abs().max() <= 1e-14 * float(nf * Sig.abs().max() * r.abs().max())
        else:
            sc.update(None, w, p, y, x, r, None)
            z = vec()
            sc.next_rz(w, r, z)
        assert (x - x1).abs().max() <= 1e-15 * float(x1.abs().max() + abs(alpha) * p.abs().max()) * 2
        assert (r - r1).abs().max() <= 1e-15 * float(r1.abs().max() + abs(alpha) * y.abs().max()) * 2
        new, tol = dot(r, z)
        assert abs(sc.rz_pq()[0] - new) <= tol
        beta, rz = sc.rz_pq()[0] / rz, sc.rz_pq()[0]
        p1 = z + beta * p
        sc.direction(beam, z, p, beam_p)
        assert (p - p1).abs().max() <= 1e-15 * float(z.abs().max() + abs(beta) * p1.abs().max()) * 4
        assert torch.equal(beam_p, beam * p)


def test_arguments_are_checked():
    from polyspec_b200 import _lib
    t = torch.zeros(64, dtype=torch.complex128, device="cuda")
    v = t.data_ptr()
    L = _lib.lib()
    assert L.ps_cgd_apply(v, v, v, v, v, 3, 1, v, v, 1 << 20, None) == -1  # in place over p
    assert L.ps_cgd_direction(v, v, v, v, 2, 1, v, None) == -1  # two fields
    assert L.ps_cgd_rz(v, v, v, 1, 1, v, v, 8, None) == -5  # workspace
