"""Transforms of maps and alm that lie at a stride (T and (E, B) parts of [batch][3][..] arrays, padded rows) against
the same transforms of contiguous copies: the same kernels on the same numbers, so equal to the last bit."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def pad(t, gap):
    """t [B][...] as a view with `gap` unused elements after every map, and its buffer."""
    n = t[0].numel()
    buf = torch.full((t.shape[0], n + gap), float("nan"), dtype=t.dtype, device=t.device)
    buf[:, :n] = t.reshape(t.shape[0], n)
    return buf[:, :n].view(t.shape) if t.dim() == 2 else buf.as_strided(t.shape, (n + gap,) + t.stride()[1:]), buf


@pytest.mark.parametrize("prec,tables", [("fp64", False), ("mixed", True), ("mixed", False)])
@pytest.mark.parametrize("spin", [0, 1, 2])
@pytest.mark.parametrize("batch", [1, 2, 3, 5, 13])
def test_strided_equals_contiguous(prec, tables, spin, batch):
    from polyspec_b200 import _lib
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(16, 37, spins=(0, 1, 2), prec=prec, autotune=False, tables=tables)
    g = torch.Generator(device="cuda").manual_seed(batch)
    nc = (2,) if spin else ()
    alm = torch.randn((batch,) + nc + (P.nalm,), dtype=torch.complex128, device="cuda", generator=g)
    maps = torch.randn((batch,) + nc + (P.npix,), dtype=torch.float64, device="cuda", generator=g)
    ref_map, ref_alm = P.synthesis(alm, spin), P.adjoint(maps, spin, 0.5)
    for gap in (1, 6):
        (a, _), (m, _) = pad(alm, gap), pad(maps, gap)
        assert torch.equal(P.synthesis(a, spin), ref_map) and torch.equal(P.adjoint(m, spin, 0.5), ref_alm)
        (om, bm), (oa, ba) = pad(torch.zeros_like(maps), gap), pad(torch.zeros_like(alm), gap)
        P._issue_synthesis(spin, batch, a.data_ptr(), a.stride(0), om.data_ptr(), om.stride(0))
        P._issue_adjoint(spin, batch, m.data_ptr(), m.stride(0), oa.data_ptr(), oa.stride(0), 0.5)
        assert torch.equal(om, ref_map) and torch.equal(oa, ref_alm)
        assert torch.isnan(bm[:, -gap:]).all() and torch.isnan(ba[:, -gap:]).all()  # nothing written between
    # strides shorter than a map are refused
    ws, n = P.workspace(batch, spin, 0)
    rc = _lib.lib().ps_synthesis_strided(P._h, alm.data_ptr(), 1, ref_map.data_ptr(), 0, batch, spin, ws.data_ptr(), n,
                                         P._stream())
    assert rc == -1
    ws, n = P.workspace(batch, spin, 1)
    rc = _lib.lib().ps_adjoint_strided(P._h, maps.data_ptr(), 1, ref_alm.data_ptr(), 0, batch, spin,
                                       ctypes.c_double(1.0), ws.data_ptr(), n, P._stream())
    assert rc == -1


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("batch,nf", [(1, 1), (1, 3), (4, 1), (4, 3)])
def test_fields_equal_single_spins(prec, batch, nf):
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(16, 37, spins=(0, 2), prec=prec, autotune=False)
    g = torch.Generator(device="cuda").manual_seed(batch)
    wide = torch.randn((batch, 4, P.nalm), dtype=torch.complex128, device="cuda", generator=g)
    maps = torch.randn((batch, 4, P.npix), dtype=torch.float64, device="cuda", generator=g)
    for a, m in ((wide[:, :nf], maps[:, :nf]), (wide[:, :nf].contiguous(), maps[:, :nf].contiguous()),
                 (wide[:, :nf].conj(), -maps.flip(1)[:, :nf])):
        om = torch.empty((batch, nf, P.npix), dtype=torch.float64, device="cuda")
        oa = torch.empty((batch, nf, P.nalm), dtype=torch.complex128, device="cuda")
        P.synthesis_fields(a, om)
        P.adjoint_fields(m, oa, 0.5)
        assert torch.equal(om[:, 0], P.synthesis(a[:, 0].clone(), 0))
        assert torch.equal(oa[:, 0], P.adjoint(m[:, 0].clone(), 0, 0.5))
        if nf == 3:
            assert torch.equal(om[:, 1:], P.synthesis(a[:, 1:].clone(), 2))
            assert torch.equal(oa[:, 1:], P.adjoint(m[:, 1:].clone(), 2, 0.5))


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_views_the_kernels_cannot_read_in_place(prec):
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(8, 20, spins=(0, 2), prec=prec, autotune=False)
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.randn((3, 2, P.nalm), dtype=torch.complex128, device="cuda", generator=g)
    ref = P.synthesis(a, 2)
    for v in (a.transpose(0, 1).contiguous().transpose(0, 1), a.permute(2, 0, 1).contiguous().permute(1, 2, 0),
              a.conj().resolve_conj().conj()):
        assert torch.equal(P.synthesis(v, 2), ref)
    one = a[:1].expand(4, 2, P.nalm)
    assert torch.equal(P.synthesis(one, 2), P.synthesis(one.contiguous(), 2))
    m = torch.randn((2, 3, 2, P.npix), dtype=torch.float64, device="cuda", generator=g)
    assert torch.equal(P.adjoint(m[:, ::2], 2), P.adjoint(m[:, ::2].contiguous(), 2))
