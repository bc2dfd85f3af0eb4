"""The workspace of FP64 transforms is their phases alone, in both directions: its size, that nothing outside of it is
written, and that the allocation-free synthesis takes what fits its 16 MiB."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax,spin,batch", [(1, 0, 0, 1), (4, 20, 0, 3), (8, 30, 2, 1), (8, 5, 3, 9),
                                                   (128, 383, 0, 5), (64, 191, 2, 4)])
def test_phases_alone(nside, lmax, spin, batch):
    import torch
    from polyspec_b200 import _lib
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(nside, lmax, spins=(0, spin), autotune=False)
    nc = 1 if spin == 0 else 2
    phases = ((4 * nside - 1) * (lmax + 1) * batch * nc * 16 + 255) // 256 * 256
    n = ctypes.c_size_t()
    for adjoint in (0, 1):
        _lib.call("ps_sht_workspace_bytes", P._h, batch, spin, adjoint, ctypes.byref(n))
        assert n.value == phases
    g = torch.Generator(device="cuda").manual_seed(nside)
    alm = torch.randn((batch,) + (2,) * (spin > 0) + (P.nalm,), dtype=torch.complex128, device="cuda", generator=g)
    want = P.synthesis(alm, spin)
    guard = 4096
    ws = torch.full((phases + 2 * guard,), 0x5a, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(want)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    args = (P._h, ctypes.c_void_p(alm.data_ptr()), ctypes.c_void_p(out.data_ptr()), batch, spin)
    _lib.call("ps_synthesis", *args, ctypes.c_void_p(ws.data_ptr() + guard), phases, stream)
    assert torch.equal(out, want)
    assert bool((ws[:guard] == 0x5a).all()) and bool((ws[-guard:] == 0x5a).all())
    assert _lib.lib().ps_synthesis(*args, ctypes.c_void_p(ws.data_ptr() + guard), phases - 1, stream) == -5
    out.zero_()
    _lib.call("ps_synthesis_noalloc", *args, stream)
    assert torch.equal(out, want)
