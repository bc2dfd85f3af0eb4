"""FP64 plans exist at every ring length up to Nside 1024, in all spins, and are refused as unsupported where the longest
convolution (16384 points from Nside 1025 on) does not fit shared memory; comparisons with an FP64 plan rest on this."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax", [(1, 40), (3, 40), (7, 100), (8, 300), (48, 143), (96, 287), (512, 20), (513, 20),
                                        (600, 50), (1024, 20)])
def test_created(nside, lmax):
    import torch
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(nside, lmax, autotune=False)
    alm = torch.zeros((1, 2, P.nalm), dtype=torch.complex128, device="cuda")
    for s in (1, 2, 3):
        assert not P.synthesis(alm, s).any()


@pytest.mark.parametrize("nside", [1025, 2048])
def test_refused(nside):
    from polyspec_b200 import _lib
    from polyspec_b200.sht import SHTPlan
    with pytest.raises(_lib.PSError) as e:
        SHTPlan(nside, 20, autotune=False)
    assert e.value.code == _lib.PS_ERR_UNSUPPORTED
