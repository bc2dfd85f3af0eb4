"""The mixed-precision synthesis reads the alm of a batch in an order of its own; field and order counts at the edges
of the tiles that bring them there (up to 32 fields; 32 to 512 values)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax", [1, 7, 30, 37])  # 3, 36, 496 and 741 values
@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 8, 9, 16, 17, 33])
@pytest.mark.parametrize("spin", [0, 2])
def test_batch_matches_fp64(lmax, batch, spin):
    from polyspec_b200.sht import SHTPlan
    if lmax < spin:
        pytest.skip("no spin-2 order below l = 2")
    mixed, exact = (SHTPlan(16, lmax, spins=(0, 2), prec=p, autotune=False) for p in ("mixed", "fp64"))
    g = torch.Generator(device="cuda").manual_seed(lmax * 100 + batch)
    shape = (batch,) + ((2,) if spin else ()) + (mixed.nalm,)
    alm = torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)
    # FP32 sums of lmax terms and the FP32 ring transform: a few 1e-7 of the map's rms per pixel
    ref = exact.synthesis(alm, spin)
    err = mixed.synthesis(alm, spin) - ref
    rms = ref.reshape(batch, -1).pow(2).mean(1).sqrt()
    assert (err.reshape(batch, -1).abs().amax(1) <= 1e-5 * rms).all()
