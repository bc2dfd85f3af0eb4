"""Which FP64 Legendre kernels run is a rule on sizes, not a timing: an FP64 plan is neither timed nor given a tile, and
two plans return the same bits whatever a tuning cache holds.  Batches beyond the largest grid, and the rule's neighbours,
agree with the other kernels to 1e-12 of the largest value (FP64 sums in another order).
"""
import json

import pytest


def test_fp64_plans_are_not_timed(monkeypatch, tmp_path):
    from polyspec_b200 import _lib, autotune
    monkeypatch.setenv("PS_TUNE_CACHE", str(tmp_path / "tune.json"))
    calls = []
    monkeypatch.setattr(_lib, "call", lambda *a: calls.append(a))
    t = autotune.Tuner(16, 47, {"fp64": "h"}, None)
    t.disk = {"%s|%s|spin%d|b1" % (t.prefix, d, s): {"pipeline": "fp64", "tile": 4}
              for d in ("synthesis", "adjoint") for s in (0, 2)}
    for direction in (0, 1):
        for spin in (0, 2):
            for B in (1, 2, 24):
                assert t.select(direction, spin, B, lambda h: calls.append("run")) == "h"
    assert "run" not in calls and calls and all(c[-1] == 0 for c in calls)
    assert not (tmp_path / "tune.json").exists()
    mixed = autotune.Tuner(16, 47, {"fp64": "h", "mixed": "m"}, None)
    assert all(tile == 0 for d in (0, 1) for s in (0, 2) for pl, tile in mixed._candidates(d, s, 2, False)
               if pl == "fp64")


@pytest.mark.gpu
@pytest.mark.parametrize("B", [1, 2, 4])
def test_bits_do_not_depend_on_the_cache(monkeypatch, tmp_path, B):
    import torch
    from polyspec_b200.sht import SHTPlan
    out = []
    for k, tiles in enumerate(({0: 1, 2: 1}, {0: 4, 2: 2})):
        cache = tmp_path / ("tune%d.json" % k)
        monkeypatch.setenv("PS_TUNE_CACHE", str(cache))
        prefix = SHTPlan(32, 64)._tuner.prefix
        cache.write_text(json.dumps({"%s|%s|spin%d|b%d" % (prefix, d, s, B): {
            "pipeline": "fp64", "tile": 1 if (d, s) == ("adjoint", 2) else tiles[s], "ms": {}}
            for d in ("synthesis", "adjoint") for s in (0, 2)}))
        P = SHTPlan(32, 64)
        g = torch.Generator(device="cuda").manual_seed(B)
        alm = torch.randn((B, 2, P.nalm), dtype=torch.complex128, device="cuda", generator=g)
        mp = torch.randn((B, 2, P.npix), dtype=torch.float64, device="cuda", generator=g)
        out.append([P.synthesis(alm[:, 0], 0), P.synthesis(alm, 2), P.adjoint(mp[:, 0], 0), P.adjoint(mp, 2)])
    assert all(torch.equal(a, b) for a, b in zip(*out))


# sides of the rule: batches, orders and rings on both sides of its lines, and a batch above 65535
@pytest.mark.gpu
@pytest.mark.parametrize("nside,lmax,B", [(1, 1, 70000), (16, 47, 5), (16, 47, 40), (32, 95, 15), (32, 95, 33), (64, 128, 5),
                                          (64, 128, 6), (64, 128, 15), (64, 128, 16), (64, 146, 3), (64, 148, 3),
                                          (64, 148, 4), (128, 256, 1), (128, 256, 2), (128, 256, 3), (128, 383, 3)])
@pytest.mark.parametrize("spin", [0, 2])
def test_sides_of_the_rule(nside, lmax, B, spin):
    import torch
    from polyspec_b200 import _lib
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(nside, lmax, spins=(0, 2), autotune=False)
    g = torch.Generator(device="cuda").manual_seed(B)
    sh = (B,) if spin == 0 else (B, 2)
    alm = torch.randn(sh + (P.nalm,), dtype=torch.complex128, device="cuda", generator=g)
    mp = torch.randn(sh + (P.npix,), dtype=torch.float64, device="cuda", generator=g)
    got = P.synthesis(alm, spin), P.adjoint(mp, spin)
    assert torch.equal(got[0], P.synthesis(alm, spin)) and torch.equal(got[1], P.adjoint(mp, spin))
    for direction, x in enumerate(got):
        for tile in ((1, 4) if spin == 0 else (1, 2) if direction == 0 else (1,)):
            if B > 65535 and tile == 1 and direction == 0:
                continue  # single maps fill a grid layer each
            _lib.call("ps_plan_set_tile", P._h, direction, spin, tile)
            ref = P.synthesis(alm, spin) if direction == 0 else P.adjoint(mp, spin)
            assert float((x - ref).abs().max()) <= 1e-12 * float(ref.abs().max())
        _lib.call("ps_plan_set_tile", P._h, direction, spin, 0)
