"""T and (Q, U) transformed in one call (their rings share a launch) against the transforms of each spin: the same
kernels on the same numbers, so equal to the last bit.  Sizes: the smallest plan, rings folded many times and not at
all, both launches of the ring transforms (work lengths up to 4096, and 8192), the largest joint batch and one more."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax,batch", [(1, 2, 1), (2, 40, 2), (16, 47, 4), (16, 47, 5), (100, 130, 3),
                                              (1024, 100, 1)])
@pytest.mark.parametrize("autotune", [False, True])
def test_joint_equals_single_spins(nside, lmax, batch, autotune, tmp_path, monkeypatch):
    from polyspec_b200.sht import SHTPlan
    monkeypatch.setenv("PS_TUNE_CACHE", str(tmp_path / "tune.json"))
    P = SHTPlan(nside, lmax, spins=(0, 2), autotune=autotune)
    g = torch.Generator(device="cuda").manual_seed(nside)
    a = torch.randn((batch, 3, P.nalm), dtype=torch.complex128, device="cuda", generator=g)
    m = torch.randn((batch, 3, P.npix), dtype=torch.float64, device="cuda", generator=g)
    om, oa = torch.empty_like(m), torch.empty_like(a)
    for _ in range(2):  # the workspace grown and kept
        n = (P.n_synthesis, P.n_adjoint)
        P.synthesis_fields(a, om)
        P.adjoint_fields(m, oa, 0.25)
        assert (P.n_synthesis, P.n_adjoint) == (n[0] + 2 * batch, n[1] + 2 * batch)
    assert torch.equal(om[:, 0], P.synthesis(a[:, 0], 0)) and torch.equal(om[:, 1:], P.synthesis(a[:, 1:], 2))
    assert torch.equal(oa[:, 0], P.adjoint(m[:, 0], 0, 0.25)) and torch.equal(oa[:, 1:], P.adjoint(m[:, 1:], 2, 0.25))


def test_refused_on_the_host():
    from polyspec_b200 import _lib
    from polyspec_b200.sht import SHTPlan
    P, M = SHTPlan(4, 8, spins=(0, 2), autotune=False), SHTPlan(4, 8, spins=(0, 2), prec="mixed", autotune=False)
    Z = SHTPlan(4, 8, spins=(0,), autotune=False)
    a = torch.zeros((1, 3, P.nalm), dtype=torch.complex128, device="cuda")
    m = torch.zeros((1, 3, P.npix), dtype=torch.float64, device="cuda")
    ws, n = P._joint_workspace(1)
    call = _lib.lib().ps_synthesis_fields
    args = lambda h, sa=0, sm=0, b=1, nb=n: call(h, a.data_ptr(), sa, m.data_ptr(), sm, b, ws.data_ptr(),  # noqa: E731
                                                 ctypes.c_size_t(nb), P._stream())
    assert args(P._h) == 0 and args(P._h, b=0) == 0
    assert args(P._h, sa=3 * P.nalm - 1) == -1 and args(P._h, sm=3 * P.npix - 1) == -1 and args(P._h, b=-1) == -1
    assert args(Z._h) == -1
    assert args(M._h) == _lib.PS_ERR_UNSUPPORTED and args(P._h, nb=n - 1) not in (0, -1)


@pytest.mark.parametrize("nside,lmax,batch", [(16, 47, 1), (128, 200, 1), (64, 100, 4)])
def test_captured_and_back_to_back(nside, lmax, batch):
    """Calls in a row share the workspace, on a stream and in a graph: each must see the one before it finished."""
    from polyspec_b200.sht import SHTPlan
    P = SHTPlan(nside, lmax, spins=(0, 2), autotune=False)
    g = torch.Generator(device="cuda").manual_seed(nside)
    x = [torch.randn((batch, 3, P.nalm), dtype=torch.complex128, device="cuda", generator=g) for _ in range(3)]
    om = [torch.empty((batch, 3, P.npix), dtype=torch.float64, device="cuda") for _ in x]
    oa = [torch.empty_like(a) for a in x]

    def go():
        for a, m, b in zip(x, om, oa):
            P.synthesis_fields(a, m)
            P.adjoint_fields(m, b)
    go()
    ref_m = [torch.cat([P.synthesis(a[:, 0], 0)[:, None], P.synthesis(a[:, 1:], 2)], 1) for a in x]
    ref_a = [torch.cat([P.adjoint(m[:, 0], 0)[:, None], P.adjoint(m[:, 1:], 2)], 1) for m in ref_m]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        go()
    for run in (go, graph.replay):
        for t in om + oa:
            t.fill_(float("nan"))
        for _ in range(20):
            run()
        assert all(torch.equal(a, b) for a, b in zip(om + oa, ref_m + ref_a))
