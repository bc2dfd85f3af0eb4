"""Timed workloads of the package: what an estimator run asks of it, through the public entry points.

The transforms behind ``PolySpec``'s map <-> alm wrappers carry every estimator, so most cases are
single wrapper calls: one T or T,Q,U map in either direction in FP64 (the default precision), the
vectors of maps that the binned and template estimators transform together (spin 0 and spin s), and
the batches of simulations of the mixed-precision backend.  Two cases are whole calls: the masked
conjugate-gradient filter and a binned-bispectrum Fisher contribution.  Sizes follow the test suite
(Nside 16), the power-spectrum workload (Nside 64, lmax 128), the bispectrum workload (Nside 256,
lmax 511 and the class's own default lmax = 3 Nside - 1), the template workload (Nside 512, lmax 1000)
and the Fisher benchmark (Nside 1024, lmax 2048).

``listed`` gives the named cases, ``draw`` another of the same ranges, ``prepare`` the state a
program holds before the call, ``run`` one call, ``work`` its unavoidable bytes and operations and
``exact`` the same outputs from a direct evaluation in torch FP64 (HEALPix ring geometry, scaled
three-term Legendre recurrences, one FFT per ring length).
"""
import contextlib
import functools
import io
import math

import numpy as np
import torch

from polyspec_b200 import PolySpec, Weightings
from polyspec_b200 import workloads as W

# flops of the Legendre stage relative to a spin-0 map, per case: 1 (T), 1 + 4 (T and a Q,U pair), 4 (a spin pair)
_MAX_COST = 5 * 1024 * 2048 ** 2


def listed():
    return [
        # a call of the size the test suite runs everywhere: launch and host latency
        dict(name="teb_to_map_16", op="to_map", nside=16, lmax=47, fields=3),
        # the power-spectrum workload's map analysis, temperature only
        dict(name="t_to_lm_64", op="to_lm", nside=64, lmax=128, fields=1),
        # an ordinary polarised synthesis at the class's default band limit
        dict(name="teb_to_map_256", op="to_map", nside=256, lmax=767, fields=3),
        # an analysis at the template workload's resolution, lmax not a multiple of any tile
        dict(name="tqu_to_lm_512", op="to_lm", nside=512, lmax=1000, fields=3),
        # the Fisher benchmark's transforms, one map set at a time
        dict(name="teb_to_map_1024", op="to_map", nside=1024, lmax=2048, fields=3),
        dict(name="tqu_to_lm_1024", op="to_lm", nside=1024, lmax=2048, fields=3),
        # 24 radial samples of a template estimator: filtered spin-1 maps, and the adjoint of their products
        dict(name="radial_to_map_vec_256", op="to_map_vec", nside=256, lmax=500, batch=24, spin=1),
        dict(name="radial_to_lm_vec_512", op="to_lm_vec", nside=512, lmax=1000, batch=24, spin=0),
        # a batch of simulations on the mixed-precision backend, both directions
        dict(name="mixed_to_map_batch_256", op="to_map_batch", nside=256, lmax=511, batch=33, fields=3),
        dict(name="mixed_to_lm_batch_256", op="to_lm_batch", nside=256, lmax=511, batch=33, fields=3),
        # the masked S^-1 filter of one T,Q,U map to the usual residual
        dict(name="sinv_cg_128", op="sinv", nside=128, lmax=256, fields=3),
        # one Monte Carlo Fisher contribution of the binned bispectrum (T and E, both parities)
        dict(name="bispectrum_fisher_128", op="bispec", nside=128, lmax=255, nbins=6),
    ]


def _cost(case):
    c = case["nside"] * case["lmax"] ** 2 * case.get("batch", 1)
    if case["op"] in ("to_map_vec", "to_lm_vec"):
        return c * (4 if case["spin"] else 1)
    return c * (5 if case.get("fields", 3) == 3 else 1)


def draw(rng):
    op = rng.choice(["to_map", "to_lm", "to_map", "to_lm", "to_map_vec", "to_lm_vec", "to_map_vec", "to_lm_vec",
                     "to_map_batch", "to_lm_batch", "sinv", "bispec"])
    if op in ("to_map", "to_lm"):
        nside = rng.choice([16, 32, 64, 128, 256, 512, 1024])
    elif op in ("to_map_vec", "to_lm_vec"):
        nside = rng.choice([16, 32, 64, 128, 256, 512])
    elif op in ("to_map_batch", "to_lm_batch"):
        nside = rng.choice([64, 128, 256])
    else:
        nside = rng.choice([32, 64, 128])
    case = dict(op=op, nside=nside, lmax=int(nside * math.exp(rng.uniform(math.log(1.2), math.log(3.0)))) - 1)
    if op in ("to_map", "to_lm", "to_map_batch", "to_lm_batch"):
        case["fields"] = rng.choice([1, 3])
    if op in ("to_map_vec", "to_lm_vec"):
        case["batch"] = int(round(math.exp(rng.uniform(math.log(2), math.log(32)))))
        case["spin"] = rng.choice([0, 0, 1, 2, 3])
    if op in ("to_map_batch", "to_lm_batch"):
        case["batch"] = rng.randint(9, 40)
    if op == "sinv":
        case["fields"] = 3
    if op == "bispec":
        case["nbins"] = rng.randint(3, 6)
    while _cost(case) > _MAX_COST:
        case["lmax"] = int(case["lmax"] * 0.9)
    return case


# ------------------------------------------------------------------------------------ states
def _spectra(lmax, fwhm):
    cl = W.fiducial_cl(lmax, True)
    beam = np.stack([W.gaussian_beam(lmax, fwhm)] * 3)
    return cl, beam


def _fwhm(nside):
    return 5120.0 / nside  # 5' at Nside 1024


def _pol(case):
    return case.get("fields", 3) == 3


@functools.lru_cache(maxsize=3)
def _base(nside, lmax, pol, prec, nl):
    """The PolySpec object a program keeps for all its maps of one geometry."""
    cl, beam = _spectra(max(lmax, 3 * nside - 1), _fwhm(nside))
    tot = W.total_cl(cl, beam, W.noise_cl(nside, len(cl['TT']) - 1, 30.0, True) if nl else None)
    if not pol:
        return PolySpec(nside, {'TT': tot['TT']}, beam=beam[0], pol=False, lmax=lmax, prec=prec)
    return PolySpec(nside, dict(tot), beam=list(beam), pol=True, lmax=lmax, prec=prec)


@functools.lru_cache(maxsize=2)
def _filter_inputs(nside):
    mask = W.point_source_mask(nside, 5.74, 100, 60.0 * 64 / nside)
    return np.stack([mask] * 3), W.white_noise_cov(nside)


@functools.lru_cache(maxsize=2)
def _filter(nside, lmax):
    cl, _ = _spectra(max(lmax, 3 * nside - 1), _fwhm(nside))
    mask, noise = _filter_inputs(nside)
    return Weightings(_base(nside, lmax, True, "fp64", True), mask, dict(cl), noise_cov=noise)


@functools.lru_cache(maxsize=2)
def _bispec(nside, lmax, nbins):
    from polyspec_b200.bspec_bin import BSpecBin
    cl, _ = _spectra(max(lmax, 3 * nside - 1), _fwhm(nside))
    mask = W.latitude_mask(nside, 15.0, 5.0)
    base = _base(nside, lmax, True, "fp64", True)
    with contextlib.redirect_stdout(io.StringIO()):
        wts = Weightings(base, np.stack([mask] * 3), dict(cl), noise_cov=W.white_noise_cov(nside))
        edges = np.unique(np.round(np.geomspace(2, lmax, nbins + 1)).astype(int))
        est = BSpecBin(base, mask, wts.make_applySinv('ideal'), edges, fields=['TTT', 'TTE', 'TEE', 'EEE'],
                       parity='both')
        est._compute_symmetry_factor()
    return est


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _lm(lmax):
    m = torch.repeat_interleave(torch.arange(lmax + 1, device="cuda"), torch.arange(lmax + 1, 0, -1, device="cuda"))
    n = m.numel()
    l = torch.arange(n, device="cuda") - m * (2 * lmax + 1 - m) // 2
    return l, m


def _grf(nside, lmax, n, nfield, gen, beamed=True):
    """n Gaussian fields [n, nfield, nlm] of the fiducial spectra (T, E, B correlated as C_l says)."""
    cl, beam = _spectra(lmax, _fwhm(nside))
    l, m = _lm(lmax)
    z = torch.randn((n, nfield, l.numel(), 2), generator=gen, device="cuda", dtype=torch.float64)
    z = torch.complex(z[..., 0], torch.where(m > 0, z[..., 1], torch.zeros_like(z[..., 1])))
    z[..., lmax + 1:] *= math.sqrt(0.5)  # m > 0
    c = {k: torch.as_tensor(v, device="cuda")[l] for k, v in cl.items()}
    b = torch.as_tensor(beam[0], device="cuda")[l] if beamed else 1.0
    out = torch.empty_like(z)
    out[:, 0] = z[:, 0] * c['TT'].sqrt() * b
    if nfield == 3:
        out[:, 1] = (z[:, 0] * (c['TE'] / c['TT'].sqrt()) + z[:, 1] * (c['EE'] - c['TE'] ** 2 / c['TT']).sqrt()) * b
        out[:, 2] = z[:, 2] * c['BB'].sqrt() * b
    return out


def _noise_maps(nside, n, nfield, gen):
    """n masked white-noise maps of 30 uK arcmin [n, nfield, npix]."""
    var = torch.as_tensor(W.white_noise_cov(nside)[:nfield], device="cuda")
    mask = torch.as_tensor(W.latitude_mask(nside, 15.0, 5.0), device="cuda")
    x = torch.randn((n, nfield, 12 * nside ** 2), generator=gen, device="cuda", dtype=torch.float64)
    return x * var.sqrt() * mask


def _input(case, seed):
    """The call's argument, from the seed alone."""
    g, op, nside, lmax = _gen(seed), case["op"], case["nside"], case["lmax"]
    nf = 3 if _pol(case) else 1
    if op == "to_map":
        return _grf(nside, lmax, 1, nf, g)[0]
    if op == "to_lm":
        return _noise_maps(nside, 1, nf, g)[0]
    if op == "to_map_batch":
        return _grf(nside, lmax, case["batch"], nf, g)
    if op == "to_lm_batch":
        return _noise_maps(nside, case["batch"], nf, g)
    if op == "to_map_vec":
        return _grf(nside, lmax, case["batch"], 1, g)[:, 0]
    if op == "to_lm_vec":
        if case["spin"] == 0:
            return _noise_maps(nside, case["batch"], 1, g)[:, 0]
        x = _noise_maps(nside, 2 * case["batch"], 1, g)[:, 0]
        x = torch.complex(x[::2].contiguous(), x[1::2].contiguous())
        return torch.stack([x, x.conj().resolve_conj()])
    if op == "sinv":
        mask, noise = _filter_inputs(nside)
        npix = 12 * nside ** 2
        x = torch.randn((3, npix), generator=g, device="cuda", dtype=torch.float64)
        signal = torch.randn((3, npix), generator=g, device="cuda", dtype=torch.float64)
        return (x * torch.as_tensor(noise, device="cuda").sqrt() + signal) * torch.as_tensor(mask, device="cuda")
    return list(_grf(nside, lmax, 2, 3, g, beamed=False))


def prepare(case, seed):
    op, nside, lmax = case["op"], case["nside"], case["lmax"]
    x = _input(case, seed)
    if op == "sinv":
        return dict(case=case, x=x, filter=_filter(nside, lmax))
    if op == "bispec":
        return dict(case=case, x=x, est=_bispec(nside, lmax, case["nbins"]))
    prec = "mixed" if op in ("to_map_batch", "to_lm_batch") else "fp64"
    return dict(case=case, x=x, base=_base(nside, lmax, _pol(case), prec, False))


def run(state):
    case, x = state["case"], state["x"]
    op = case["op"]
    if op == "to_map":
        return state["base"].to_map(x)
    if op == "to_lm":
        return state["base"].to_lm(x)
    if op == "to_map_batch":
        return state["base"].to_map_batch(x)
    if op == "to_lm_batch":
        return state["base"].to_lm_batch(x)
    if op == "to_map_vec":
        return state["base"].to_map_vec(x, output_spin=case["spin"])
    if op == "to_lm_vec":
        return state["base"].to_lm_vec(x, spin=case["spin"])
    if op == "sinv":
        return state["filter"].applySinv_optimal(x, preconditioner="harmonic", nstep=500, thresh=1e-6)
    return state["est"].compute_fisher_contribution(0, a_lms=x)


# ------------------------------------------------------------------------------------ work
def _transform_work(nside, lmax, n0, ns):
    """n0 spin-0 maps and ns spin pairs: alm and map once each; Legendre sums and ring FFTs."""
    nlm, npix = (lmax + 1) * (lmax + 2) // 2, 12 * nside ** 2
    nmap = n0 + 2 * ns
    flops = 2 * nside * nlm * (4.0 * n0 + 16.0 * ns) + nmap * 2.5 * npix * math.log2(4 * nside)
    return nmap * (16.0 * nlm + 8.0 * npix), flops


def work(case):
    nside, lmax, op = case["nside"], case["lmax"], case["op"]
    nlm, npix = (lmax + 1) * (lmax + 2) // 2, 12 * nside ** 2
    pol = _pol(case)
    if op in ("to_map", "to_lm", "to_map_batch", "to_lm_batch"):
        b, f = _transform_work(nside, lmax, case.get("batch", 1), case.get("batch", 1) if pol else 0)
    elif op in ("to_map_vec", "to_lm_vec"):
        n, s = case["batch"], case["spin"]
        b, f = _transform_work(nside, lmax, n if s == 0 else 0, n if s else 0)
        if s:  # one harmonic input for two complex maps, or two complex maps for two harmonic outputs
            b = n * (16.0 * nlm + 32.0 * npix) if op == "to_map_vec" else n * (32.0 * nlm + 32.0 * npix)
    elif op == "sinv":
        # the starting point, the right-hand side and its residual, then at least two steps
        _, f = _transform_work(nside, lmax, 1, 1)
        b, f = 3 * (8.0 * npix * 3 + 16.0 * nlm), f * (4 + 2 * 2)
    else:
        # per field and weighting: H maps of every (bin, field) in spin 1 and 2, the adjoints of their pairs
        # in both spins and the filter of the rows it makes
        h = 2 * case["nbins"]
        _, f = _transform_work(nside, lmax, 0, 4 * 2 * h + 4 * 2 * h * (h + 1) // 2)
        b = 2 * 3 * 16.0 * nlm
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------ direct FP64 evaluation
def _rings(nside):
    """cos(theta), 1 - cos, 1 + cos of the north rings and the equator, and every ring's (start, length, phi0)."""
    i = torch.arange(1, 2 * nside + 1, dtype=torch.float64)
    cap = i < nside
    omz = torch.where(cap, i * i / (3.0 * nside ** 2), 1.0 - (2 * nside - i) * 2.0 / (3.0 * nside))
    z = torch.where(cap, 1.0 - omz, (2 * nside - i) * 2.0 / (3.0 * nside))
    ring = []
    npix = 12 * nside ** 2
    for k in range(1, 4 * nside):
        ii = k if k <= 2 * nside else 4 * nside - k
        if ii < nside:
            start = 2 * ii * (ii - 1) if k <= 2 * nside else npix - 2 * ii * (ii + 1)
            ring.append((start, 4 * ii, math.pi / (4 * ii)))
        else:
            start = 2 * nside * (nside - 1) + (k - nside) * 4 * nside
            ring.append((start, 4 * nside, math.pi / (4 * nside) if (k - nside) % 2 == 0 else 0.0))
    return z.cuda(), omz.cuda(), (1.0 + z).cuda(), ring


def _scaled(mant, e):
    """mant 2^e as (v, k): v 2^(800 k), k <= 0, and |v| small while k < 0."""
    k = torch.where(e <= -400, -torch.div(-400 - e, 800, rounding_mode="floor") - 1, torch.zeros_like(e))
    return torch.ldexp(mant, (e - 800 * k).double()), k


def _legendre(nside, lmax, s):
    """Yields l and, for m = 0..l on the north rings, lambda_lm (s = 0) or the halves of the sum and the difference of
    the +s and -s functions; negligible values are 0."""
    z, omz, opz, _ = _rings(nside)
    sh, ch = (0.5 * omz).sqrt(), (0.5 * opz).sqrt()
    R, dev = len(z), z.device
    x = z[:, None]
    nfun = 1 if s == 0 else 2
    cur = [torch.zeros((R, lmax + 1), dtype=torch.float64, device=dev) for _ in range(nfun)]
    prev = [torch.zeros_like(c) for c in cur]
    k = torch.zeros((R, lmax + 1), dtype=torch.int32, device=dev)

    def power(base, n):  # base^n as mantissa and exponent, by squaring
        r, re = torch.full_like(base, 0.5), torch.ones_like(base, dtype=torch.int32)
        b, be = torch.frexp(base)
        while n:
            if n & 1:
                r, d = torch.frexp(r * b)
                re = re + be + d
            b, d = torch.frexp(b * b)
            be = 2 * be + d
            n >>= 1
        return r, re

    def norm(n, j, l):  # sqrt(C(n, j) (2 l + 1) / 4 pi) as mantissa and exponent
        c = math.comb(n, j) * (2 * l + 1)
        e = max(0, c.bit_length() - 64)
        e += e & 1
        v, d = math.frexp(math.sqrt((c >> e) / (4 * math.pi)))
        return v, e // 2 + d

    def seed(m):
        l = max(m, s)
        v, e = norm(2 * l, l + min(m, s), l)
        a, ae = power(sh, l + min(m, s))
        b, be = power(ch, l - min(m, s))
        c, ce = power(sh, l - min(m, s))
        d, de = power(ch, l + min(m, s))
        f, fe = torch.frexp(a * b * v)
        g, ge = torch.frexp(c * d * v)
        fe, ge = fe + ae + be + e, ge + ce + de + e
        sf = -1.0 if m & 1 else 1.0
        sg = sf if m >= s else (-1.0 if s & 1 else 1.0)
        if s == 0:
            cur[0][:, m], k[:, m] = (lambda t: (t[0] * sf, t[1]))(_scaled(f, fe))
            return
        big = torch.maximum(fe, ge)
        one, kk = _scaled(torch.ones_like(f), big)
        cur[0][:, m] = one * torch.ldexp(f, torch.clamp(fe - big, min=-1070).double()) * sf
        cur[1][:, m] = one * torch.ldexp(g, torch.clamp(ge - big, min=-1070).double()) * sg
        k[:, m] = kk

    m = torch.arange(lmax + 1, dtype=torch.float64, device=dev)
    for l in range(lmax + 1):
        if l == s:
            for mm in range(s + 1):
                seed(mm)
        elif l > s:
            seed(l)
        n = l + 1
        if l >= s:
            live = k[:, :n] == 0
            v = [torch.where(live, c[:, :n], 0.0) for c in cur]
            yield l, (v[0] if s == 0 else (0.5 * (v[0] + v[1]), 0.5 * (v[0] - v[1])))
            mm = m[:n]
            rho = lambda L: ((L * L - mm * mm).clamp(min=0) * (L * L - s * s)).clamp(min=0).sqrt()  # noqa: E731
            r1, q = rho(l + 1.0), math.sqrt((2 * l + 3.0) * (2 * l + 1.0))
            A = q * (l + 1.0) / r1
            D = q * mm * s / (max(l, 1) * r1)
            C = math.sqrt((2 * l + 3.0) / max(2 * l - 1.0, 1.0)) * (l + 1.0) * rho(float(l)) / (max(l, 1) * r1)
            for i in range(nfun):
                nxt = (A * x + (D if i == 0 else -D)) * cur[i][:, :n] - C * prev[i][:, :n]
                prev[i][:, :n] = cur[i][:, :n]
                cur[i][:, :n] = nxt
            if l % 8 == 7:
                up = cur[0][:, :n].abs() if s == 0 else torch.maximum(cur[0][:, :n].abs(), cur[1][:, :n].abs())
                up = (k[:, :n] < 0) & (up > 2.0 ** 400)
                for v in cur + prev:
                    v[:, :n] = torch.where(up, v[:, :n] * 2.0 ** -800, v[:, :n])
                k[:, :n] += up.int()


def _alm_at(alm, l, lmax):
    m = torch.arange(l + 1, device="cuda")
    return alm[..., m * (2 * lmax + 1 - m) // 2 + l]


def _sign(l):
    return 1.0 - 2.0 * ((l + torch.arange(l + 1, device="cuda")) % 2)


def _exact_synthesis(nside, lmax, alm, s):
    """alm [B, nc, nlm] -> maps [B, nc, npix], nc = 1 (s = 0) or 2 (G, C -> Q, U)."""
    B, nc, _ = alm.shape
    north = torch.zeros((B, nc, 2 * nside, lmax + 1), dtype=torch.complex128, device="cuda")
    south = torch.zeros_like(north)
    for l, F in _legendre(nside, lmax, s):
        a, sg = _alm_at(alm, l, lmax)[:, :, None], _sign(l)
        if s == 0:
            t = F * a
            north[..., :l + 1] += t
            south[..., :l + 1] += t * sg
            continue
        Fe, Fo = F if s % 2 == 0 else (F[1], F[0])  # the even one multiplies G in Q
        se, so = (sg, -sg) if s % 2 == 0 else (-sg, sg)
        for out, e, o in ((north, Fe, Fo), (south, Fe * se, Fo * so)):
            out[:, 0, :, :l + 1] -= e * a[:, 0] + 1j * (o * a[:, 1])
            out[:, 1, :, :l + 1] += 1j * (o * a[:, 0]) - e * a[:, 1]
    _, _, _, ring = _rings(nside)
    maps = torch.empty((B, nc, 12 * nside ** 2), dtype=torch.float64, device="cuda")
    m = torch.arange(lmax + 1, device="cuda")
    for k, (start, n, phi0) in enumerate(ring):
        c = (north[:, :, k] if k < 2 * nside else south[:, :, 4 * nside - 2 - k]) * torch.exp(1j * phi0 * m.double())
        c[..., 0] = c[..., 0].real + 0j
        pad = torch.zeros((B, nc, -(-(lmax + 1) // n) * n), dtype=torch.complex128, device="cuda")
        pad[..., :lmax + 1] = c
        up = pad.reshape(B, nc, -1, n).sum(2)
        pad[..., 0] = 0
        down = torch.roll(pad.reshape(B, nc, -1, n).sum(2).flip(-1), 1, -1).conj()
        maps[:, :, start:start + n] = torch.fft.ifft(up + down, norm="forward").real
    return maps


def _exact_adjoint(nside, lmax, maps, s):
    """maps [B, nc, npix] -> alm [B, nc, nlm], times pi / (3 nside^2)."""
    B, nc, _ = maps.shape
    _, _, _, ring = _rings(nside)
    north = torch.empty((B, nc, 2 * nside, lmax + 1), dtype=torch.complex128, device="cuda")
    south = torch.zeros_like(north)
    m = torch.arange(lmax + 1, device="cuda")
    for k, (start, n, phi0) in enumerate(ring):
        p = torch.fft.fft(maps[:, :, start:start + n])[..., m % n] * torch.exp(-1j * phi0 * m.double())
        if k < 2 * nside:
            north[:, :, k] = p
        else:
            south[:, :, 4 * nside - 2 - k] = p
    plus, minus = north + south, north - south
    del north, south
    alm = torch.zeros((B, nc, (lmax + 1) * (lmax + 2) // 2), dtype=torch.complex128, device="cuda")
    for l, F in _legendre(nside, lmax, s):
        n = l + 1
        even = _sign(l) > 0
        mm = torch.arange(n, device="cuda")
        idx = mm * (2 * lmax + 1 - mm) // 2 + l
        P, M = plus[..., :n], minus[..., :n]
        if s == 0:
            alm[..., idx] = (F * torch.where(even, P, M)).sum(2)
            continue
        Fe, Fo = F if s % 2 == 0 else (F[1], F[0])
        flip = even if s % 2 == 0 else ~even
        e = (Fe * torch.where(flip, P, M)).sum(2)
        o = (Fo * torch.where(flip, M, P)).sum(2)
        alm[:, 0, idx] = -e[:, 0] - 1j * o[:, 1]
        alm[:, 1, idx] = 1j * o[:, 0] - e[:, 1]
    return alm * (math.pi / (3.0 * nside ** 2))


def _exact_to_map(nside, lmax, alm):
    out = [_exact_synthesis(nside, lmax, alm[:, :1], 0)]
    if alm.shape[1] == 3:
        out.append(_exact_synthesis(nside, lmax, alm[:, 1:], 2))
    return torch.cat(out, 1)


def _exact_to_lm(nside, lmax, maps):
    out = [_exact_adjoint(nside, lmax, maps[:, :1], 0)]
    if maps.shape[1] == 3:
        out.append(_exact_adjoint(nside, lmax, maps[:, 1:], 2))
    return torch.cat(out, 1)


def _exact_sinv(case, d):
    """The preconditioned conjugate gradients of C^-1 + B Y^H W N^-1 W Y B, from the Wiener start, to 1e-6."""
    nside, lmax = case["nside"], case["lmax"]
    cl, beam = _spectra(max(lmax, 3 * nside - 1), _fwhm(nside))
    tot = W.total_cl(cl, beam, W.noise_cl(nside, len(cl['TT']) - 1, 30.0, True))
    mask, noise = _filter_inputs(nside)
    area = 4 * math.pi / (12 * nside ** 2)

    def matrix(c):
        z = np.zeros_like(c['TT'])
        rows = [[c['TT'], c['TE'], z], [c['TE'], c['EE'], z], [z, z, c['BB']]]
        return np.moveaxis(np.asarray(rows)[:, :, :lmax + 1], 2, 0)

    C, inv_tot, b = matrix(cl), np.linalg.inv(matrix(tot)), beam[0][:lmax + 1]
    inv = np.linalg.inv(C)
    nl = np.asarray([noise[i][mask[i] > 0.99].mean() * area for i in range(3)])
    inv_s = inv + b[:, None, None] ** 2 * np.diag(1.0 / nl)
    inv_s[:2] = inv_s[2]
    l, m = _lm(lmax)
    per_lm = lambda a: torch.as_tensor(a, device="cuda")[l]  # noqa: E731
    sigma, inv, start = per_lm(np.linalg.inv(inv_s)), per_lm(inv), per_lm(C @ (b[:, None, None] * inv_tot))
    b, mw = per_lm(b), torch.where(m > 0, 2.0, 1.0)
    mask, icov = torch.as_tensor(mask, device="cuda"), 1.0 / torch.as_tensor(noise, device="cuda")
    mul = lambda a, v: torch.einsum("iab,bi->ai", a.to(torch.complex128), v)  # noqa: E731
    dot = lambda u, v: float(((u * v.conj()).real * mw).sum())  # noqa: E731
    to_lm = lambda t: _exact_to_lm(nside, lmax, t[None])[0]  # noqa: E731
    A = lambda v: mul(inv, v) + b * to_lm(mask ** 2 * icov / area * _exact_to_map(nside, lmax, (b * v)[None])[0])  # noqa: E731
    x0 = mul(start, to_lm(d))
    rhs = b * to_lm(d * icov / area * mask)
    r = rhs - A(x0)
    x, z = torch.zeros_like(r), mul(sigma, r)
    rz, rz0, p = dot(r, z), dot(rhs, mul(sigma, rhs)), z
    for _ in range(40):
        Ap = A(p)
        alpha = rz / dot(p, Ap)
        x, r = x + alpha * p, r - alpha * Ap
        z = mul(sigma, r)
        rz, old = dot(r, z), rz
        if rz / rz0 < 1e-6:
            break
        p = z + rz / old * p
    return mul(inv, x + x0)


def exact(case, seed):
    op, nside, lmax = case["op"], case["nside"], case["lmax"]
    if op == "bispec":
        return None
    x = _input(case, seed)
    if op == "to_map":
        return _exact_to_map(nside, lmax, x[None])[0]
    if op == "to_map_batch":
        return _exact_to_map(nside, lmax, x)
    if op == "to_lm":
        return _exact_to_lm(nside, lmax, x[None])[0]
    if op == "to_lm_batch":
        return _exact_to_lm(nside, lmax, x)
    if op == "sinv":
        return _exact_sinv(case, x)
    s = case["spin"]
    if op == "to_map_vec":
        if s == 0:
            return _exact_synthesis(nside, lmax, x[:, None], 0)[:, 0]
        y = _exact_synthesis(nside, lmax, torch.stack([-x, torch.zeros_like(x)], 1), s)
        return torch.stack([torch.complex(y[:, 0], y[:, 1]), torch.complex(y[:, 0], -y[:, 1])])
    if s == 0:
        return _exact_adjoint(nside, lmax, x[:, None], 0)[:, 0]
    y = _exact_adjoint(nside, lmax, torch.stack([x[0].real, x[0].imag], 1).contiguous(), s)
    return torch.stack([-(y[:, 0] + 1j * y[:, 1]), -(-1.0) ** s * (y[:, 0] - 1j * y[:, 1])])
