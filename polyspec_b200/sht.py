"""Device-side HEALPix SHTs through libpscuda (torch tensors in, torch tensors out).

``SHTPlan(nside, lmax)`` wraps one ``ps_plan``.  Its transforms take and
return CUDA tensors in the ducc0 layout used by the reference
(polyspec/base.py:147-282):

* spin 0:   alm ``complex128 [B, nalm]``    <->  map ``float64 [B, npix]``
* spin s>0: alm ``complex128 [B, 2, nalm]`` <->  map ``float64 [B, 2, npix]``
  (components G, C <-> Q, U)

``adjoint`` is ducc0's ``adjoint_synthesis`` times ``scale``.

With ``autotune=True`` (default) the first call of each (direction, spin,
batch bucket) of a ``prec='mixed'`` plan times the candidate tile shapes of its
Legendre kernels and, up to eight maps, the FP64 pipeline (an FP64 plan is kept
beside the mixed one) and keeps the fastest (polyspec_b200.autotune; choices
cached in JSON).  The FP64 kernels win for small batches (and are exact to FP64),
the tensor-core pipeline above 12 (spin s) to 16 maps (spin 0): Nside 256, lmax 511,
spin 2, synthesis of 2 / 12 / 33 maps 0.24 / 0.79 / 2.14 ms in FP64 and 0.57 / 0.79 /
1.68 ms mixed.

FP64 results do not depend on timings: the same call gives the same bits in every
process.  A map's last bits (1e-15) may depend on the size of the batch it comes in,
since small and large batches run on kernels that order their sums differently.

Legendre tables (``tables='auto'``, mixed precision only): the first transform
of a spin builds the plan's FP32 Legendre table of that spin
(``ps_plan_build_table``) when it fits in ``table_fraction`` of the free device
memory (default 0.45, or the environment variable PS_TABLE_MEM_FRACTION); the
Legendre stages of that spin then stream the table through tensor-core GEMMs.
Where it does not fit (Nside 2048 at lmax 4096 needs 137 GB for spin 0) the
on-the-fly kernels run.  ``tables=True`` builds regardless of the budget (and
raises if the allocation fails), ``tables=False`` never builds.
"""
import ctypes
import os

import torch

from . import _lib


def nalm(lmax):
    return (lmax + 1) * (lmax + 2) // 2


class SHTPlan:
    def __init__(self, nside, lmax=None, spins=(0, 1, 2, 3), prec="fp64", device=None, autotune=True,
                 tables="auto", table_fraction=None, table_format=None):
        if not torch.cuda.is_available():
            raise RuntimeError("the CUDA backend needs a GPU (no CPU fallback)")
        self.nside = int(nside)
        self.lmax = 3 * self.nside - 1 if lmax is None else int(lmax)
        self.npix = 12 * self.nside ** 2
        self.nalm = nalm(self.lmax)
        self.device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
        self.prec = prec
        mask = 0
        for s in spins:
            mask |= 1 << int(s)
        self.spins = tuple(spins)
        h = ctypes.c_void_p()
        with torch.cuda.device(self.device):
            _lib.call("ps_plan_create", self.nside, self.lmax, self.lmax, mask,
                      _lib.PS_PREC_FP64 if prec == "fp64" else _lib.PS_PREC_MIXED, ctypes.byref(h))
        self._h = h
        self._ws = None
        self._ws_need = {}  # (batch, spin, adjoint) -> bytes; they depend on the tables
        # Legendre table format of a mixed plan: 'tf32x3' (FP32 values, split by the kernels) or
        # 'bf16x3' (BF16 hi + mid + lo planes in the tensor core's operand layout, 1.5x the bytes)
        if table_format is None:
            table_format = os.environ.get("PS_TABLE_FORMAT", "tf32x3")
        if table_format not in ("tf32x3", "bf16x3"):
            raise ValueError("table_format must be 'tf32x3' or 'bf16x3'")
        self.table_format = table_format
        if prec != "fp64":
            _lib.call("ps_plan_set_table_format", h, 1 if table_format == "bf16x3" else 0)
        # autotuning: tile shapes of this plan and, for mixed precision, an FP64 plan
        # beside it for the small-batch path
        self._h64 = None
        self._tuner = None
        if autotune:
            from .autotune import Tuner
            handles = {"fp64" if prec == "fp64" else "mixed": h}
            if prec != "fp64":
                h64 = ctypes.c_void_p()
                with torch.cuda.device(self.device):
                    rc = _lib.lib().ps_plan_create(self.nside, self.lmax, self.lmax, mask, _lib.PS_PREC_FP64,
                                                   ctypes.byref(h64))
                # an FP64 plan may be unsupported where the mixed one is not (at Nside 2048 the
                # FP64 Bluestein work arrays exceed shared memory): tune the mixed tiles only then
                if rc == _lib.PS_OK:
                    self._h64 = h64
                    handles["fp64"] = h64
                elif rc != _lib.PS_ERR_UNSUPPORTED:
                    _lib.check("ps_plan_create", rc)
            self._tuner = Tuner(self.nside, self.lmax, handles, self.device)
        # counters of transforms issued through this plan
        self.n_synthesis = 0
        self.n_adjoint = 0
        # Legendre tables: spins already tried (built or refused)
        self.tables = tables if prec != "fp64" else False
        self.table_fraction = float(table_fraction if table_fraction is not None
                                    else os.environ.get("PS_TABLE_MEM_FRACTION", 0.45))
        self._tab_tried = set()

    # ------------------------------------------------------------ Legendre tables
    def table_bytes(self, spin):
        n = ctypes.c_size_t()
        _lib.call("ps_plan_table_bytes", self._h, int(spin), ctypes.byref(n))
        return int(n.value)

    def has_table(self, spin):
        v = ctypes.c_int()
        _lib.call("ps_plan_has_table", self._h, int(spin), ctypes.byref(v))
        return bool(v.value)

    def build_table(self, spin, force=False):
        """Build the FP32 Legendre table of `spin` (mixed plans).  Without `force`, only when
        it fits in table_fraction of the free device memory; returns whether the plan has it."""
        spin = int(spin)
        if self.prec == "fp64":
            return False
        if self.has_table(spin):
            return True
        need = self.table_bytes(spin)
        with torch.cuda.device(self.device):
            free, _ = torch.cuda.mem_get_info()
            if not force and need > self.table_fraction * free:
                torch.cuda.empty_cache()
                free, _ = torch.cuda.mem_get_info()
                if need > self.table_fraction * free:
                    return False
            rc = _lib.lib().ps_plan_build_table(self._h, spin, self._stream())
            if rc == _lib.PS_ERR_NOMEM:
                torch.cuda.empty_cache()
                rc = _lib.lib().ps_plan_build_table(self._h, spin, self._stream())
            if rc == _lib.PS_ERR_NOMEM and not force:
                return False
            _lib.check("ps_plan_build_table", rc)
        self._ws_need.clear()
        return True

    def drop_tables(self):
        _lib.call("ps_plan_drop_tables", self._h)
        self._ws_need.clear()
        self._tab_tried.clear()

    def _maybe_table(self, spin):
        if self.tables is False or spin in self._tab_tried:
            return
        self._tab_tried.add(spin)
        self.build_table(spin, force=self.tables is True)

    def __del__(self):
        for name in ("_h", "_h64"):
            h = getattr(self, name, None)
            if h is not None and h.value and _lib._lib is not None:
                _lib.lib().ps_plan_destroy(h)
                setattr(self, name, None)

    # ------------------------------------------------------------ autotuning
    def _pick(self, key, run):
        """Plan handle for `key` = (direction, spin, batch); `run(handle)` issues the
        transform.  With autotuning, the first call of a key times every pipeline and
        tile shape (polyspec_b200.autotune)."""
        if self._tuner is None:
            return self._h
        direction, spin, B = key
        table = self.prec != "fp64" and self.has_table(spin)
        return self._tuner.select(0 if direction == "synthesis" else 1, spin, B, run, table=table)

    def error_flag(self, reset=True):
        """Device error flag of the plan (set by a kernel whose bounded wait expired)."""
        v = ctypes.c_int()
        _lib.call("ps_plan_error_flag", self._h, ctypes.byref(v), int(reset))
        return int(v.value)

    # ------------------------------------------------------------ workspace
    def workspace(self, batch, spin, adjoint):
        key = (int(batch), int(spin), int(adjoint))
        need = self._ws_need.get(key)
        if need is None:
            need = 0
            for h in (self._h, self._h64):
                if h is None:
                    continue
                n = ctypes.c_size_t()
                _lib.call("ps_sht_workspace_bytes", h, *key, ctypes.byref(n))
                need = max(need, int(n.value))
            self._ws_need[key] = need
        if self._ws is None or self._ws.numel() < need:
            self._ws = torch.empty(max(need, 256), dtype=torch.uint8, device=self.device)
        return self._ws, need

    def _joint(self, B):
        # T and (Q, U) in one call (ps_synthesis_fields): FP64 plans, while a spin's rings do not fill the device by
        # themselves; more maps gain less and would hold the phases of both spins at once
        return self.prec == "fp64" and B <= 4

    def _joint_workspace(self, B):
        need = self._ws_need.get(B)
        if need is None:
            n = ctypes.c_size_t()
            _lib.call("ps_fields_workspace_bytes", self._h, B, ctypes.byref(n))
            need = self._ws_need[B] = int(n.value)
        if self._ws is None or self._ws.numel() < need:
            self._ws = torch.empty(need, dtype=torch.uint8, device=self.device)
        return self._ws, need

    @staticmethod
    def _stream():
        # the current stream's handle, without building a torch.cuda.Stream (4 us a call)
        return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())

    def _check_alm(self, alm, spin):
        ncomp = 1 if spin == 0 else 2
        if alm.dtype != torch.complex128 or not alm.is_cuda:
            raise TypeError("alm must be a complex128 CUDA tensor")
        if alm.shape[-1] != self.nalm:
            raise ValueError("Wrong number of alm coefficients!")
        if spin > 0 and (alm.dim() < 2 or alm.shape[-2] != 2):
            raise ValueError("spin > 0 needs alm[..., 2, nalm] (G, C)")
        lead = alm.shape[:-2] if spin > 0 else alm.shape[:-1]
        B = 1
        for d in lead:
            B *= int(d)
        return lead, B, ncomp

    @staticmethod
    def _maps_in(t, nf, n):
        """(tensor, stride) of an input [..., n] (nf = 1) or [..., nf, n] for the strided entry points: read
        in place where each map's fields are contiguous and the maps lie at one stride, else copied."""
        if t.is_conj():
            t = t.resolve_conj()
        if t.is_neg():
            t = t.resolve_neg()
        if t.is_contiguous():
            return t, nf * n
        if (t.dim() == (2 if nf == 1 else 3) and t.stride(-1) == 1 and (nf == 1 or t.stride(-2) == n)
                and t.stride(0) >= nf * n):
            return t, t.stride(0)
        return t.contiguous(), nf * n

    def _synthesis_call(self, spin, B, alm, alm_stride, out, map_stride):
        """run(handle): synthesis of B maps at the addresses and strides of ps_synthesis_strided."""
        ws, nbytes = self.workspace(B, spin, 0)

        def run(h):
            _lib.call("ps_synthesis_strided", h, alm, alm_stride, out, map_stride, B, spin, ws.data_ptr(), nbytes,
                      self._stream())
        return run

    def _issue_synthesis(self, spin, B, alm, alm_stride, out, map_stride):
        self._maybe_table(spin)
        run = self._synthesis_call(spin, B, alm, alm_stride, out, map_stride)
        run(self._pick(("synthesis", spin, B), run))
        self.n_synthesis += B

    def _adjoint_call(self, spin, B, map, map_stride, out, alm_stride, scale):
        """run(handle): adjoint of B maps at the addresses and strides of ps_adjoint_strided."""
        ws, nbytes = self.workspace(B, spin, 1)

        def run(h):
            _lib.call("ps_adjoint_strided", h, map, map_stride, out, alm_stride, B, spin, float(scale), ws.data_ptr(),
                      nbytes, self._stream())
        return run

    def _issue_adjoint(self, spin, B, map, map_stride, out, alm_stride, scale):
        self._maybe_table(spin)
        run = self._adjoint_call(spin, B, map, map_stride, out, alm_stride, scale)
        run(self._pick(("adjoint", spin, B), run))
        self.n_adjoint += B

    def synthesis(self, alm, spin=0):
        spin = int(spin)
        lead, B, ncomp = self._check_alm(alm, spin)
        alm, stride = self._maps_in(alm, ncomp, self.nalm)
        shape = tuple(lead) + ((2,) if spin > 0 else ()) + (self.npix,)
        out = torch.empty(shape, dtype=torch.float64, device=alm.device)
        if B > 0:
            self._issue_synthesis(spin, B, alm.data_ptr(), stride, out.data_ptr(), 0)
        return out

    def synthesis_fields(self, alm, out):
        """alm [B, nf, nalm] -> out [B, nf, npix]: T (spin 0) and, of three fields, (E, B) -> (Q, U), read
        and written where they lie."""
        self._check_alm(alm, 0)
        B, nf = alm.shape[0], alm.shape[1]
        alm, stride = self._maps_in(alm, nf, self.nalm)
        if B > 0:
            a, o = alm.data_ptr(), out.data_ptr()
            if nf == 3 and self._joint(B):
                self._pick(("synthesis", 0, B), lambda h: self._synthesis_call(0, B, a, stride, o, 3 * self.npix)(h))
                self._pick(("synthesis", 2, B), lambda h: self._synthesis_call(
                    2, B, a + 16 * self.nalm, stride, o + 8 * self.npix, 3 * self.npix)(h))
                ws, nbytes = self._joint_workspace(B)
                _lib.call("ps_synthesis_fields", self._h, a, stride, o, 3 * self.npix, B, ws.data_ptr(), nbytes,
                          self._stream())
                self.n_synthesis += 2 * B
                return
            self._issue_synthesis(0, B, a, stride, o, nf * self.npix)
            if nf == 3:
                self._issue_synthesis(2, B, a + 16 * self.nalm, stride, o + 8 * self.npix, nf * self.npix)

    def synthesis_pm(self, alm, spin):
        """(+s, -s) maps [2, n, npix] (complex128) of the spin-s transform of (G, C) = (-alm, 0), alm [n, nalm]."""
        spin = int(spin)
        self._check_alm(alm, 0)
        if alm.dim() != 2:
            raise ValueError("alm must be [n, nalm]")
        alm, _ = self._maps_in(alm.contiguous(), 1, self.nalm)
        B = alm.shape[0]
        out = torch.empty((2, B, self.npix), dtype=torch.complex128, device=alm.device)
        if B > 0:
            self._maybe_table(spin)
            ws, nbytes = self.workspace(B, spin, 0)

            def run(h):
                _lib.call("ps_synthesis_pm", h, alm.data_ptr(), out.data_ptr(), out.data_ptr() + 16 * B * self.npix, B,
                          spin, ws.data_ptr(), nbytes, self._stream())
            # the FP64 kernels follow a rule of their own here, a mixed plan has two pipelines to choose from
            run(self._h if self.prec == "fp64" else self._pick(("synthesis", spin, B), run))
            self.n_synthesis += B
        return out

    def weighted_roundtrip(self, alm, weight, lscale=None, scale=1.0, out=None):
        """Fused  out = scale * lscale * Y^H W Y (lscale * alm)  for every field of alm [B, nf, nalm]
        (nf = 1: T, spin 0; nf = 3: T spin 0 and (E, B) spin 2), weight [nf, npix] float64,
        lscale [nf, nalm] float64 or None (ps_sht_weighted_roundtrip: the maps stay in shared
        memory).  Returns None when a spin lacks its Legendre table (the caller composes
        synthesis, weight and adjoint instead)."""
        if self.prec == "fp64" or alm.dim() != 3 or alm.shape[1] not in (1, 3):
            return None
        B, nf = alm.shape[0], alm.shape[1]
        spins = [(0, 0)] if nf == 1 else [(0, 0), (2, 1)]
        for spin, _ in spins:
            self._maybe_table(spin)
            if not self.has_table(spin):
                return None
        alm = alm.contiguous()
        if out is None:
            out = torch.empty_like(alm)
        w = weight.contiguous()
        ls = lscale.contiguous() if lscale is not None else None
        for spin, c0 in spins:
            n = ctypes.c_size_t()
            _lib.call("ps_roundtrip_workspace_bytes", self._h, B, spin, ctypes.byref(n))
            if self._ws is None or self._ws.numel() < n.value:
                self._ws = torch.empty(max(n.value, 256), dtype=torch.uint8, device=self.device)
            off = c0 * self.nalm * 16
            _lib.call("ps_sht_weighted_roundtrip", self._h, ctypes.c_void_p(alm.data_ptr() + off),
                      ctypes.c_void_p(out.data_ptr() + off), nf * self.nalm, B, spin,
                      ctypes.c_void_p(w.data_ptr() + c0 * self.npix * 8),
                      ctypes.c_void_p(ls.data_ptr() + c0 * self.nalm * 8) if ls is not None else ctypes.c_void_p(0),
                      float(scale), ctypes.c_void_p(self._ws.data_ptr()), self._ws.numel(), self._stream())
        self.n_synthesis += B * len(spins)
        self.n_adjoint += B * len(spins)
        return out

    def _check_map(self, map, spin):
        if map.dtype != torch.float64 or not map.is_cuda:
            raise TypeError("map must be a float64 CUDA tensor")
        if map.shape[-1] != self.npix:
            raise ValueError("map has %d pixels, expected %d" % (map.shape[-1], self.npix))
        if spin > 0 and (map.dim() < 2 or map.shape[-2] != 2):
            raise ValueError("spin > 0 needs map[..., 2, npix] (Q, U)")
        lead = map.shape[:-2] if spin > 0 else map.shape[:-1]
        B = 1
        for d in lead:
            B *= int(d)
        return lead, B, 1 if spin == 0 else 2

    def adjoint(self, map, spin=0, scale=1.0, out=None):
        spin = int(spin)
        lead, B, ncomp = self._check_map(map, spin)
        map, stride = self._maps_in(map, ncomp, self.npix)
        shape = tuple(lead) + ((2,) if spin > 0 else ()) + (self.nalm,)
        if out is None:
            out = torch.empty(shape, dtype=torch.complex128, device=map.device)
        elif (tuple(out.shape) != shape or out.dtype != torch.complex128 or out.device != map.device
              or not out.is_contiguous() or out.is_conj()):
            raise ValueError("out must be a contiguous complex128 tensor of shape %s" % (shape,))
        if B > 0:
            self._issue_adjoint(spin, B, map.data_ptr(), stride, out.data_ptr(), 0, scale)
        return out

    def adjoint_fields(self, maps, out, scale=1.0):
        """maps [B, nf, npix] -> out [B, nf, nalm]: T (spin 0) and, of three fields, (Q, U) -> (E, B), read
        and written where they lie."""
        self._check_map(maps, 0)
        B, nf = maps.shape[0], maps.shape[1]
        maps, stride = self._maps_in(maps, nf, self.npix)
        if B > 0:
            m, o = maps.data_ptr(), out.data_ptr()
            if nf == 3 and self._joint(B):
                self._pick(("adjoint", 0, B), lambda h: self._adjoint_call(0, B, m, stride, o, 3 * self.nalm, scale)(h))
                self._pick(("adjoint", 2, B), lambda h: self._adjoint_call(
                    2, B, m + 8 * self.npix, stride, o + 16 * self.nalm, 3 * self.nalm, scale)(h))
                ws, nbytes = self._joint_workspace(B)
                _lib.call("ps_adjoint_fields", self._h, m, stride, o, 3 * self.nalm, B, float(scale), ws.data_ptr(),
                          nbytes, self._stream())
                self.n_adjoint += 2 * B
                return
            self._issue_adjoint(0, B, m, stride, o, nf * self.nalm, scale)
            if nf == 3:
                self._issue_adjoint(2, B, m + 8 * self.npix, stride, o + 16 * self.nalm, nf * self.nalm, scale)

    def adjoint_pm(self, plus, minus, spin, scale=1.0):
        """(+s, -s) harmonics [2, n, nalm] of the complex maps plus, minus [n, npix] (ps_adjoint_pm)."""
        spin = int(spin)
        for t in (plus, minus):
            if t.dtype != torch.complex128 or not t.is_cuda:
                raise TypeError("maps must be complex128 CUDA tensors")
            if t.dim() != 2 or t.shape[-1] != self.npix or t.shape != plus.shape:
                raise ValueError("maps of shape %s, expected [n, %d] twice" % (tuple(t.shape), self.npix))
        plus, _ = self._maps_in(plus.contiguous(), 1, self.npix)
        minus, _ = self._maps_in(minus.contiguous(), 1, self.npix)
        B = plus.shape[0]
        out = torch.empty((2, B, self.nalm), dtype=torch.complex128, device=plus.device)
        if B > 0:
            self._maybe_table(spin)
            ws, nbytes = self.workspace(B, spin, 1)
            gc = torch.empty_like(out)

            def run(h):
                _lib.call("ps_adjoint_pm", h, plus.data_ptr(), minus.data_ptr(), gc.data_ptr(), out.data_ptr(),
                          out.data_ptr() + 16 * B * self.nalm, B, spin, float(scale), ws.data_ptr(), nbytes,
                          self._stream())
            run(self._pick(("adjoint", spin, B), run))
            self.n_adjoint += B
        return out
