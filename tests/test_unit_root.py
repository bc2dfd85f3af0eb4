"""The plan's roots of unity e^{i pi q / den} against 80-bit numbers, over ring lengths, chirp indices and signs.

Tolerance 1.3e-16: cos and sin to 0.55 ulp of values below one (6e-17) and the rounding of the sum that corrects
them (5.6e-17), with the second order of the correction far below.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def root(tmp_path_factory):
    d = tmp_path_factory.mktemp("unit")
    (d / "u.cpp").write_text('#include "ps_unit.h"\nextern "C" void unit(const int64_t* q, int64_t n, int64_t den, double* '
                             'o) {\n  for (int64_t i = 0; i < n; ++i) ps::unit_root(q[i], den, o[2 * i], o[2 * i + 1]);\n}\n')
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "polyspec_b200", "csrc"),
                           str(d / "u.cpp"), "-o", str(d / "u.so")])
    lib = ctypes.CDLL(str(d / "u.so"))

    def f(q, den):
        q = np.ascontiguousarray(q, dtype=np.int64)
        out = np.empty((len(q), 2))
        lib.unit(q.ctypes.data_as(ctypes.c_void_p), ctypes.c_int64(len(q)), ctypes.c_int64(den),
                 out.ctypes.data_as(ctypes.c_void_p))
        return out
    return f


@pytest.mark.parametrize("den", [1, 2, 3, 4, 8, 12, 20, 512, 1020, 4092, 4096, 8188, 16384])
def test_roots(root, den):
    pi = np.longdouble("3.14159265358979323846264338327950288")
    j = np.arange(-2 * den, 2 * den + 1)
    for q in (j, j * np.abs(j), j + (1 << 40) * 2 * den):
        got = root(q, den)
        a = pi * (q % (2 * den)).astype(np.longdouble) / den
        for k, want in enumerate((np.cos(a), np.sin(a))):
            assert float(np.abs(got[:, k] - want).max()) < 1.3e-16
    for q, w in ((0, (1, 0)), (den, (-1, 0)), (-den, (-1, 0)), (2 * den, (1, 0))):
        assert tuple(root([q], den)[0]) == w
    if den % 2 == 0:
        assert tuple(root([den // 2], den)[0]) == (0, 1) and tuple(root([-(den // 2)], den)[0]) == (0, -1)
