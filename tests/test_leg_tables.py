"""Coefficients of the FP64 Legendre recurrences against the closed forms in 50 digits: c_l, d_l and gam_l of the chain
that the plan's tables are made from.

Tolerance 1.2e-16 relative: each is rounded once (2^-53 = 1.1e-16), the chain's own errors are of order l 2^-104.
"""
import ctypes
import decimal
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def chain(tmp_path_factory):
    d = tmp_path_factory.mktemp("leg")
    (d / "t.cpp").write_text('#include "ps_legtab.h"\nextern "C" void chain(int m, int s, int n, double* o) {\n'
                             '  ps::LegChain t(m, s);\n  for (int i = 0; i < n; ++i, t.step()) '
                             't.values(o[3 * i], o[3 * i + 1], o[3 * i + 2]);\n}\n')
    subprocess.check_call(["g++", "-O2", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "polyspec_b200", "csrc"),
                           str(d / "t.cpp"), "-o", str(d / "t.so")])
    lib = ctypes.CDLL(str(d / "t.so"))

    def f(m, s, n):
        out = np.empty((n, 3))
        lib.chain(m, s, n, out.ctypes.data_as(ctypes.c_void_p))
        return out
    return f


@pytest.mark.parametrize("m,s", [(0, 0), (1, 0), (2, 0), (7, 0), (100, 0), (2047, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2),
                                 (3, 2), (900, 2), (0, 3), (5, 3), (3071, 3)])
def test_chain(chain, m, s):
    decimal.getcontext().prec = 50
    D = decimal.Decimal
    n, l0 = 3000, max(m, s)
    got = chain(m, s, n)

    def rho2(x):
        return D((x * x - m * m) * (x * x - s * s))

    def A2(x):  # squared coefficient of the step from x to x + 1 (spin 0: a_{x+1}^2)
        return D((2 * x + 3) * (2 * x + 1) * (x + 1) ** 2) / rho2(x + 1)
    gam = [D(1), D(1)]
    A = [A2(l0).sqrt()]
    for i in range(n):
        lam = l0 + i
        if i > 0:
            A.append(A2(lam).sqrt())
            gam.append(A[i] / A[i - 1] * gam[i - 1])
        c = A[i] * gam[i] / gam[i + 1]
        d = c * m * s / (lam * (lam + 1)) if s else D(0)
        for have, want in zip(got[i], (c, d, gam[i])):
            assert abs(D(float(have)) - want) <= D("1.2e-16") * abs(want)
