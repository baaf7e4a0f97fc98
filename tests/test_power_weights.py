"""CPU: the weights of the adjoint's quadratic form against exact rational
arithmetic in the exactly known 2 cosh K, 2 sinh K to 60 digits.

Bar 8e-16: two powers (one unit in the last place each), three products, one
sum, the correction factor and the scaling (half a unit each): 2 * 2.2e-16 +
3 * 1.1e-16.  Powers of the rounded 2 cosh K alone are off by up to L / 2 units
(3e-15 at L = 30).
"""
import os
import shutil
import subprocess
from decimal import Decimal, getcontext

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def exact(K, L):
    getcontext().prec = 60
    e = Decimal(K).exp()
    c, s = e + 1 / e, e - 1 / e
    def power(x, n):
        return Decimal(1) if n == 0 else x ** n
    out = []
    for k in range(L + 1):
        r = Decimal(0)
        if k < L:
            r += (L - k) * power(c, L - k - 1) * power(s, k + 1)
        if k > 0:
            r += k * power(c, L - k + 1) * power(s, k - 1)
        out.append(r / 2 ** L)
    return out


def test_against_exact(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("needs g++")
    exe = str(tmp_path / "power_weights_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "latttmat_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "power_weights_check.cpp"), "-o", exe], check=True)
    rng = np.random.default_rng(0)
    pts = [(float(K), int(L)) for K, L in zip(rng.uniform(0.2, 0.9, 20), rng.integers(4, 31, 20))]
    pts += [(-0.37, 24), (1.7, 30), (0.0, 12), (1e-3, 16), (-2.5, 31)]
    r = subprocess.run([exe], input="".join("%s %d\n" % (K.hex(), L) for K, L in pts), capture_output=True, text=True,
                       check=True)
    for (K, L), line in zip(pts, r.stdout.splitlines()):
        got = [float.fromhex(t) for t in line.split()]
        assert len(got) == L + 1
        for g, w in zip(got, exact(K, L)):
            assert (g == 0.0 and w == 0) or abs(Decimal(g) - w) <= Decimal(8e-16) * abs(w), (K, L)
