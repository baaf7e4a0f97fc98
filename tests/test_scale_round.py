"""CPU: scale_round, the FP32 products' v * weight * factor rounded to FP32
once, against the same in FP64 (the form it replaces), compiled for the host.

Bar: two roundings to FP32, 2^-23 of the value, and one unit of the smallest
subnormal (the double-float form is within the last rounding of the exact
product, the FP64 form rounds a value within 2^-51 of it).
"""
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not shutil.which("g++") or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = str(tmp_path_factory.mktemp("cpp") / "scale_round_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(CUDA, "include"),
                    "-I", os.path.join(ROOT, "latttmat_gb300", "csrc"), "-I", os.path.join(ROOT, "tests", "cpp"),
                    os.path.join(ROOT, "tests", "cpp", "scale_round_check.cpp"), "-o", out], check=True)
    return out


def run(exe, kind, hi, lo, t, S):
    """scale_round and the FP64 form of the same values"""
    lines = ["%d %s %s %s %s" % (kind, float(a).hex(), float(b).hex(), float(c).hex(), float(S).hex())
             for a, b, c in zip(hi, lo, t)]
    r = subprocess.run([exe], input="\n".join(lines) + "\n", capture_output=True, text=True, check=True)
    got = np.array([float.fromhex(v) if "n" not in v else float(v) for v in r.stdout.split()])
    with np.errstate(all="ignore"):
        want = ((hi.astype(np.float64) + lo.astype(np.float64)) * t * S).astype(np.float32).astype(np.float64)
    return got, want


def values(seed, kind, vexp, texp, n=400):
    r = np.random.default_rng(seed)
    v = np.ldexp(r.uniform(-1, 1, n), r.integers(-vexp, vexp + 1, n))
    t = np.ldexp(r.uniform(0.5, 1, n), r.integers(-texp, texp + 1, n))
    hi = v.astype(np.float32)
    lo = (v - hi).astype(np.float32) if kind else np.zeros_like(hi)
    hi[:3], lo[:3] = 0.0, 0.0
    return hi, lo, t


def check(got, want):
    fin = np.isfinite(want)
    assert np.array_equal(np.isnan(got), np.isnan(want))
    assert np.array_equal(got[~fin & ~np.isnan(want)], want[~fin & ~np.isnan(want)])
    assert np.all(np.abs(got[fin] - want[fin]) <= 2.0 ** -23 * np.abs(want[fin]) + 2.0 ** -149)


# the factor is held as two FP32 words inside 2^-120 .. 2^120, and as FP64 alone outside
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("S", [1.0, 3.1, 2.0 ** -119, 2.0 ** -121, 2.0 ** -122 * 1.3, 2.0 ** 119, 2.0 ** 121, 1e-60,
                               1e60, 1e-300, 1e300, 0.0, -2.5, np.inf])
def test_factor_range(exe, kind, S):
    # values and weights that bring the result back into the FP32 range, and those that leave it
    e = int(np.clip(np.frexp(S)[1], -140, 140)) if np.isfinite(S) else 0
    for seed, (vexp, texp, shift) in enumerate([(3, 3, 0), (20, 30, 0), (10, 10, -e // 2), (60, 60, -e // 2)]):
        hi, lo, t = values(seed, kind, vexp, texp)
        sh = int(np.clip(shift, -60, 60))
        hi, lo, t = np.ldexp(hi, sh), np.ldexp(lo, sh), np.ldexp(t, shift)
        # (an overflow of the two-word form near the largest FP32 value is another test's)
        with np.errstate(all="ignore"):
            y = np.abs((hi.astype(np.float64) + lo) * t * S)
        keep = ~((y > 1e37) & np.isfinite(y) & (2.0 ** -120 < S) & (S < 2.0 ** 120))
        check(*run(exe, kind, hi[keep], lo[keep], t[keep], S))


# a factor inside the range whose product with the value leaves it, at both ends: infinities as FP64 rounds them
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("S", [1e30, 1e35, 2.0 ** 118, 1e25, 1.0, 1e-25, 1e-35, 2.0 ** -118])
def test_results_at_the_ends(exe, kind, S):
    for seed, end in enumerate((2.0 ** 127, 2.0 ** 128, 2.0 ** 129, 1e45, 2.0 ** -110, 2.0 ** -126, 2.0 ** -140, 1e-50)):
        r = np.random.default_rng(seed)
        t = np.ldexp(r.uniform(0.5, 1, 400), r.integers(-30, 31, 400))
        v = np.clip(end * r.uniform(0.5, 1.5, 400) / (S * t), 1e-36, 3e38) * r.choice([-1.0, 1.0], 400)
        hi = v.astype(np.float32)
        lo = (v - hi).astype(np.float32) if kind else np.zeros_like(hi)
        check(*run(exe, kind, hi, lo, t, S))


def test_infinite_and_nan_values(exe):
    hi = np.array([np.inf, -np.inf, np.nan, 5e8, 1e4], dtype=np.float32)
    for S in (1.0, 1e30, 1e35, 1e-35, 1e60):
        check(*run(exe, 0, hi, np.zeros_like(hi), np.ones(5), S))


# small values under large weights and small factors: the value times the factor's power of two is subnormal
@pytest.mark.parametrize("kind", [0, 1])
def test_subnormal_partial_products(exe, kind):
    r = np.random.default_rng(0)
    for S in (2.0 ** -80, 2.0 ** -118, 2.0 ** -40):
        v = np.ldexp(r.uniform(-1, 1, 400), r.integers(-125, -60, 400))
        t = np.ldexp(r.uniform(0.5, 1, 400), r.integers(40, 91, 400))
        hi = v.astype(np.float32)
        lo = (v - hi).astype(np.float32) if kind else np.zeros_like(hi)
        check(*run(exe, kind, hi, lo, t, S))


@pytest.mark.parametrize("vexp,texp", [(3, 3), (30, 40), (120, 60), (126, 100), (60, 900)])
def test_without_factor(exe, vexp, texp):
    hi, lo, t = values(vexp, 0, vexp, texp)
    hi[5:9] = np.inf, -np.inf, np.nan, 0.0
    t[8:10] = np.inf, 0.0
    check(*run(exe, 2, hi, lo, t, 1.0))
