"""The FP32 velocity factor formed from FP32 pairs against the FP64 product's rounding.

Whatever the function settles has to be float((m p) f) bit for bit: random operands over all magnitudes, products on and
beside the rounding boundaries of FP32 (where it must not settle wrongly), and operands out of range, zero,
negative, infinite or NaN (which it has to leave to the caller).
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HEADER = Path(__file__).resolve().parent.parent / "score_gb300" / "csrc" / "velocity32.h"
SRC = """
#include "velocity32.h"
extern "C" void run(const uint64_t* m, const uint64_t* p, const uint32_t* code, float* v, unsigned char* ok, long n) {
    for (long i = 0; i < n; ++i) ok[i] = score::velocity32(m[i], p[i], code[i], v[i]);
}
"""
FACE, CORNER = {4, 10, 12, 13, 15, 21, 26}, {0, 2, 6, 8, 17, 19, 23, 25}
SF = np.array([1.0 if c in FACE else 0.6494 if c in CORNER else 0.7957 for c in range(27)])


@pytest.fixture(scope="module")
def settle(tmp_path_factory):
    d = tmp_path_factory.mktemp("velocity32")
    (d / "v.cpp").write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC", f"-I{HEADER.parent}", "-o", d / "v.so", d / "v.cpp"],
                   check=True)
    lib = C.CDLL(str(d / "v.so"))

    def run(m, p, code):
        m, p, code = (np.ascontiguousarray(x) for x in (m, p, code.astype(np.uint32)))
        v, ok = np.empty(m.size, np.float32), np.empty(m.size, np.uint8)
        lib.run(*(C.c_void_p(x.ctypes.data) for x in (m, p, code, v, ok)), C.c_long(m.size))
        return v, ok.astype(bool)

    return run


def check(settle, m, p, code, least):
    v, ok = settle(m, p, code)
    with np.errstate(over="ignore", under="ignore", invalid="ignore"):
        ref = ((m * p) * SF[code]).astype(np.float32)
    assert np.array_equal(v[ok].view(np.uint32), ref[ok].view(np.uint32))
    assert ok.mean() >= least
    return ok


@pytest.mark.parametrize("lo, hi, least", [(-14, -8, 0.999), (-24, 10, 0.9), (-300, 300, 0.0)])
def test_random_products(settle, lo, hi, least):
    rng = np.random.default_rng(5)
    n = 2_000_000
    m = 10.0 ** rng.uniform(lo, hi, n)
    p = 10.0 ** rng.uniform(4, 8, n)
    check(settle, m, p, rng.integers(0, 27, n), least)


@pytest.mark.parametrize("code", [26, 18, 0])
def test_rounding_boundaries(settle, code):
    """Products within a few units of the FP64 product's last place of the middle between two FP32 numbers."""
    rng = np.random.default_rng(6)
    n = 400_000
    mid = (rng.integers(1 << 23, 1 << 24, n).astype(np.float64) + 0.5) * 2.0 ** rng.integers(-60, -20, n)
    p = 10.0 ** rng.uniform(4, 8, n)
    m = mid / (p * SF[code])
    m = m.view(np.uint64) + rng.integers(-4, 5, n).astype(np.uint64)
    ok = check(settle, m.view(np.float64), p, np.full(n, code), 0.0)
    assert ok.mean() < 0.01
    # the same at some distance, on both sides of the margin
    m = m + (rng.integers(-1 << 14, 1 << 14, n)).astype(np.uint64)
    check(settle, m.view(np.float64), p, np.full(n, code), 0.0)


def test_left_to_the_caller(settle):
    bad = np.array([0.0, -0.0, -1e-10, np.inf, -np.inf, np.nan, 5e-324, 1e-300, 1e300])
    good = np.full(bad.size, 1e6)
    code = np.full(bad.size, 12)
    assert not settle(bad, good, code)[1].any() and not settle(good, bad, code)[1].any()
    ext = np.array([2.0**-91, 2.0**91, 2.0**-90, 2.0**89])
    check(settle, ext, np.full(4, 1e6), np.full(4, 3), 0.0)
