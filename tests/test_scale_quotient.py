"""The scale pass forms RN_fp32(s / unit) (quant.py:21-23) from the reciprocal of the unit in two parts and one correction
by the exact remainder (fp4_post_b200/csrc/quantize.cu, scale_bytes4).  The same operations in C, against the division, on
random pairs and on pairs whose quotient lies on an E4M3 tie or next to one."""
import ctypes as C
import subprocess

import numpy as np
import pytest

PROGRAM = """
#include <math.h>
void quotient(const float* s, const float* unit, float* out, long n) {
  for (long i = 0; i < n; ++i) {
    const float y = 1.0f / unit[i], rest = fmaf(-unit[i], y, 1.0f) * y;
    const float q = fmaf(s[i], y, s[i] * rest);
    out[i] = fmaf(fmaf(-unit[i], q, s[i]), y, q);
  }
}
"""


@pytest.fixture(scope="module")
def quotient(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotient")
    (d / "q.c").write_text(PROGRAM)
    subprocess.run(["gcc", "-O2", "-ffp-contract=off", "-shared", "-fPIC", str(d / "q.c"), "-lm", "-o", str(d / "q.so")], check=True)
    f = C.CDLL(str(d / "q.so")).quotient
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_long]

    def call(s, unit):
        out = np.empty_like(s)
        f(s.ctypes.data, unit.ctypes.data, out.ctypes.data, s.size)
        return out
    return call


def _pairs(rng, kind: int, n: int):
    low, high = (1e30, 5.6e37) if kind == 3 else (1e-8, 1e30)            # the largest scale of a finite maximum is 5.67e37
    smax = np.exp(rng.uniform(np.log(low), np.log(high), size=n // 1000)).astype(np.float32).repeat(1000)
    unit = (smax / np.float32(448.0)).astype(np.float32)
    if kind == 0:        # block scales spread over six decades below the largest
        s = (smax * np.exp(rng.uniform(np.log(1e-6), 0, size=n)).astype(np.float32)).astype(np.float32)
    elif kind == 1:      # quotients on an E4M3 tie (normal and subnormal range), then up to 6 fp32 steps off it
        e, m = rng.integers(-9, 9, size=n), rng.integers(0, 8, size=n)
        tie = (1 + (m + 0.5) / 8) * np.exp2(e)
        s = (tie * unit.astype(np.float64)).astype(np.float32)
        s = (s.view(np.int32) + rng.integers(-6, 7, size=n).astype(np.int32)).view(np.float32)
    else:                # uniform below the largest (3: of those whose reciprocals' second parts are subnormal)
        s = (smax * rng.uniform(0, 1, size=n).astype(np.float32)).astype(np.float32)
    return np.minimum(np.maximum(s, np.float32(1e-9)), smax), unit


@pytest.mark.parametrize("kind", [0, 1, 2, 3])
def test_corrected_product_is_the_rounded_quotient(quotient, kind):
    rng = np.random.default_rng(kind)
    for _ in range(3):
        s, unit = (np.ascontiguousarray(t) for t in _pairs(rng, kind, 2_000_000))
        want = (s / unit).astype(np.float32)
        normal = want >= np.float32(2.0 ** -100)           # far below E4M3's smallest byte the remainder may underflow
        got = quotient(s, unit)
        assert np.array_equal(got[normal], want[normal])
        assert np.all(got[~normal] < 2.0 ** -20)


def test_maxima_of_bf16_tensors(quotient):
    """Every pair of bf16 mantissas: block maxima that sit exactly on E4M3 ties of the largest one's scale, in ten binades."""
    m = (np.arange(128, 256) / 128.0).astype(np.float32)
    top, a, e = np.meshgrid(m, m, np.exp2(-np.arange(10)).astype(np.float32), indexing="ij")
    keep = a * e <= top

    def scale(amax):
        return ((amax / np.float32(6)).astype(np.float32) + np.float32(1e-9)).astype(np.float32)
    s, unit = scale((a * e)[keep]), (scale(top[keep]) / np.float32(448)).astype(np.float32)
    assert np.array_equal(quotient(s, unit), (s / unit).astype(np.float32))


def test_what_is_not_a_number_stays_so(quotient):
    """An infinite maximum gives a scale and a unit that are NaN, and so does a pass that gave up on a load: every byte is NaN then."""
    nan = np.float32("nan")
    s, unit = np.array([nan, 1.0, 1e-9, nan], np.float32), np.array([1.0, nan, nan, nan], np.float32)
    assert np.isnan(quotient(s, unit)).all()
