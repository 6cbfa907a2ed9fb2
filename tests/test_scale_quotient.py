"""The scale pass forms RN_fp32(s / unit) (quant.py:21-23) from the reciprocal of the unit in two parts and one correction
by the exact remainder (fp4_post_b200/csrc/quantize.cu, scale_bytes4).  The same operations in C, against the division, on
random pairs and on pairs whose quotient lies on an E4M3 tie or next to one."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from test_scale_fast_path import _pairs

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


@pytest.mark.parametrize("kind", [0, 1, 2])
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


def test_units_whose_reciprocals_have_a_subnormal_second_part(quotient):
    rng = np.random.default_rng(3)
    smax = np.exp(rng.uniform(np.log(1e30), np.log(5.6e37), size=6000)).astype(np.float32).repeat(1000)      # the largest scale of a finite maximum is 5.67e37
    unit = (smax / np.float32(448.0)).astype(np.float32)
    s = np.maximum((smax * rng.uniform(0, 1, size=smax.size).astype(np.float32)).astype(np.float32), np.float32(1e-9))
    assert np.array_equal(quotient(s, unit), (s / unit).astype(np.float32))


def test_what_is_not_a_number_stays_so(quotient):
    """An infinite maximum gives a scale and a unit that are NaN, and so does a pass that gave up on a load: every byte is NaN then."""
    nan = np.float32("nan")
    s, unit = np.array([nan, 1.0, 1e-9, nan], np.float32), np.array([1.0, nan, nan, nan], np.float32)
    assert np.isnan(quotient(s, unit)).all()
