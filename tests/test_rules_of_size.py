"""Rules of size of the quantizers and the fused norm (fp4_post_b200/csrc/rows_shape.cuh), compiled with the host compiler: both sides of
each line as they were timed."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fp4_post_b200" / "csrc"
PROGRAM = """
#include "rows_shape.cuh"
extern "C" int staged(int64_t rows, int64_t cols, int fp32_gamma, int norm) {
  return metis::norm_rows_staged(rows, cols / 16, fp32_gamma != 0, norm != 0, cols % 64 == 0);
}
extern "C" int ctas(int64_t rows, int64_t cols, int fp32, int mean, int rows_out, int cols_out) {
  const int64_t pitch = cols * (fp32 ? 4 : 2);
  return metis::tile_ctas_per_sm(rows * pitch, pitch % 128 != 0, mean != 0, fp32 != 0, rows_out != 0, cols_out != 0);
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "rules.cpp"), "-o", str(d / "rules.so")], check=True)
    L = C.CDLL(str(d / "rules.so"))
    L.staged.argtypes = [C.c_int64, C.c_int64, C.c_int, C.c_int]
    L.ctas.argtypes = [C.c_int64, C.c_int64] + [C.c_int] * 4
    return L


# rows, columns, fp32 gamma, norm written -> whether the row in shared memory was the faster one of the two
@pytest.mark.parametrize("call,staged", [((65536, 512, 0, 0), 0), ((16383, 1024, 0, 0), 0), ((16384, 528, 0, 0), 1), ((1024, 1040, 0, 0), 1), ((65536, 4096, 0, 0), 1),
                                         ((3000, 2560, 0, 1), 0), ((1300, 2576, 0, 1), 1), ((2048, 1552, 0, 0), 0), ((2048, 3584, 0, 0), 1), ((3400, 1552, 0, 0), 1), ((65536, 2560, 0, 1), 0), ((4096, 1088, 0, 1), 0), ((16384, 1088, 0, 1), 1),
                                         ((16384, 1232, 0, 1), 0), ((6000, 3584, 0, 1), 1), ((8192, 3584, 0, 1), 0), ((8192, 4096, 0, 1), 1), ((12000, 4096, 0, 1), 0),
                                         ((1300, 2048, 1, 0), 1), ((6000, 2048, 1, 0), 0), ((12000, 2064, 1, 0), 0), ((4096, 2576, 1, 0), 1), ((16384, 1536, 1, 0), 1),
                                         ((16384, 1552, 1, 0), 0), ((32768, 2048, 1, 1), 1), ((32768, 2064, 1, 1), 0), ((8192, 4080, 1, 1), 1), ((16384, 1232, 1, 1), 1)])
def test_the_faster_place_for_a_row(rules, call, staged):
    assert rules.staged(*call) == staged


# rows, columns, fp32, mean, row-major output, transposed output -> the faster number of CTAs per SM
@pytest.mark.parametrize("call,ctas", [((65536, 4096, 0, 0, 1, 1), 3), ((11680, 4112, 0, 0, 1, 0), 3), ((15568, 4112, 0, 0, 1, 0), 2), ((54192, 8304, 0, 0, 1, 0), 2),
                                       ((23360, 4112, 0, 1, 1, 0), 3), ((31136, 4112, 0, 1, 1, 0), 2), ((15568, 4112, 1, 1, 1, 0), 2), ((15568, 4112, 0, 0, 0, 1), 2),
                                       ((31136, 4112, 0, 1, 0, 1), 2), ((7712, 8304, 1, 1, 0, 1), 3), ((15056, 8304, 1, 1, 0, 1), 2), ((11680, 4112, 0, 1, 1, 1), 3),
                                       ((15568, 4112, 0, 0, 1, 1), 2), ((23360, 4112, 0, 1, 1, 1), 2), ((21088, 8304, 0, 0, 1, 1), 1), ((54192, 8304, 0, 1, 1, 1), 2)])
def test_the_faster_number_of_tile_ctas(rules, call, ctas):
    assert rules.ctas(*call) == ctas
