"""Launch shape of the row-major quantizer (fp4_post_b200/csrc/rows_shape.cuh), compiled with the host compiler: whatever the
tensor, the CTAs that leave a record are never more than the scratch has room for."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fp4_post_b200" / "csrc"
PROGRAM = """
#include "rows_shape.cuh"
extern "C" int max_records() { return metis::kMaxRecords; }
extern "C" void shape(int64_t rows, int64_t blocks, int64_t resident, int records, int64_t* out) {
  const metis::RowsShape s = metis::rows_shape(rows, blocks, resident, records != 0);
  out[0] = s.bx; out[1] = s.gx; out[2] = s.gy; out[3] = s.records;
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("rows_shape")
    (d / "shape.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "shape.cpp"), "-o", str(d / "shape.so")], check=True)
    L = C.CDLL(str(d / "shape.so"))
    L.shape.argtypes = [C.c_int64, C.c_int64, C.c_int64, C.c_int, C.POINTER(C.c_int64)]
    out = (C.c_int64 * 4)()

    def call(rows, blocks, resident=148 * 8, records=True):
        L.shape(rows, blocks, resident, int(records), out)
        return tuple(out)
    call.max_records = L.max_records()
    return call


@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5, 7, 8, 16, 31, 64])
def test_records_fit_for_every_width_the_kernel_takes(shape, rows):
    dropped = 0
    for blocks in range(1, 2 ** 16 // rows + 1):            # from 2^20 elements on the tile kernel takes over
        for resident in (148, 148 * 8):
            bx, gx, gy, records = shape(rows, blocks, resident)
            assert gx * bx >= blocks and (gx - 1) * bx < blocks and gy >= 1 and 256 % bx == 0
            assert not records or gx * gy <= shape.max_records, (rows, blocks)
            dropped += not records
    assert (dropped > 0) == (rows <= 3)                     # the fallback is reached, and by rows of that width only


def test_without_room_for_records_none_are_left(shape):
    for rows, blocks in ((1, 4), (300, 256), (65535, 16), (1, 65504)):
        assert not shape(rows, blocks, records=False)[3]


def test_large_grids_are_cut_to_the_records(shape):
    bx, gx, gy, records = shape(1 << 20, 3 * 256)           # rows of three CTAs, four waves of 1184 without records
    assert records and gx == 3 and gy == shape.max_records // 3
    assert shape(1 << 20, 3 * 256, records=False)[2] == 148 * 8 * 4 // 3
