"""Order in which the epilogue of the CTA-pair product drains its accumulators (fp4_post_b200/csrc/pair_drain.cuh), compiled with the
host compiler: however far one epilogue warp falls behind, no tile's products overwrite columns that it still has to read; and the
rule for the number of warps."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fp4_post_b200" / "csrc"
PROGRAM = """
#include "pair_drain.cuh"
using metis::PairDrain;
extern "C" int chunks() { return PairDrain::kChunks; }
extern "C" int stride() { return PairDrain::kStride; }
extern "C" int chunk(int parts, int part, int k, int odd) { return PairDrain::chunk(parts, part, k, odd); }
extern "C" int before_release(int parts) { return PairDrain::before_release(parts); }
extern "C" int arrivals(int parts) { return PairDrain::arrivals(parts); }
extern "C" int epilogue_parts(int N, int stages, int rounds, int vectors, int addend, int fp32) {
  return metis::pair_epilogue_parts(N, stages, rounds, vectors, addend != 0, fp32 != 0);
}
"""


@pytest.fixture(scope="module")
def drain(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_drain")
    (d / "drain.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{CSRC}", str(d / "drain.cpp"), "-o", str(d / "drain.so")], check=True)
    return C.CDLL(str(d / "drain.so"))


@pytest.mark.parametrize("parts", [2, 4])
def test_every_chunk_is_read_once(drain, parts):
    n = drain.chunks()
    for odd in (0, 1):
        assert sorted(drain.chunk(parts, part, k, odd) for part in range(parts) for k in range(n // parts)) == list(range(n))


@pytest.mark.parametrize("parts", [2, 4])
def test_a_warp_that_falls_behind_loses_nothing(drain, parts):
    n, stride, warps, tiles = drain.chunks(), drain.stride(), 2 * 4 * parts, 6

    def columns(tile):                                       # of its whole accumulator
        return set(range((tile % 2) * stride, (tile % 2) * stride + 32 * n))
    for part in range(parts):
        program = []                                         # of one warp of this part: what it does, tile by tile
        for tile in range(tiles):
            for k in range(n // parts):
                if k == drain.before_release(parts):
                    program.append(("arrive", tile, None))
                first = (tile % 2) * stride + 32 * drain.chunk(parts, part, k, tile % 2)
                program.append(("read", tile, set(range(first, first + 32))))
        for at in range(len(program)):                       # it stops in front of this step, all others run on
            arrived = {tile for what, tile, _ in program[:at] if what == "arrive"}
            started = 0                                      # the last tile whose products may have begun
            while started + 1 < tiles and warps - 1 + (started in arrived) >= drain.arrivals(parts):
                started += 1
            for what, tile, cols in program[at:]:
                for later in range(tile + 1, started + 1):
                    assert what != "read" or not cols & columns(later), (parts, part, at, tile, later)


# Both sides of each line as it was timed: columns, stages, rounds, row vectors, addend, fp32 -> the faster of two and four.
@pytest.mark.parametrize("shape,parts", [((8192, 4, 14, 0, 0, 0), 4), ((8192, 6, 14, 0, 0, 0), 2), ((8192, 16, 14, 0, 0, 0), 2), ((8192, 6, 2, 0, 0, 0), 4), ((8192, 6, 3, 0, 0, 0), 2),
                                         ((8192, 7, 14, 1, 0, 0), 4), ((8192, 8, 14, 1, 0, 0), 2), ((8192, 8, 5, 1, 0, 0), 2), ((8192, 18, 4, 1, 0, 0), 2),
                                         ((8192, 9, 2, 1, 0, 1), 4), ((8192, 14, 7, 2, 0, 0), 2), ((8192, 13, 3, 0, 1, 0), 2), ((8192, 18, 2, 0, 1, 0), 2), ((8192, 18, 4, 1, 1, 0), 2), ((8192, 16, 14, 2, 0, 0), 2), ((8192, 20, 3, 2, 0, 1), 4),
                                         ((8192, 12, 14, 0, 1, 0), 4), ((8192, 16, 14, 0, 1, 0), 2), ((8192, 14, 6, 0, 1, 0), 2), ((8192, 16, 14, 1, 1, 0), 4),
                                         ((8192, 20, 14, 1, 1, 0), 2), ((8192, 20, 14, 2, 1, 0), 4), ((8192, 32, 3, 2, 1, 0), 2),
                                         ((4096, 6, 2, 0, 0, 1), 2), ((8192, 2, 14, 0, 1, 1), 2), ((8192, 32, 2, 0, 1, 1), 2), ((8192, 16, 8, 1, 1, 1), 2),
                                         ((8192, 12, 14, 2, 1, 1), 4), ((8192, 32, 14, 2, 1, 1), 2), ((144, 4, 1, 0, 0, 0), 2), ((176, 5, 1, 0, 1, 0), 2), ((5296, 2, 1, 0, 1, 0), 2), ((256, 4, 1, 0, 0, 0), 4)])
def test_the_faster_number_of_warps(drain, shape, parts):
    assert drain.epilogue_parts(*shape) == parts
