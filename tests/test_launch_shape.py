"""CPU tests of the rules that deal an advection launch out over the device
(launch_shape.hpp, compiled on its own), on a device of 148 SMs: a tuning that limits
the blocks per SM keeps the lanes that it asks for."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dpa_b200" / "csrc"

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "launch_shape.hpp"
int main(int argc, char** argv) {
  for (int i = 1; i + 4 < argc; i += 5)
    std::printf("%u %u\n", dpa::advect_block(uint32_t(atoi(argv[i])), uint32_t(atoi(argv[i + 1])),
                                             uint32_t(atoi(argv[i + 2])), strtoull(argv[i + 3], 0, 10),
                                             148, atoi(argv[i + 4])),
                dpa::particles_per_warp(strtoull(argv[i + 3], 0, 10), 148));
}
"""


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC),
                    str(d / "driver.cpp"), "-o", str(d / "driver")], check=True)

    def run(*cases):
        out = subprocess.run([str(d / "driver")] + [str(v) for c in cases for v in c],
                             capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


# tuned block, tuned blocks per SM, the kernel's threads, lanes, resident -> block
@pytest.mark.parametrize("case,block", [
    ((0, 0, 256, 50000, 4), 64),      # 196 blocks of 256: uneven
    ((0, 2, 256, 50000, 4), 256),     # ... but the tuning's limit counts blocks of 256
    ((0, 1, 256, 50000, 4), 256),
    ((0, 4, 256, 90000, 4), 256),
    ((128, 0, 256, 50000, 4), 128),   # the tuning's block
    ((128, 2, 256, 50000, 4), 128),
    ((0, 0, 256, 50000, 0), 256),     # a field that limits the threads per SM
    ((0, 0, 256, 151552, 4), 256),    # four even blocks on every SM
    ((0, 0, 256, 151553, 4), 256),    # more than fit at once
    ((0, 0, 256, 75776, 4), 256),     # two even blocks on every SM
    ((0, 0, 256, 75777, 4), 64),
    ((0, 0, 256, 37888, 4), 256),     # one block on every SM
    ((0, 2, 256, 20000, 4), 160),     # fewer lanes than SMs x 256: spread, tuned or not
    ((0, 0, 256, 20000, 4), 160)])
def test_threads_per_block(shape, case, block):
    assert shape(case)[0][0] == block


def test_particles_per_warp(shape):
    counts = {1: 1, 1184: 1, 1185: 2, 2368: 2, 2369: 4, 9472: 8, 9473: 16, 18944: 16, 18945: 32}
    got = shape(*[(0, 0, 256, n, 4) for n in counts])
    assert [w for _, w in got] == list(counts.values())
