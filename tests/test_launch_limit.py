"""CPU test of the rule that limits the threads per SM of a launch (launch_shape.hpp,
compiled on its own): a limit that depends on the steps holds above a third of a cell a
step, whatever the step's sign; one that does not holds always."""
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dpa_b200" / "csrc"

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "launch_shape.hpp"
int main(int argc, char** argv) {
  if (argc == 3)
    std::printf("%.17g", dpa::limit_speed(strtod(argv[1], 0), strtod(argv[2], 0)));
  else
    std::printf("%u", dpa::limited_threads(uint32_t(atoi(argv[1])), strtof(argv[2], 0),
                                           strtof(argv[3], 0)));
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("limit")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", str(CSRC),
                    str(d / "driver.cpp"), "-o", str(d / "driver")], check=True)
    return str(d / "driver")


@pytest.mark.parametrize("limit,speed,dt,threads", [
    (0, 0.0, 0.5, 0), (0, 2.0, 0.5, 0),             # no limit
    (768, 0.0, 0.0, 768), (768, 0.0, 0.01, 768),    # one that holds always
    (768, 1.0, 0.33, 0), (768, 1.0, 0.34, 768), (768, 1.0, -0.34, 768), (768, 1.0, -0.33, 0),
    (768, 2.5, 0.13, 0), (768, 2.5, 0.14, 768), (768, 1e-30, 1e30, 768), (768, 1e30, 0.0, 0)])
def test_limit(driver, limit, speed, dt, threads):
    out = subprocess.run([driver, str(limit), str(speed), str(dt)], capture_output=True, text=True,
                         check=True).stdout
    assert int(out) == threads


# A field whose velocity changes by more than a twentieth in a cell is limited from a fifth
# of a cell a step on.
@pytest.mark.parametrize("speed,change,cells", [
    (1.0, 0.0, 1 / 3), (1.0, 0.049, 1 / 3), (1.0, 0.051, 0.2), (3.0, 0.14, 1 / 3), (3.0, 2.0, 0.2),
    (0.0, 0.0, None)])
def test_speed(driver, speed, change, cells):
    out = float(subprocess.run([driver, str(speed), str(change)], capture_output=True, text=True,
                               check=True).stdout)
    if cells is None:
        assert out == 0.0
        return
    for factor, threads in ((0.999, 0), (1.001, 768)):
        dt = factor * cells / speed
        got = subprocess.run([driver, "768", str(out), str(dt)], capture_output=True, text=True,
                             check=True).stdout
        assert int(got) == threads
