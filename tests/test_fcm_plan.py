"""Which grids the force-coupling solver transforms itself (csrc/fcm_plan.cuh): those on which a call with particles
everywhere was measured no slower than with the library's transforms, and the factors it transforms them by.  The rule
is host code, compiled here by itself."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "cufcm_fil_b200" / "csrc"

MAIN = r"""
#include "fcm_plan.cuh"
#include <cstdio>
#include <cstdlib>
int main(int argc, char **argv) {
    if (argc == 2) {
        for (int r : cufil::fftk::radices(std::atoi(argv[1]))) std::printf("%d ", r);
        return 0;
    }
    std::printf("%d", cufil::fftk::supported(std::atoi(argv[1]), std::atoi(argv[2]), std::atoi(argv[3])) ? 1 : 0);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-I", str(CSRC), "-x", "c++", str(d / "main.cpp"), "-o",
                    str(d / "plan")], check=True)
    return lambda *a: subprocess.run([str(d / "plan"), *map(str, a)], check=True, capture_output=True, text=True).stdout


# (grid, own transforms): with particles everywhere the library's were more than 4% faster on the grids marked 0
@pytest.mark.parametrize("grid,own", [
    ((192, 192, 192), 1), ((200, 200, 200), 1), ((256, 256, 256), 1), ((270, 270, 270), 1), ((320, 320, 320), 1),
    ((384, 384, 384), 1), ((512, 512, 512), 1), ((432, 432, 432), 1), ((200, 200, 216), 1), ((128, 256, 256), 1),
    ((1024, 512, 256), 1), ((1000, 200, 200), 1), ((512, 128, 128), 1),
    ((2048, 64, 64), 0), ((2048, 256, 256), 0), ((1024, 1024, 16), 0), ((1024, 1024, 64), 0), ((128, 1000, 100), 0),
    ((128, 128, 1000), 0), ((256, 32, 1000), 0), ((32, 480, 480), 0), ((8, 1000, 1000), 0), ((64, 512, 512), 0),
    ((100, 250, 250), 0), ((144, 256, 256), 0), ((144, 270, 270), 0), ((128, 270, 270), 0), ((108, 270, 270), 0),
    ((216, 216, 216), 0), ((128, 243, 243), 0), ((256, 324, 324), 0), ((512, 243, 243), 0), ((512, 324, 324), 0),
    ((1458, 81, 81), 0), ((100, 729, 100), 0),
    ((128, 128, 128), 0), ((352, 256, 256), 0), ((255, 256, 256), 0), ((256, 1080, 256), 0), ((2560, 1024, 1024), 0)])
def test_grids(plan, grid, own):
    assert plan(*grid) == str(own)


@pytest.mark.parametrize("n,want", [(60, "5 4 3 "), (64, "8 8 "), (81, "3 3 3 3 "), (250, "5 5 5 2 "), (1000, "8 5 5 5 "),
                                    (1024, "8 8 8 2 "), (77, "")])
def test_radices(plan, n, want):
    assert plan(n) == want
