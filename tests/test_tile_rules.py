"""The mixed stage's rule for blocks with extra thread rows, compiled for each tile height: it may
not count on more resident blocks of that shape an SM than the kernels' register budget and the
SM's 2048 threads leave (else such blocks run in two rounds, which cost up to 14 %)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include "tns_tile.cuh"
int main() {
    using namespace tns;
    std::printf("%d %d %d", STAGE_MX_RIM_PER_SM, RIM_MINB, NTHREADS + TJ * RIM_ROWS);
}
"""


@pytest.mark.parametrize("ti", [4, 8, 16])
def test_rim_blocks_counted_on_are_resident(ti, tmp_path):
    if shutil.which("nvcc") is None:
        pytest.skip("nvcc is needed to compile the rule")
    (tmp_path / "rule.cu").write_text(SRC)
    subprocess.run(["nvcc", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-DTNS_TI={ti}",
                    "-I" + os.path.join(ROOT, "2d-turbulent-navier-stokes_b200", "csrc"), str(tmp_path / "rule.cu"),
                    "-o", str(tmp_path / "rule")], check=True)
    lines, budget, threads = map(int, subprocess.run([str(tmp_path / "rule")], check=True, capture_output=True,
                                                     text=True).stdout.split())
    assert lines <= budget and budget * threads <= 2048
