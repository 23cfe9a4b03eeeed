"""CPU test of host-callable helpers of the plan build (csrc/plan_build.cuh).

molecule_lane_cost: non-decreasing in the molecule's primitive pairs, never above the schedule's
bound, the bound itself for large molecules.  nonzero_end: the first pair without kept primitive pairs of a
run in descending kept count, against a linear scan, for every run of up to 40 pairs and every
sub-run.  The work queues end each bra's ket run there."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <vector>
#include "plan_build.cuh"
using namespace molints;
int main() {
    int bad = 0;
    for (int n = 0; n <= 40; ++n)
        for (int z = 0; z <= n; ++z) {
            std::vector<int> npp(n + 1, 0);
            for (int k = 0; k < n - z; ++k) npp[k] = 1 + (n - z - k) / 3;
            for (int b = 0; b <= n; ++b)
                for (int e = b; e <= n; ++e) {
                    int want = b;
                    while (want < e && npp[want] > 0) ++want;
                    if (nonzero_end(npp.data(), b, e) != want) ++bad;
                }
        }
    for (double bound : {5.0, 30.0, 80.0, 640.0, 1e6}) {
        double prev = 0.0;
        for (double npp = 0.0; npp < 1e6; npp = npp * 1.3 + 1.0) {
            const double c = molecule_lane_cost(npp, bound);
            if (!(c > 0.0) || c < prev || c > bound) ++bad;
            prev = c;
        }
        if (bound <= 1e4 && molecule_lane_cost(1e6, bound) != bound) ++bad;
    }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_nonzero_end(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src = tmp_path / "t.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1",
                    "--expt-relaxed-constexpr", "-I", str(CSRC), "-o", str(exe), str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
