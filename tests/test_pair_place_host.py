"""CPU test of pair_place (csrc/plan_build.cuh): the place that each pair of a short list counts for
itself, against the stable sort and prefix sum that order a long one, for lists of one pair up to the
longest short one, runs of one pair up to all of them, and keys with ties (few kept counts, with and
without a Qabs bucket above them)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"

PROGRAM = r"""
#include <algorithm>
#include <cstdio>
#include <numeric>
#include <random>
#include <vector>
#include "plan_build.cuh"
using namespace molints;
int main() {
    std::mt19937 rng(5);
    int bad = 0;
    for (int n : {1, 2, 31, 32, 33, 257, 1830, kPlaceMaxPairs})
        for (int run : {1, 3, 32, 100, n})
            for (int buckets : {1, 256}) {
                std::vector<int> seg(n), npp(n), order(n);
                std::vector<unsigned long long> key(n);
                for (int k = 0; k < n; ++k) {
                    seg[k] = k && rng() % run ? seg[k - 1] : k;
                    npp[k] = rng() % 3 ? (int)(rng() % 37) : 0;
                    key[k] = ((unsigned long long)seg[k] << 20) | ((rng() % buckets) << 8) | (unsigned)(36 - npp[k]);
                }
                std::iota(order.begin(), order.end(), 0);
                std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return key[a] < key[b]; });
                int prim = 0;
                for (int p = 0; p < n; ++p) {
                    const int k = order[p];
                    int before = 0, off = 0;
                    for (int lane = 0; lane < 32; ++lane) {
                        const PairPlace s = pair_place(key.data(), npp.data(), seg.data(), n, k, lane, 32);
                        before += s.before;
                        off += s.prim;
                    }
                    bad += seg[k] + before != p || off != prim;
                    prim += npp[k];
                }
            }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_pair_place(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src = tmp_path / "t.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-I", str(CSRC), "-o", str(exe), str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
