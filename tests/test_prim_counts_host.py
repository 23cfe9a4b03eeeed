"""CPU tests of the primitive-quartet counts and indices of kernels that walk them as one list, for
contractions up to the longest that are accepted (255 primitives a shell, 255^4 quartets)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"

GENERIC = r"""
#include <cstdio>
#include <initializer_list>
#include "eri_generic.cuh"
using namespace molints;
int main() {
    int bad = 0;
    const int lists[][4] = {{1, 1, 1, 1}, {3, 1, 2, 5}, {164, 164, 164, 164}, {125, 125, 125, 125},
                            {255, 255, 255, 1}, {216, 216, 216, 216}, {255, 255, 255, 255}};
    for (const auto &np : lists) {
        const unsigned long long want = 1ull * np[0] * np[1] * np[2] * np[3];
        const unsigned n = gen_prim_count(np);
        bad += n != want;
        // the kernel's loop: steps of at most 96 primitive quartets, up to the last one
        bad += want + 96 > 0xffffffffull;
        for (unsigned long long k : {0ull, want / 3, want / 2, want - 1}) {
            const GenPrims p = gen_prim((unsigned)k, np);
            bad += p.a < 0 || p.a >= np[0] || p.b < 0 || p.b >= np[1] || p.c < 0 || p.c >= np[2] || p.d < 0 || p.d >= np[3];
            bad += ((1ull * p.a * np[1] + p.b) * np[2] + p.c) * np[3] + p.d != k;
        }
    }
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def _run(program, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    src = tmp_path / "t.cu"
    src.write_text(program)
    exe = tmp_path / "t"
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-I", str(CSRC), "-o", str(exe), str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_generic_kernel(tmp_path):
    _run(GENERIC, tmp_path)


RYS = r"""
#include <cstdio>
#include <initializer_list>
#include "rys_common.cuh"
using namespace molints;
int main() {
    int bad = 0;
    const unsigned long long top = 255ull * 255;
    for (unsigned long long nb : {1ull, 7ull, 216ull * 216, top})
        for (unsigned long long nk : {1ull, 49ull, 216ull * 216, top}) {
            const unsigned n = rys_prim_count((int)nb, (int)nk);
            bad += n != nb * nk || nb * nk + 128 > 0xffffffffull;
        }
    // the batches of a quartet of nq primitive quartets, in a round that goes on for a longer one
    for (unsigned nq : {0u, 1u, 31u, 32u, 33u, 100u})
        for (int pb : {1, 7, 32, 128}) {
            unsigned sum = 0;
            for (unsigned g0 = 0; g0 < 300; g0 += pb) {
                const int n = rys_batch(nq, g0, pb);
                bad += n < 0 || n > pb;
                sum += n;
            }
            bad += sum != nq;
        }
    const unsigned big = rys_prim_count((int)top, (int)top);
    bad += rys_batch(big, 0, 32) != 32 || rys_batch(big, big - 5, 32) != 5 || rys_batch(big, big, 32) != 0;
    std::printf("%d\n", bad);
    return bad != 0;
}
"""


def test_rys_kernels(tmp_path):
    _run(RYS, tmp_path)
