"""CPU test of the rule by which a plan's executes are captured (csrc/graph_rule.h): one letter per
execute's output, and per execute whether it runs uncaptured (e), is captured (c) or launches the graph
(l).  "x" stands for a change that makes the graph stale (the context's scratch moved)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "graph_rule.h"
int main(int, char **argv) {
    static char buf[256];
    molints::GraphRule rule;
    const void *graph = nullptr;  // the output that has one
    for (const char *p = argv[1]; *p; ++p) {
        if (*p == 'x') { graph = nullptr; continue; }
        const void *out = buf + *p;
        const auto step = rule.next(out, graph == out);
        if (step == molints::GraphRule::CAPTURE) graph = out;
        std::putchar("ecl"[step]);
    }
    return 0;
}
"""


@pytest.mark.parametrize("order,steps", [
    ("AAAA", "ecll"),
    ("ABAB", "eeee"),
    ("AABAB", "ecele"),        # B's executes are never two in a row
    ("AABABABB", "ecelelec"),
    ("AABBA", "ecece"),        # the graph is B's: A starts over
    ("AAxAA", "eccl"),
    ("AABxAA", "eceec"),
])
def test_rule(tmp_path, order, steps):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no g++")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "t"), str(src)], check=True)
    r = subprocess.run([str(tmp_path / "t"), order], capture_output=True, text=True, check=True)
    assert r.stdout == steps
