"""CPU test of the unrolled HRR sides the Rys kernels run (gen_rys.HrrSide) against the closed form
of the transfer (gen_rys.hrr_terms), for every shell pair of the pair classes, in exact rational
arithmetic: the two are the same polynomial."""
import random
import re
import sys
from fractions import Fraction
from pathlib import Path

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"))
import gen_rys  # noqa: E402


@pytest.mark.parametrize("la,lb", gen_rys.pair_classes())
def test_side_equals_closed_form(la, lb):
    rng = random.Random(10 * la + lb)
    rows = gen_rys.block_components(la, la + lb)
    index = {c: i for i, c in enumerate(rows)}
    side = gen_rys.HrrSide(la, lb, index)
    frac = lambda: Fraction(rng.randint(-50, 50), rng.randint(1, 9))  # noqa: E731
    env = {"inp": [frac() for _ in rows], "x": frac(), "y": frac(), "z": frac(), "fma": lambda a, b, c: a * b + c}
    for line in side.lines:
        name, expr = re.fullmatch(r"const double (\w+) = (.*);", line).groups()
        env[name] = eval(expr.replace("in[", "inp["), env)
    got = [eval(e.replace("in[", "inp["), env) for e in side.out]
    mono = [env["x"] ** a * env["y"] ** b * env["z"] ** c for a, b, c in gen_rys.MONOS]
    want = [sum(k * mono[m] * env["inp"][s] for s, m, k in terms) for terms in gen_rys.hrr_terms(la, lb, index)]
    assert got == want
