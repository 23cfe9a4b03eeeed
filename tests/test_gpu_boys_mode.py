"""Which Boys function each class pair evaluates, per method and mode: s, p, d and f shells of nearly
equal exponents on two centres, so that every quartet between the centres has T between 30.6 and 31.6,
where the reference mode's asymptotic form and the exact function differ most (5e-13 to 1.5e-11 in the
d and f class pairs).  Against the long-double HGP restatement in the two modes; the FP64 restatement is
within 2e-15 of it on this basis, so 1e-13 separates rounding from the mode."""
import re
import sys
from pathlib import Path

import numpy as np
import pytest

import molints_b200 as mi

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"))
import gen_eri  # noqa: E402

sys.path.pop(0)

TOL = 1e-13
# class pairs whose AUTO kernel is Rys although an HGP kernel exists, and that evaluate the exact function
# in the reference mode too
EXACT_UNDER_AUTO = {"dpdp", "dddd", "fppp"}
PAIRS = ["ss", "ps", "pp", "ds", "dp", "fs", "dd", "fp", "fd", "ff"]


def _basis():
    r = np.sqrt(30.6)
    u = np.array([0.3, 0.5, np.sqrt(0.66)])
    return mi.Shells.from_list([(c, l, [(1.0 + 0.01 * l, 1.0)])
                                for c in (np.zeros(3), r * u) for l in range(4)], "modes")


def _by_class(sh, *diffs):
    """{class pair: largest entry of each vector}; f exponents are above d's, so (f, d) pairs are (f d|."""
    l = np.concatenate([[x] * mi.basis.ncart(int(x)) for x in sh.L])
    i, j = np.tril_indices(len(l))
    cls = np.array([PAIRS.index("spdf"[max(a, b)] + "spdf"[min(a, b)]) for a, b in zip(l[i], l[j])])
    ij, kl = np.tril_indices(len(cls))
    hi, lo = np.maximum(cls[ij], cls[kl]), np.minimum(cls[ij], cls[kl])
    return {PAIRS[x] + PAIRS[y]: [float(np.max(d[(hi == x) & (lo == y)])) for d in diffs]
            for x in range(len(PAIRS)) for y in range(x + 1)}


@pytest.fixture(scope="module")
def case(oracle):
    sh = _basis()
    with oracle.stable_orientation():
        mode = oracle.eri_packed_hgp_ld(sh, nthreads=0)
        with oracle.exact_boys():
            exact = oracle.eri_packed_hgp_ld(sh, nthreads=0)
    return sh, mode, exact


def test_the_basis_tells_the_modes_apart(case):
    sh, mode, exact = case
    diff = {c: v[0] for c, v in _by_class(sh, np.abs(mode - exact)).items()}
    for c in ("dddp", "ddpp", "ddps", "ddds", "dppp", "dpds", "fsdp", "fsfs", "fpds", "fdps", *EXACT_UNDER_AUTO):
        assert diff[c] > 4 * TOL, c


def _engine():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from molints_b200 import engine
    return engine, engine.Engine(0)


@pytest.mark.gpu
@pytest.mark.parametrize("method", ["auto", "hgp", "rys"])
def test_reference_mode(case, method):
    sh, mode, exact = case
    engine, eng = _engine()
    names = ["spdf"[a] + "spdf"[b] for a, b in engine.PAIR_CLASSES]
    hgp = {gen_eri.tag_of(X, Y) for X, Y in gen_eri.class_pairs()}
    try:
        table = {names[x] + names[y]: v & 3 for (x, y), v in eng.class_methods().items()}
        got = eng.eri_packed(sh, boys=engine.BOYS_REFERENCE,
                             method={"auto": engine.METHOD_AUTO, "hgp": engine.METHOD_HGP,
                                     "rys": engine.METHOD_RYS}[method])
    finally:
        eng.close()
    for c, (dm, dx) in _by_class(sh, np.abs(got - mode), np.abs(got - exact)).items():
        if method == "rys" or c not in hgp:
            follows = False
        elif method == "hgp" or table[c] != engine.METHOD_RYS:
            follows = True
        else:
            follows = c not in EXACT_UNDER_AUTO
        assert (dm if follows else dx) < TOL, (c, dm, dx)


@pytest.mark.gpu
@pytest.mark.parametrize("method", [0, 1, 2])
def test_exact_mode(case, method):
    sh, _, exact = case
    engine, eng = _engine()
    try:
        got = eng.eri_packed(sh, boys=engine.BOYS_EXACT, method=method)
    finally:
        eng.close()
    assert np.max(np.abs(got - exact)) < TOL


@pytest.mark.parametrize("n", range(1, 8))
def test_limit_rule_gives_the_asymptotic_family(n):
    """sum_i g_i h_i^2m = (2m-1)!! / 2^m sqrt(pi) / 2 for m < 2n: a Rys kernel that takes its nodes and
    weights from the limits at X >= 30 evaluates the reference mode's F_m (all terms positive; a table
    entry's rounding enters 2n times at most)."""
    text = (Path(gen_eri.__file__).parent / "generated" / "rys_tables.cu").read_text()
    o = n * (n - 1) // 2
    x2, w = (np.array([float.fromhex(v) for v in re.findall(r"0x[0-9a-fp.+-]+", re.search(
        name + r"\[\d+\] = \{(.*?)\};", text, re.S).group(1))])[o:o + n] for name in ("kRysHermX2", "kRysHermW"))
    f = np.sqrt(np.pi) / 2
    for m in range(2 * n):
        assert abs(np.sum(w * x2 ** m) - f) <= 1e-14 * f, m
        f *= (2 * m + 1) / 2
