"""CPU test of the Rys class kernels' generated sources (generated/rys_*.cu), their statements run in
numpy the way rys_common.cuh runs them, against the oracle: for the group kernels the column update on
whole 2-D tables, the bra HRR per column and the ket HRR per row with the strides of the shared buffers, and the
threads' parts; for the lane-split kernels a root's tables in registers and its products."""
import math
import re
import sys
import zlib
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import pytest

import molints_b200 as mi

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "molecularintegrals.jl_b200" / "csrc"))
import gen_rys  # noqa: E402

sys.path.pop(0)


def fma(a, b, c):
    return a * b + c


def _statements(text):
    """C statements of fma expressions as Python code."""
    text = re.sub(r"\(void\)\w+; ?", "", text)
    text = re.sub(r"const double ", "", text)
    text = re.sub(r"\bin\[", "inp[", text)
    lines = [ln.strip().rstrip(";") for ln in text.splitlines() if ln.strip()]
    # several declarations in one statement
    lines = [re.sub(r", (?=\w+ = )", "; ", ln) for ln in lines]
    return compile("\n".join(lines), "<kernel>", "exec")


def _body(src, name):
    return re.search(name + r"\([^)]*\) \{\n(.*?)\n    \}", src, re.S).group(1)


def _norm_prims(l, prims):
    ex, co = np.array([p[0] for p in prims]), np.array([p[1] for p in prims])
    s = sum(co[i] * co[j] * (2 * np.sqrt(ex[i] * ex[j]) / (ex[i] + ex[j])) ** (l + 1.5)
            for i in range(len(ex)) for j in range(len(ex)))
    return [(e, c / np.sqrt(s) * (2 * e / np.pi) ** 0.75 * (4 * e) ** (l / 2)) for e, c in zip(ex, co)]


def _pairs(la, lb, pa, pb, A, B):
    c0 = math.sqrt(2.0) * math.pi ** 1.25
    out = []
    for a, ca in _norm_prims(la, pa):
        for b, cb in _norm_prims(lb, pb):
            z = a + b
            P = (a * A + b * B) / z
            out.append(SimpleNamespace(zeta=z, oo2z=0.5 / z, P=P, PA=P - A, pax=(P - A)[0], pay=(P - A)[1], paz=(P - A)[2],
                                       kab=c0 * ca * cb * math.exp(-a * b / z * np.sum((A - B) ** 2)) / z))
    return out


def _tables(bra, ket, u, w, E, F):
    """rys_tables_of: the three tables of one (primitive quartet, root), [axis][a (F + 1) + c]."""
    r2 = 1.0 / (bra.zeta + ket.zeta)
    PQ = bra.P - ket.P
    ez, zz = ket.zeta * r2, bra.zeta * r2
    b10, b01, b00 = bra.oo2z * (1 - ez * u), ket.oo2z * (1 - zz * u), 0.5 * r2 * u
    out = np.zeros((3, E + 1, F + 1))
    for x in range(3):
        c00, d00 = bra.PA[x] - ez * PQ[x] * u, ket.PA[x] + zz * PQ[x] * u
        I = out[x]
        I[0, 0] = bra.kab * ket.kab * math.sqrt(r2) * w if x == 0 else 1.0
        for a in range(E):
            I[a + 1, 0] = c00 * I[a, 0] + (a * b10 * I[a - 1, 0] if a else 0.0)
        for c in range(F):
            for a in range(E + 1):
                I[a, c + 1] = d00 * I[a, c] + (c * b01 * I[a, c - 1] if c else 0.0) + (a * b00 * I[a - 1, c] if a else 0.0)
    return out.reshape(3, -1)


def _group(src, C, tag, quartets, AB, CD):
    """rys_contract and rys_hrr of one quartet; quartets: per primitive quartet its roots' tables."""
    E, F, NA, NC, NAB, NCD = (C[k] for k in ("E", "F", "NA", "NC", "NAB", "NCD"))
    NCP, NCDP, S = C["NCP"], C["NCDP"], C["S"]
    assert S == (E + 1) * (F + 1) and NCP >= NC and NCDP >= NCD
    col = [int(v) for v in re.search(r"kCol_" + tag + r"\[\d+\] = \{ (.*?) \}", src).group(1).split(",")]
    norm = [float(v) for v in re.search(r"kNormAB_" + tag + r"\[\d+\] = \{(.*?)\}", src, re.S).group(1).split(",") if v.strip()]
    tabs = np.array([t.reshape(-1) for roots in quartets for t in roots])  # an item's tables: axis stride S
    acc = np.zeros((NA, NC))
    update = _statements(_body(src, "col_update"))
    for c2, cp in enumerate(col):
        cx, cy, cz = cp & 15, (cp >> 4) & 15, cp >> 8
        env = {"fma": fma, "acc": [0.0] * NA,
               "x": [tabs[:, a * (F + 1) + cx] for a in range(E + 1)],
               "y": [tabs[:, S + a * (F + 1) + cy] for a in range(E + 1)],
               "z": [tabs[:, 2 * S + a * (F + 1) + cz] for a in range(E + 1)]}
        exec(update, env)
        acc[:, c2] = [np.sum(v) for v in env["acc"]]
    mid, stg = np.full(NAB * NCP, np.nan), np.full(NAB * NCDP, np.nan)
    out = {}
    exec(_statements(_body(src, "bra_hrr")), {"fma": fma, "inp": list(acc), "out": out, "nrm": 1.0,
                                              "x": AB[0], "y": AB[1], "z": AB[2]})
    for r, v in out.items():
        mid[r + np.arange(NC)] = v
    rows = mid.reshape(NAB, NCP)
    out = {}
    exec(_statements(_body(src, "ket_hrr")), {"fma": fma, "inp": list(rows.T), "out": out, "nrm": np.array(norm),
                                              "x": CD[0], "y": CD[1], "z": CD[2]})
    for s, v in out.items():
        stg[np.arange(NAB) * NCDP + s] = v
    return stg.reshape(NAB, NCDP)[:, :NCD]


def _lane(src, tag, t, prims, AB, CD):
    """A lane-split kernel's block over all primitive quartets, then the closed-form transfer."""
    code = _statements(re.search(r"rys_root<\d+>\(R, T, k, u, w\);\n(.*?)\n            \}\n", src, re.S).group(1))
    acc = [0.0] * t["nblk"]
    for bra, ket, u, w in prims:
        r2 = 1.0 / (bra.zeta + ket.zeta)
        PQ = bra.P - ket.P
        for k in range(len(u)):
            exec(code, {"fma": fma, "acc": acc, "u": u[k], "w": w[k], "r2": r2, "ez": ket.zeta * r2, "zz": bra.zeta * r2,
                        "pref": bra.kab * ket.kab * math.sqrt(r2), "bra": bra, "ket": ket,
                        "PQx": PQ[0], "PQy": PQ[1], "PQz": PQ[2]})
    mono = [[v[0] ** m[0] * v[1] ** m[1] * v[2] ** m[2] for m in gen_rys.MONOS] for v in (AB, CD)]
    blk = np.array(acc).reshape(t["na"], t["nc"])
    mid = np.array([sum(k * mono[0][m] * blk[s] for s, m, k in terms) for terms in t["bra"]])
    out = np.array([sum(k * mono[1][m] * mid[:, s] for s, m, k in terms) for terms in t["ket"]]).T
    return out * np.outer(t["norm_ab"], t["norm_cd"])


@pytest.mark.parametrize("X,Y", gen_rys.class_pairs())
def test_statements_match_oracle(oracle, X, Y):
    tag = gen_rys.tag_of(X, Y)
    src = (gen_rys.OUT_DIR / f"rys_{tag}.cu").read_text()
    rng = np.random.default_rng(zlib.crc32(repr((X, Y, "kernel")).encode()))
    ls = [*X, *Y]
    centres = [rng.uniform(-1.2, 1.2, 3) for _ in range(4)]
    shells = [(xyz, l, mi.basis._random_shell(rng, l, int(rng.integers(1, 3)), 0.3, 6.0)) for l, xyz in zip(ls, centres)]
    with oracle.exact_boys():
        ref = oracle.shell_quartet(mi.Shells.from_list(shells), 0, 1, 2, 3).reshape(-1)
    A, B, C, D = centres
    bras, kets = _pairs(*X, shells[0][2], shells[1][2], A, B), _pairs(*Y, shells[2][2], shells[3][2], C, D)
    nr = sum(ls) // 2 + 1
    prims = []
    for bra in bras:
        for ket in kets:
            PQ = bra.P - ket.P
            prims.append((bra, ket, *oracle.rys_roots(nr, bra.zeta * ket.zeta / (bra.zeta + ket.zeta) * float(PQ @ PQ))))
    if gen_rys.is_lane(X, Y):
        got = _lane(src, tag, gen_rys.class_tables(X, Y), prims, A - B, C - D)
    else:
        K = {k: int(v) for k, v in re.findall(r"(\w+) = (\d+)", src.split("// stage 2")[0])}
        assert K["NR"] == nr
        got = _group(src, K, tag, [[_tables(b, k, u[r], w[r], K["E"], K["F"]) for r in range(nr)] for b, k, u, w in prims],
                     A - B, C - D)
    assert np.max(np.abs(got.reshape(-1) - ref)) < 1e-12 * max(1.0, np.max(np.abs(ref)))


@pytest.mark.parametrize("X,Y", [c for c in gen_rys.class_pairs() if not gen_rys.is_lane(*c)])
def test_threads_cover_a_round_once(X, Y):
    """RysPart: every (ket pair, primitive quartet, root) and every (ket pair, share, column) of a round
    has one thread, and the threads that add up a column's shares are lanes of one warp."""
    t = gen_rys.class_tables(X, Y)
    G, W, H, PB, NR, NC = t["G"], t["W"], t["H"], t["pb"], t["nr"], t["nc"]
    one, two = [], []
    for lane in range(G):
        ni = PB * NR
        w1 = min(lane // ni, W)
        if w1 < W:
            one.append((w1, (lane - w1 * ni) // NR, (lane - w1 * ni) % NR))
        w2 = min(lane // (H * NC), W)
        if w2 < W:
            two.append((w2, lane // NC - w2 * H, lane % NC))
    assert sorted(one) == [(w, b, r) for w in range(W) for b in range(PB) for r in range(NR)]
    assert sorted(two) == [(w, h, c) for w in range(W) for h in range(H) for c in range(NC)]
    assert W == 1 or G == 32
    assert H == 1 or (G == 32 and W * H * NC <= 32 and H & (H - 1) == 0)
    assert t["smem_group"] >= max(W * PB * NR * t["SI"], W * t["nab"] * (t["ncp"] + t["ncdp"])) and t["SI"] >= 3 * t["S"]
