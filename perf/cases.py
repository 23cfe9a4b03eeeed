"""The calls that the engine's speed is measured by: what a quantum-chemistry program has it do.

Kinds of call (``case["kind"]``):

  host    all_twoe_ints(shells): the drop-in driver, host arrays in, packed host vector out
  device  Engine.eri_packed_device: the drop-in call into a device vector; plan creation included
  plan    Plan.execute of a one-molecule plan kept by the program, as a captured CUDA graph
  batch   Plan.execute of one plan over several molecules, as a captured CUDA graph
  jk      Plan.jk: Coulomb and exchange matrices of a density, one per SCF iteration
  serve   Engine.submit / poll / release of a burst of requests to the 8-slot server

Molecules are the synthetic ones of the package's workload generators: jittered-lattice geometries,
a third of the atoms heavy, log-uniform exponents, random contractions.  The recipes:

  sto3g   the built-in minimal basis on carbon and hydrogen (K = 3, s and p)
  sv      split valence (heavy: s6 s3 p3 s1 p1, hydrogen: s3 s1), exponents 0.1 .. 5e3
  pol     polarised (heavy: s7 s7 s1 p3 p1 d1, hydrogen: s3 s1 p1), exponents 0.1 .. 1e4
  polf    pol with an uncontracted f shell on the heavy atoms
  qz      one s, p, d, f and g shell on each heavy atom (s and p contracted)

The sizes of a case (atoms, recipes, options) are in the case; geometries, exponents and
coefficients come from the seed.
"""
from __future__ import annotations

import importlib
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

_ROOT = Path(__file__).resolve().parent.parent
_PKG = "molints_b200"


def _package():
    """The package of this repository (its directory name is not an identifier)."""
    if _PKG not in sys.modules:
        root = Path.cwd() if (Path.cwd() / "molecularintegrals.jl_b200").is_dir() else _ROOT
        d = root / "molecularintegrals.jl_b200"
        spec = importlib.util.spec_from_file_location(_PKG, d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[_PKG] = mod
        spec.loader.exec_module(mod)
    return sys.modules[_PKG]


def _engine_module():
    _package()
    return importlib.import_module(_PKG + ".engine")


# The accuracy options of the batch and serving workloads' mixed mode: every result within 1e-9
# of the exact integral.
FP32_CUTOFF = 1e-3
SCREEN_CUTOFF = 5e-10
SERVE_SLOTS = 8


def listed():
    return [
        # a small molecule in a minimal basis (staggered ethane's size, 16 functions) through the
        # drop-in driver: the shortest call there is, all latency
        {"name": "drop_in_minimal_8", "kind": "host", "recipe": "sto3g", "atoms": "8", "boys": "reference"},
        # the drop-in call once per geometry (an optimisation or dynamics step): a 24-atom
        # split-valence molecule of 104 functions, plan creation and execute
        {"name": "drop_in_split_valence_24", "kind": "device", "recipe": "sv", "atoms": "24",
         "method": "auto", "boys": "reference"},
        # the same call through the Rys driver, on ethane's size with polarisation functions
        # (60 functions, l <= 2)
        {"name": "drop_in_rys_polarised_8", "kind": "device", "recipe": "pol", "atoms": "8",
         "method": "rys", "boys": "exact"},
        # integrals recomputed from a kept plan: 24 atoms, split valence (l <= 1)
        {"name": "plan_split_valence_24", "kind": "plan", "recipe": "sv", "atoms": "24", "boys": "exact"},
        # ... 8 atoms with polarisation functions (l <= 2)
        {"name": "plan_polarised_8", "kind": "plan", "recipe": "pol", "atoms": "8", "boys": "exact"},
        # ... 11 atoms of the serving mix, f shells on the heavy atoms (l <= 3, odd sizes)
        {"name": "plan_f_shells_11", "kind": "plan", "recipe": "polf", "atoms": "11", "boys": "exact"},
        # ... two atoms of a quadruple-zeta-like basis with g shells (l <= 4)
        {"name": "plan_g_shells_2", "kind": "plan", "recipe": "qz", "atoms": "2", "boys": "exact"},
        # one plan of the 256-molecule batch's kind: eight molecules of 6 to 35 atoms, recipes
        # alternating, 1.2e9 integrals; FP64
        {"name": "batch_fp64_8", "kind": "batch", "recipe": "sv,pol", "atoms": "6,9,13,17,21,26,30,35",
         "precision": "fp64", "boys": "exact"},
        # ... the same in mixed precision with Schwarz screening
        {"name": "batch_mixed_8", "kind": "batch", "recipe": "sv,pol", "atoms": "6,9,13,17,21,26,30,35",
         "precision": "mixed", "boys": "exact"},
        # J and K for one density per SCF iteration: 24 atoms, split valence
        {"name": "jk_split_valence_24", "kind": "jk", "recipe": "sv", "atoms": "24", "boys": "exact"},
        # ... 15 atoms with polarisation functions
        {"name": "jk_polarised_15", "kind": "jk", "recipe": "pol", "atoms": "15", "boys": "exact"},
        # a burst of sixteen requests of mixed sizes (half with f shells) to the server, mixed
        # precision as the serving workload
        {"name": "serve_burst_16", "kind": "serve", "recipe": "pol,polf",
         "atoms": "2,3,5,6,8,9,11,12,4,7,10,13,3,6,9,14", "precision": "mixed", "boys": "exact"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo - 0.49), math.log(hi + 0.49)))))


def _integrals(recipe, natom):
    """Packed integrals of a batch molecule: 9 or 15 functions on a heavy atom, 2 or 5 on a hydrogen."""
    heavy = max(1, natom // 3)
    n = heavy * (9 if recipe == "sv" else 15) + (natom - heavy) * (2 if recipe == "sv" else 5)
    return n * (n + 1) * (n * n + n + 2) // 8


def draw(rng):
    """One more case: the same kinds of call, sizes spread over the ranges they are used in."""
    kind = rng.choice(["host", "device", "device", "plan", "plan", "plan", "batch", "batch", "jk", "jk", "serve"])
    boys = rng.choice(["reference", "exact"])
    if kind == "host":
        if rng.random() < 0.5:
            return {"kind": kind, "recipe": "sto3g", "atoms": str(_log_int(rng, 2, 20)), "boys": boys}
        return {"kind": kind, "recipe": rng.choice(["sv", "pol"]), "atoms": str(_log_int(rng, 2, 9)), "boys": boys}
    if kind == "device":
        recipe = rng.choice(["sv", "pol"])
        return {"kind": kind, "recipe": recipe, "atoms": str(_log_int(rng, 3, 36 if recipe == "sv" else 16)),
                "method": rng.choice(["auto", "auto", "hgp", "rys"]), "boys": boys}
    if kind in ("plan", "jk"):
        recipe = rng.choice(["sv", "pol", "polf"] + (["qz"] if kind == "plan" else []))
        if recipe == "qz":
            return {"kind": kind, "recipe": recipe, "atoms": str(rng.randint(1, 2)), "hydrogens": rng.randint(0, 4),
                    "boys": boys}
        top = {"sv": 40, "pol": 24, "polf": 16}[recipe] if kind == "plan" else {"sv": 32, "pol": 18, "polf": 10}[recipe]
        return {"kind": kind, "recipe": recipe, "atoms": str(_log_int(rng, 3, top)), "boys": boys}
    if kind == "batch":
        n = _log_int(rng, 2, 24)
        precision = rng.choice(["fp64", "mixed"])
        while True:  # at most the listed batch's integrals
            atoms = [rng.randint(4, 35) for _ in range(n)]
            if sum(_integrals("sv" if m % 2 == 0 else "pol", a) for m, a in enumerate(atoms)) <= 1.16e9:
                break
        return {"kind": kind, "recipe": "sv,pol", "atoms": ",".join(map(str, atoms)), "precision": precision,
                "boys": boys}
    n = _log_int(rng, 3, 24)
    return {"kind": kind, "recipe": "pol,polf", "atoms": ",".join(str(rng.randint(2, 14)) for _ in range(n)),
            "precision": rng.choice(["fp64", "mixed"]), "boys": boys}


# ------------------------------------------------------------------------------ inputs
def _molecule(recipe, natom, hydrogens, seed):
    b = _package().basis
    if recipe == "sto3g":
        rng = np.random.default_rng(seed)
        heavy = max(1, natom // 4)
        pos = b._lattice_atoms(rng, heavy, natom - heavy)
        return b.build_basis([b.atom(6 if a < heavy else 1, *pos[a]) for a in range(natom)], "sto3g")
    if recipe == "qz":
        return b.synthetic_molecule(seed, natom, hydrogens, [(0, 2), (1, 2), (2, 1), (3, 1), (4, 1)],
                                    [(0, 2), (1, 1)], 0.3, 8.0, f"qz{natom}")
    heavy = max(1, natom // 3)
    if recipe == "sv":
        return b.synthetic_molecule(seed, heavy, natom - heavy, b.SPLIT_VALENCE_HEAVY, b.SPLIT_VALENCE_H,
                                    0.1, 5e3, f"sv{natom}")
    return b.synthetic_molecule(seed, heavy, natom - heavy, b.POLARISED_C, b.POLARISED_H, 0.1, 1e4,
                                f"{recipe}{natom}", heavy_extra=[(3, 1)] if recipe == "polf" else [])


def _molecules(case, seed):
    recipes = case["recipe"].split(",")
    return [_molecule(recipes[m % len(recipes)], int(n), int(case.get("hydrogens", 0)), 1000 * int(seed) + m)
            for m, n in enumerate(case["atoms"].split(","))]


def _density(n, seed):
    """A symmetric matrix of the size of a density."""
    d = np.random.default_rng(seed).normal(size=(n, n)) / math.sqrt(n)
    return 0.5 * (d + d.T)


def _options(case, E):
    opts = {"boys": E.BOYS_EXACT if case["boys"] == "exact" else E.BOYS_REFERENCE}
    if case.get("precision") == "mixed":
        opts.update(precision=E.MIXED, fp32_cutoff=FP32_CUTOFF, screen_cutoff=SCREEN_CUTOFF)
    if "method" in case:
        opts["method"] = {"auto": E.METHOD_AUTO, "hgp": E.METHOD_HGP, "rys": E.METHOD_RYS}[case["method"]]
    return opts


class _DeviceVector:
    """A served result (device pointer) as torch reads it, without a copy."""

    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False), "version": 3}


_served = False  # the default engine's server runs


def prepare(case, seed):
    global _served
    E = _engine_module()
    eng = E.default_engine()
    eng.set_stream(torch.cuda.current_stream().cuda_stream)
    mols = _molecules(case, seed)
    opts = _options(case, E)
    state = {"kind": case["kind"], "E": E, "eng": eng, "opts": opts}

    def vector(n):
        return torch.empty(n, dtype=torch.float64, device="cuda")

    if case["kind"] == "host":
        state["shells"] = mols[0]
    elif case["kind"] == "device":
        state.update(shells=mols[0], out=vector(mols[0].npacked))
    elif case["kind"] in ("plan", "batch"):
        plan = eng.plan(mols[0], **opts) if case["kind"] == "plan" else eng.plan_batch(mols, **opts)
        plan.set_graph(True)
        state.update(plan=plan, out=vector(plan.npacked))
    elif case["kind"] == "jk":
        n = mols[0].nbf
        state.update(plan=eng.plan(mols[0], **opts), D=torch.from_numpy(_density(n, seed)).cuda(),
                     J=torch.empty(n, n, dtype=torch.float64, device="cuda"),
                     K=torch.empty(n, n, dtype=torch.float64, device="cuda"))
    else:
        if not _served:
            eng.serve_start(SERVE_SLOTS)
            _served = True
        state.update(mols=mols, out=[vector(m.npacked) for m in mols])
    return state


def run(state):
    kind = state["kind"]
    if kind == "host":
        return state["E"].all_twoe_ints(state["shells"], boys=state["opts"]["boys"])
    if kind == "device":
        state["eng"].eri_packed_device(state["shells"], state["out"].data_ptr(), **state["opts"])
        return state["out"]
    if kind in ("plan", "batch"):
        state["plan"].execute(state["out"].data_ptr())
        return state["out"]
    if kind == "jk":
        state["plan"].jk(state["D"].data_ptr(), state["J"].data_ptr(), state["K"].data_ptr())
        return {"J": state["J"], "K": state["K"]}
    # the program takes each result into its own buffer and gives the request back
    requests = [state["eng"].submit(m, **state["opts"]) for m in state["mols"]]
    for r, out in zip(requests, state["out"]):
        r.poll(-1)
        out.copy_(torch.as_tensor(_DeviceVector(r.device_ptr(), r.npacked), device="cuda"))
    torch.cuda.current_stream().synchronize()
    for r in requests:
        r.release()
    return state["out"]


# ------------------------------------------------------------------------------ work
def _pair_counts(shells):
    """{(la, lb): (pairs, primitive pairs, sum of squares of a pair's primitive pairs)} with the
    primitive pairs whose Gaussian overlap factor exp(-ab/(a+b) R^2) is at least 1e-18."""
    out = {}
    xyz = np.asarray(shells.xyz).reshape(-1, 3)
    ex = [np.asarray(shells.expn[o:o + k]) for o, k in zip(shells.prim_off, shells.nprim)]
    for i in range(shells.nshell):
        for j in range(i + 1):
            r2 = float(np.sum((xyz[i] - xyz[j]) ** 2))
            a, b = ex[i][:, None], ex[j][None, :]
            k = int(np.count_nonzero(a * b / (a + b) * r2 < 41.4))
            c = tuple(sorted((int(shells.L[i]), int(shells.L[j])), reverse=True))
            n, s, s2 = out.get(c, (0, 0, 0))
            out[c] = (n + 1, s + k, s2 + k * k)
    return out


def work(case):
    """Bytes: the basis read once and the results written once (J/K: the density read, two
    matrices written).  Flops: the VRR, contraction and HRR of the unique quartets over the
    primitive quartets that are not negligible (the counts of the package's flops module)."""
    _package()
    F = importlib.import_module(_PKG + ".flops")
    flops = nbytes = 0.0
    for sh in _molecules(case, 0):
        counts = _pair_counts(sh)
        order = sorted(counts, key=lambda c: (c[0] + c[1], c[0]))
        for x, X in enumerate(order):
            nx, sx, qx = counts[X]
            for Y in order[:x + 1]:
                ny, sy, _ = counts[Y]
                nq, kq = (nx * (nx + 1) / 2, (sx * sx + qx) / 2) if X == Y else (nx * ny, sx * sy)
                flops += kq * F.per_prim_flops(*X, *Y) + nq * F.hrr_flops(*X, *Y)
        n_in = 8 * (3 * sh.nshell + 2 * len(sh.expn)) + 12 * sh.nshell
        nbytes += n_in + (24 * sh.nbf ** 2 if case["kind"] == "jk" else 8 * sh.npacked)
        if case["kind"] == "jk":
            flops += 12.0 * sh.npacked  # two Coulomb and four exchange updates per integral
    return {"bytes": nbytes, "flops": flops}


# ------------------------------------------------------------------------------ exact values
# The integrals by the McMurchie-Davidson scheme in 64 bits: Hermite expansion coefficients of
# every primitive pair, Hermite Coulomb integrals from the Boys function, contracted by einsum.
# It shares no step with the engine's HGP and Rys recurrences.

def _components(l):
    c = [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]
    if l == 3:  # the package lists xzz before xyz
        c[4], c[5] = c[5], c[4]
    return c


def _fact2(n):
    return float(np.prod(np.arange(n, 0, -2))) if n > 0 else 1.0


def _hermite(order):
    return [(t, u, v) for t in range(order + 1) for u in range(order + 1 - t) for v in range(order + 1 - t - u)]


def _norms(l, a, c):
    """Normalised coefficients of one contracted shell (without the component factor)."""
    s = np.sum(c[:, None] * c[None, :] * (2 * np.sqrt(a[:, None] * a[None, :]) / (a[:, None] + a[None, :])) ** (l + 1.5))
    return c * (2 * a / math.pi) ** 0.75 * (4 * a) ** (0.5 * l) / math.sqrt(s)


class _ExactPairs:
    """The shell pairs of one class: primitive pairs with their Hermite coefficient tensors."""

    def __init__(self, sh, la, lb, pairs, dev):
        xyz = np.asarray(sh.xyz).reshape(-1, 3)
        first = np.concatenate([[0], np.cumsum([(l + 1) * (l + 2) // 2 for l in sh.L])])
        a, b, k, A, B, own = [], [], [], [], [], []
        fn = []
        ncomp = [np.array([1 / math.sqrt(_fact2(2 * x - 1) * _fact2(2 * y - 1) * _fact2(2 * z - 1))
                           for x, y, z in _components(l)]) for l in (la, lb)]
        for n, (i, j) in enumerate(pairs):
            prim = []
            for s in (i, j):
                o, m = int(sh.prim_off[s]), int(sh.nprim[s])
                e = np.asarray(sh.expn[o:o + m], dtype=np.float64)
                prim.append((e, _norms(int(sh.L[s]), e, np.asarray(sh.coef[o:o + m], dtype=np.float64))))
            (ea, ca), (eb, cb) = prim
            aa, bb = [x.ravel() for x in np.meshgrid(ea, eb, indexing="ij")]
            a.append(aa)
            b.append(bb)
            k.append(np.outer(ca, cb).ravel())
            A.append(np.repeat(xyz[i][None], aa.size, 0))
            B.append(np.repeat(xyz[j][None], aa.size, 0))
            own.append(np.full(aa.size, n))
            fn.append((first[i], first[j]))
        a, b, k, own = (np.concatenate(v) for v in (a, b, k, own))
        A, B = np.concatenate(A), np.concatenate(B)
        p = a + b
        ab = A - B
        pa, pb = -(b / p)[:, None] * ab, (a / p)[:, None] * ab
        k = k * np.exp(-a * b / p * np.sum(ab * ab, axis=1)) / p
        L = la + lb
        E = [self._expansion(la, lb, p, pa[:, x], pb[:, x]) for x in range(3)]
        herm = _hermite(L)
        ca, cb = _components(la), _components(lb)
        T = np.zeros((a.size, len(ca) * len(cb), len(herm)))
        for x, m in enumerate(ca):
            for y, n in enumerate(cb):
                f = k * ncomp[0][x] * ncomp[1][y]
                for h, (t, u, v) in enumerate(herm):
                    if t <= m[0] + n[0] and u <= m[1] + n[1] and v <= m[2] + n[2]:
                        T[:, x * len(cb) + y, h] = f * E[0][m[0], n[0], t] * E[1][m[1], n[1], u] * E[2][m[2], n[2], v]
        self.order, self.herm, self.ncomp = L, herm, len(ca) * len(cb)
        self.p = torch.from_numpy(p).to(dev)
        self.P = torch.from_numpy(A + pa).to(dev)
        self.T = torch.from_numpy(T).to(dev)
        self.own = torch.from_numpy(own).to(dev)
        self.start = np.searchsorted(own, np.arange(len(pairs) + 1))
        i = np.array([f[0] for f in fn])[:, None, None] + np.arange(len(ca))[None, :, None]
        j = np.array([f[1] for f in fn])[:, None, None] + np.arange(len(cb))[None, None, :]
        hi, lo = np.maximum(i, j), np.minimum(i, j)
        self.ij = torch.from_numpy((hi * (hi + 1) // 2 + lo).reshape(len(pairs), -1)).to(dev)

    @staticmethod
    def _expansion(la, lb, p, pa, pb):
        """E[i, j, t] of one axis (the exponential factor is in the pair's coefficient)."""
        E = np.zeros((la + 1, lb + 1, la + lb + 2, p.size))
        E[0, 0, 0] = 1.0
        for i in range(la + 1):
            for j in range(lb + 1):
                if i == j == 0:
                    continue
                src, x = (E[i - 1, j], pa) if i > 0 else (E[i, j - 1], pb)
                for t in range(i + j + 1):
                    v = x * src[t] + (t + 1) * src[t + 1]
                    if t > 0:
                        v = v + src[t - 1] / (2 * p)
                    E[i, j, t] = v
        return E


def _boys(order, T, t_switch):
    """F_0 .. F_order; from t_switch the asymptotic form, as the Boys mode of the case has it."""
    x = T.clamp(max=t_switch)
    term = torch.full_like(x, 1.0 / (2 * order + 1))
    total = term.clone()
    for k in range(1, int(3 * t_switch + 40)):
        term = term * (2 * x / (2 * order + 2 * k + 1))
        total += term
    low = torch.exp(-x)
    F = [None] * (order + 1)
    F[order] = low * total
    for m in range(order - 1, -1, -1):
        F[m] = (2 * x * F[m + 1] + low) / (2 * m + 1)
    far = T >= t_switch
    big = torch.where(far, T, torch.ones_like(T))
    g = 0.5 * torch.sqrt(math.pi / big)
    for m in range(order + 1):
        F[m] = torch.where(far, g, F[m])
        g = g * (2 * m + 1) / (2 * big)
    return F


def _coulomb(order, alpha, R, t_switch):
    """Hermite Coulomb integrals {(t, u, v): tensor}, t+u+v <= order."""
    F = _boys(order, alpha * (R * R).sum(-1), t_switch)
    X = R.unbind(-1)
    cur = {}
    for n in range(order, -1, -1):
        nxt = {(0, 0, 0): (-2 * alpha) ** n * F[n]}
        for h in sorted(_hermite(order - n), key=sum):
            if h == (0, 0, 0):
                continue
            ax = max(range(3), key=lambda d: h[d])
            one = tuple(h[d] - (d == ax) for d in range(3))
            v = X[ax] * cur[one]
            if one[ax] > 0:
                v = v + one[ax] * cur[tuple(one[d] - (d == ax) for d in range(3))]
            nxt[h] = v
        cur = nxt
    return cur


def _exact_packed(sh, t_switch, dev):
    """The packed vector of one molecule."""
    out = torch.zeros(sh.npacked, dtype=torch.float64, device=dev)
    by = {}
    for i in range(sh.nshell):
        for j in range(i + 1):
            a, b = (i, j) if sh.L[i] >= sh.L[j] else (j, i)
            by.setdefault((int(sh.L[a]), int(sh.L[b])), []).append((a, b))
    cls = [_ExactPairs(sh, la, lb, v, dev) for (la, lb), v in sorted(by.items(), key=lambda c: (sum(c[0]), c[0]))]
    room = 1 << (27 if dev == "cuda" else 21)
    for x, X in enumerate(cls):
        for Y in cls[:x + 1]:
            order = X.order + Y.order
            nh = len(_hermite(order)) * 2
            cell = max(2 * len(X.herm) * len(Y.herm), nh, 2 * X.ncomp * Y.ncomp, 2 * X.ncomp * len(Y.herm), 8)
            index = {h: n for n, h in enumerate(_hermite(order))}
            sel = torch.tensor([[index[tuple(s + t for s, t in zip(g, h))] for h in Y.herm] for g in X.herm], device=dev)
            sign = torch.tensor([(-1.0) ** sum(h) for h in Y.herm], dtype=torch.float64, device=dev)
            nket = len(Y.start) - 1
            # chunks of whole shell pairs on both sides
            k0 = 0
            while k0 < nket:
                k1 = k0 + 1
                while k1 < nket and (Y.start[k1 + 1] - Y.start[k0]) * cell * 16 <= room:
                    k1 += 1
                ks = slice(int(Y.start[k0]), int(Y.start[k1]))
                nk = ks.stop - ks.start
                b0 = k0 if X is Y else 0
                nbra = len(X.start) - 1
                while b0 < nbra:
                    b1 = b0 + 1
                    while b1 < nbra and (X.start[b1 + 1] - X.start[b0]) * nk * cell <= room:
                        b1 += 1
                    bs = slice(int(X.start[b0]), int(X.start[b1]))
                    nb = bs.stop - bs.start
                    if nb and nk:
                        p, q = X.p[bs][:, None], Y.p[ks][None, :]
                        alpha = p * q / (p + q)
                        C = _coulomb(order, alpha, X.P[bs][:, None] - Y.P[ks][None], t_switch)
                        pref = 2 * math.pi ** 2.5 / torch.sqrt(p + q)
                        C = torch.stack([C[h] * pref for h in _hermite(order)], -1)
                        M = C[..., sel.reshape(-1)].reshape(nb, nk, len(X.herm), len(Y.herm)) * sign
                        del C
                        G = torch.matmul(X.T[bs][:, None], M)
                        del M
                        G = torch.matmul(G, Y.T[ks][None].transpose(-1, -2))  # [nb, nk, ab, cd]
                        S = torch.zeros(nb, k1 - k0, X.ncomp, Y.ncomp, dtype=torch.float64, device=dev)
                        S.index_add_(1, Y.own[ks] - k0, G)
                        del G
                        Q = torch.zeros(b1 - b0, k1 - k0, X.ncomp, Y.ncomp, dtype=torch.float64, device=dev)
                        Q.index_add_(0, X.own[bs] - b0, S)
                        ij, kl = X.ij[b0:b1][:, None, :, None], Y.ij[k0:k1][None, :, None, :]
                        hi, lo = torch.maximum(ij, kl), torch.minimum(ij, kl)
                        out[(hi * (hi + 1) // 2 + lo).reshape(-1)] = Q.reshape(-1)
                    b0 = b1
                k0 = k1
    return out


def exact(case, seed):
    mols = _molecules(case, seed)
    # about 20 s: primitive quartets weighted by the size of the Hermite tables
    cost = 0.0
    for sh in mols:
        c = _pair_counts(sh)
        k = np.array([int(x) * int(y) for i, x in enumerate(sh.nprim) for y in sh.nprim[:i + 1]], dtype=float)
        w = sum(s for _, s, _ in c.values()) / max(1, sum(n for n, _, _ in c.values()))
        lmax = max(la + lb for la, lb in c)
        cost += (k.sum() ** 2) * max(1.0, w / 8) * (1 + lmax) ** 2
    if cost > 4e11:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    t_switch = 40.0 if case["boys"] == "exact" or case.get("method") == "rys" else 30.0
    vecs = [_exact_packed(sh, t_switch, dev) for sh in mols]
    if case["kind"] == "serve":
        return vecs
    if case["kind"] == "batch":
        return torch.cat(vecs)
    if case["kind"] != "jk":
        return vecs[0]
    n = mols[0].nbf
    if n > 170:
        return None
    i = torch.arange(n, device=dev)
    hi, lo = torch.maximum(i[:, None], i[None]), torch.minimum(i[:, None], i[None])
    pair = hi * (hi + 1) // 2 + lo
    D = torch.from_numpy(_density(n, seed)).to(dev)
    J = torch.empty(n, n, dtype=torch.float64, device=dev)
    K = torch.empty(n, n, dtype=torch.float64, device=dev)
    for r in range(n):  # (r q | s t) for all q, s, t
        a, b = torch.maximum(pair[r][:, None, None], pair[None]), torch.minimum(pair[r][:, None, None], pair[None])
        V = vecs[0][a * (a + 1) // 2 + b]
        J[r] = (V * D[None]).sum((1, 2))
        K[r] = torch.einsum("qst,qt->s", V, D)
    return {"J": J, "K": K}
