"""Generate the per-class ERI kernels (CUDA C for sm_100a).

This is the engine's counterpart of the reference's ``vrr_autogen`` (src/HGP.jl:432-534),
which emits unrolled, branch-free Julia VRR code per (amax, cmax).  Here one kernel is
emitted per class pair (la lb | lc ld) with la >= lb, lc >= ld and the bra class at or
above the ket class.  Each kernel evaluates one contracted shell quartet per thread:

  * the HGP vertical recurrence of src/HGP.jl:135-242 -- the a-build (eq. 6a with c = 0,
    :180-197) and the c-build (eq. 6d, :204-240) -- unrolled and pruned to the
    [a0|c0]^(m) entries the class needs, in registers (FP64, or FP32 for MIXED quartets);
  * contraction over the primitive quartets in FP64 after the VRR (cvrr, :50-68);
  * the horizontal recurrences of chrr (:87-114) on the contracted block, bra then ket;
  * the component norms 1/sqrt((2I-1)!!(2J-1)!!(2K-1)!!) and the packed iindex store of
    the quartet's unique integrals.

Run ``python gen_eri.py`` to (re)write ``generated/``; the build does it automatically.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

HERE = Path(__file__).resolve().parent
OUT_DIR = HERE / "generated"


def _load_gen_rys():
    import importlib.util
    if "gen_rys" in sys.modules:
        return sys.modules["gen_rys"]
    spec = importlib.util.spec_from_file_location("gen_rys", HERE / "gen_rys.py")
    mod = importlib.util.module_from_spec(spec)
    sys.modules["gen_rys"] = mod
    spec.loader.exec_module(mod)
    return mod


gen_rys = _load_gen_rys()
LMAX = 3            # shell angular momentum of the classes considered
LMAX_ALL_HGP = 2    # every class pair of shells up to d has an HGP kernel
LTAB = 2 * LMAX     # AO tables must reach la + lb
# Class pairs with an f shell get an HGP kernel when their VRR has at most this many entries
# (the low-L partners of f, e.g. (fs|ss), (fp|ps)); the rest run only the Rys kernels.
HGP_MAX_VRR = 500
# Classes whose VRR has fewer entries than this get no FP32 variant: their primitive
# quartet is dominated by the FP64 prefactors and Boys function, so an FP32 VRR would only
# add registers and divergence.  MIXED plans run them in FP64.
MIXED_MIN_VRR = 40
# Two-phase stores: classes with at most this many outputs per quartet have their HRR write the
# chunk's blocks into dynamic shared memory (4 warps x 32 blocks x 8 B each: up to 162 KB) and
# the warp copies them to the scratch as one contiguous run
STAGE_MAX_OUT = 162
# Pair classes whose bounds the Rys bound kernel computes although an HGP kernel exists: the HGP
# (dd|dd) kernel's straight-line code takes 34 us for a handful of pairs
RYS_BOUND = {(2, 2)}
# J/K digestion: blocks of at most this many outputs are digested from registers; larger ones sit in
# local memory, read by a loop over A's components
JK_UNROLL_MAX_OUT = 36
# Resident blocks asked of the compiler where it misses a step by a few registers: (ps|ss) takes 66,
# seven blocks of 128; eight at 64 registers: 1030 -> 1001 us over 1.17e9 integrals on B200 (the J/K
# instantiation would spill 60 bytes for it and is left as it is)
MIN_BLOCKS = {((1, 0), (0, 0)): 8}


# ------------------------------------------------------------------ AO tables
def shell_components(l):
    """src/Basis.jl:269-279 order (x-power descending, then y), l=3 with xzz before xyz."""
    comps = [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]
    if l == 3:
        comps[4], comps[5] = comps[5], comps[4]
    return comps


AO = []           # cumulative AO list (ao2m, src/Basis.jl:306-314), 0-based
NAO = []          # cumulative counts (nao, src/Basis.jl:320-321)
for _l in range(LTAB + 1):
    AO.extend(shell_components(_l))
    NAO.append(len(AO))
AO_INDEX = {c: i for i, c in enumerate(AO)}


def lof(a):
    return sum(AO[a])


def shell_range(l):
    return range(NAO[l - 1] if l > 0 else 0, NAO[l])


def shift_dir(a):
    """First argmax of the powers (shift_direction, src/Basis.jl:346-354)."""
    m = AO[a]
    return max(range(3), key=lambda i: (m[i], -i))


def shift_minus(a, i):
    m = list(AO[a])
    if m[i] == 0:
        return -1
    m[i] -= 1
    return AO_INDEX[tuple(m)]


def shift_plus(a, i):
    m = list(AO[a])
    m[i] += 1
    return AO_INDEX[tuple(m)]


def dfact2(n):
    r = 1
    while n > 1:
        r *= n
        n -= 2
    return r


def comp_norm(a):
    I, J, K = AO[a]
    return 1.0 / math.sqrt(dfact2(2 * I - 1) * dfact2(2 * J - 1) * dfact2(2 * K - 1))


XYZ = "xyz"


# ------------------------------------------------------------------ classes
def pair_classes(lmax=LMAX):
    """Shell-pair classes (la, lb), la >= lb, ordered by la+lb then la."""
    cls = [(la, lb) for la in range(lmax + 1) for lb in range(la + 1)]
    return sorted(cls, key=lambda c: (c[0] + c[1], c[0]))


def class_pairs(lmax=LMAX):
    """Class pairs (X|Y), X at or above Y, that get an HGP kernel."""
    cls = pair_classes(lmax)
    out = []
    for i, X in enumerate(cls):
        for j in range(i + 1):
            Y = cls[j]
            if max(X + Y) > LMAX_ALL_HGP and \
                    len(vrr_entries(X[0], X[0] + X[1], Y[0], Y[0] + Y[1])) > HGP_MAX_VRR:
                continue
            out.append((X, Y))
    return out


def tag_of(X, Y):
    L = "spdfg"
    return f"{L[X[0]]}{L[X[1]]}{L[Y[0]]}{L[Y[1]]}"


# ------------------------------------------------------------------ VRR plan
def vrr_entries(e_lo, e_hi, f_lo, f_hi):
    """Needed [a0|c0]^(m) entries, in an order where every entry follows its inputs."""
    need = set()
    stack = [(a, c, 0) for a in range(NAO[e_lo - 1] if e_lo else 0, NAO[e_hi])
             for c in range(NAO[f_lo - 1] if f_lo else 0, NAO[f_hi])]
    while stack:
        key = stack.pop()
        if key in need:
            continue
        need.add(key)
        stack.extend(vrr_deps(*key))
    return sorted(need, key=lambda k: (k[1], k[0], k[2]))


def vrr_deps(a, c, m):
    if c == 0:
        if a == 0:
            return []
        i = shift_dir(a)
        am = shift_minus(a, i)
        amm = shift_minus(am, i)
        d = [(am, 0, m), (am, 0, m + 1)]
        if amm >= 0:
            d += [(amm, 0, m), (amm, 0, m + 1)]
        return d
    i = shift_dir(c)
    cm = shift_minus(c, i)
    cmm = shift_minus(cm, i)
    am = shift_minus(a, i)
    d = [(a, cm, m), (a, cm, m + 1)]
    if am >= 0:
        d.append((am, cm, m + 1))
    if cmm >= 0:
        d += [(a, cmm, m), (a, cmm, m + 1)]
    return d


def vname(a, c, m):
    return f"v{a}_{c}_{m}"


def vrr_line(a, c, m):
    """The recurrence of src/HGP.jl:189-190 / :218-236 for one entry."""
    if c == 0:
        if a == 0:
            return f"const VT {vname(0, 0, m)} = (VT)(pref * F[{m}]);"
        i = shift_dir(a)
        am = shift_minus(a, i)
        amm = shift_minus(am, i)
        x = XYZ[i]
        s = f"PA{x} * {vname(am, 0, m)} + WP{x} * {vname(am, 0, m + 1)}"
        if amm >= 0:
            k = AO[am][i]
            s += (f" + (VT){k}.0 * oo2z * ({vname(amm, 0, m)} - rho_z * "
                  f"{vname(amm, 0, m + 1)})")
        return f"const VT {vname(a, 0, m)} = {s};"
    i = shift_dir(c)
    cm = shift_minus(c, i)
    cmm = shift_minus(cm, i)
    am = shift_minus(a, i)
    x = XYZ[i]
    s = f"QC{x} * {vname(a, cm, m)} + WQ{x} * {vname(a, cm, m + 1)}"
    if am >= 0:
        s += f" + (VT){AO[a][i]}.0 * oo2ze * {vname(am, cm, m + 1)}"
    if cmm >= 0:
        k = AO[cm][i]
        s += f" + (VT){k}.0 * oo2e * ({vname(a, cmm, m)} - rho_e * {vname(a, cmm, m + 1)})"
    return f"const VT {vname(a, c, m)} = {s};"


def vrr_terms(a, c):
    """The recurrence of entry (a, c)^(0) as (factor, entry) products."""
    if c == 0:
        if a == 0:
            return [("pref", "F[0]")]
        i = shift_dir(a)
        am = shift_minus(a, i)
        amm = shift_minus(am, i)
        x = XYZ[i]
        t = [(f"PA{x}", vname(am, 0, 0)), (f"WP{x}", vname(am, 0, 1))]
        if amm >= 0:
            k = AO[am][i]
            t.append((f"{k}.0 * oo2z", f"({vname(amm, 0, 0)} - rho_z * {vname(amm, 0, 1)})"))
        return t
    i = shift_dir(c)
    cm = shift_minus(c, i)
    cmm = shift_minus(cm, i)
    am = shift_minus(a, i)
    x = XYZ[i]
    t = [(f"QC{x}", vname(a, cm, 0)), (f"WQ{x}", vname(a, cm, 1))]
    if am >= 0:
        t.append((f"{AO[a][i]}.0 * oo2ze", vname(am, cm, 1)))
    if cmm >= 0:
        k = AO[cm][i]
        t.append((f"{k}.0 * oo2e", f"({vname(a, cmm, 0)} - rho_e * {vname(a, cmm, 1)})"))
    return t


# ------------------------------------------------------------------ HRR plan
class HrrPlan:
    """(ab|cd) from the contracted [a0|c0] block: bra HRR then ket HRR (src/HGP.jl:92-114)."""

    def __init__(self, la, lb, lc, ld):
        self.la, self.lb, self.lc, self.ld = la, lb, lc, ld
        self.lines = []
        self.done = {}
        e, f = la + lb, lc + ld
        self.acc_a = [a for l in range(la, e + 1) for a in shell_range(l)]
        self.acc_c = [c for l in range(lc, f + 1) for c in shell_range(l)]
        self.acc_index = {(a, c): i * len(self.acc_c) + j
                          for i, a in enumerate(self.acc_a) for j, c in enumerate(self.acc_c)}
        self.targets = []
        for a in shell_range(la):
            for b in shell_range(lb):
                for c in shell_range(lc):
                    for d in shell_range(ld):
                        self.targets.append((a, b, c, d, self.ket(a, b, c, d)))

    def bra(self, a, b, c):
        if b == 0:
            return f"acc[{self.acc_index[(a, c)]}]"
        key = ("h", a, b, c)
        if key in self.done:
            return self.done[key]
        j = shift_dir(b)
        bm = shift_minus(b, j)
        t1 = self.bra(shift_plus(a, j), bm, c)
        t2 = self.bra(a, bm, c)
        name = f"h{a}_{b}_{c}"
        self.lines.append(f"const double {name} = {t1} + AB{XYZ[j]} * {t2};")
        self.done[key] = name
        return name

    def ket(self, a, b, c, d):
        if d == 0:
            return self.bra(a, b, c)
        key = ("k", a, b, c, d)
        if key in self.done:
            return self.done[key]
        j = shift_dir(d)
        dm = shift_minus(d, j)
        t1 = self.ket(a, b, shift_plus(c, j), dm)
        t2 = self.ket(a, b, c, dm)
        name = f"k{a}_{b}_{c}_{d}"
        self.lines.append(f"const double {name} = {t1} + CD{XYZ[j]} * {t2};")
        self.done[key] = name
        return name


# ------------------------------------------------------------------ emit
def rys_lane_lines(X, Y, hp):
    """One root's 2-D tables in registers (the recurrences of gen_rys) and its products into acc:
    the body of the root loop of a lane-split Rys kernel."""
    e, f = X[0] + X[1], Y[0] + Y[1]
    out = []
    for x in XYZ:
        out.append(f"const double C{x} = fma(-ez * PQ{x}, u, bra.pa{x}), D{x} = fma(zz * PQ{x}, u, ket.pa{x});")
        out.append(f"(void)C{x}; (void)D{x};")
    for x in XYZ:
        for c in range(f + 1):
            for a in range(e + 1):
                n = f"{x}{a}_{c}"
                if a == c == 0:
                    out.append(f"const double {n} = {'pref * w' if x == 'x' else '1.0'};")
                elif c == 0:
                    s = f"C{x} * {x}{a - 1}_0" + (f" + {a - 1}.0 * b10 * {x}{a - 2}_0" if a > 1 else "")
                    out.append(f"const double {n} = {s};")
                else:
                    s = f"D{x} * {x}{a}_{c - 1}"
                    s += f" + {c - 1}.0 * b01 * {x}{a}_{c - 2}" if c > 1 else ""
                    s += f" + {a}.0 * b00 * {x}{a - 1}_{c - 1}" if a else ""
                    out.append(f"const double {n} = {s};")
    for a in hp.acc_a:
        for c in hp.acc_c:
            m, n = AO[a], AO[c]
            out.append(f"acc[{hp.acc_index[(a, c)]}] = fma(x{m[0]}_{n[0]} * y{m[1]}_{n[1]}, z{m[2]}_{n[2]}, "
                       f"acc[{hp.acc_index[(a, c)]}]);")
    return out


def has_schwarz(X):
    """Whether the HGP bound kernel computes the bounds of pair class X (else the Rys one does)."""
    return (X, X) in class_pairs() and X not in RYS_BOUND


def emit_class_pair(X, Y, rys=False):
    """The lane-split class kernel of (X|Y): HGP, or (rys) the same kernel with the primitive
    quartets by Rys quadrature (gen_rys: class pairs of small blocks)."""
    (la, lb), (lc, ld) = X, Y
    tag = tag_of(X, Y) + ("_rys" if rys else "")
    e, f = la + lb, lc + ld
    M = e + f
    entries = vrr_entries(la, e, lc, f)
    hp = HrrPlan(la, lb, lc, ld)
    nacc = len(hp.acc_a) * len(hp.acc_c)
    na, nb, nc, nd = [len(shell_range(l)) for l in (la, lb, lc, ld)]
    nout = na * nb * nc * nd
    ind = "        "
    # entries that only go into the block: in FP64 their products are added to it one by one (an FMA
    # each), without forming the entry; entries of the FP32 variant are formed and added in FP64
    used = {d for k in entries for d in vrr_deps(*k)}
    block = [(a, c) for a in hp.acc_a for c in hp.acc_c]
    leaf = {(a, c) for a, c in block if (a, c, 0) not in used}
    vrr_code = "\n".join(ind + "    " + vrr_line(*k) for k in entries if k[2] or (k[0], k[1]) not in leaf)
    acc64, acc32 = [], []
    for a, c in block:
        i = hp.acc_index[(a, c)]
        if (a, c) not in leaf:
            acc64.append(f"acc[{i}] += (double){vname(a, c, 0)};")
            acc32.append(acc64[-1])
            continue
        t = vrr_terms(a, c)
        if M == 1 and a:  # (ps|ss): W - P = -rho_z (P - Q), used once an axis
            x = XYZ[shift_dir(a)]
            t = [(f"PA{x}", vname(0, 0, 0)), (f"PQ{x}", f"(-ez * {vname(0, 0, 1)})")]
        e = f"acc[{i}]"
        for f, v in t[::-1]:
            e = f"fma({f}, {v}, {e})"
        acc64.append(f"acc[{i}] = {e};")
        acc32 += [vrr_line(a, c, 0), f"acc[{i}] += (double){vname(a, c, 0)};"]
    has32 = len(entries) >= MIXED_MIN_VRR and not rys
    bounds = f", JK ? 1 : {MIN_BLOCKS[(X, Y)]}" if (X, Y) in MIN_BLOCKS and not rys else ""

    def lines(x, extra=""):
        return "\n".join(f"{ind}    {extra}{ln}" for ln in x)
    acc_code = lines(acc64) if not has32 else (
        f"{ind}    if constexpr (sizeof(VT) == 8) {{\n{lines(acc64, '    ')}\n{ind}    }} else {{\n"
        f"{lines(acc32, '    ')}\n{ind}    }}")
    hrr_code = "\n".join("    " + ln for ln in hp.lines)
    out_code = []
    for x, (a, b, c, d, expr) in enumerate(hp.targets):
        g = comp_norm(a) * comp_norm(b) * comp_norm(c) * comp_norm(d)
        if abs(g - 1.0) < 1e-15:
            out_code.append(f"    res[{x}] = {expr};")
        else:
            out_code.append(f"    res[{x}] = {expr} * {g!r};")
    out_code = "\n".join(out_code)
    stores = []
    for ia in range(na):
        for ib in range(nb):
            for ic in range(nc):
                for id_ in range(nd):
                    x = ((ia * nb + ib) * nc + ic) * nd + id_
                    conds = []
                    if la == lb:
                        conds.append(f"(!dab || {ia} >= {ib})")
                    if lc == ld:
                        conds.append(f"(!dcd || {ic} >= {id_})")
                    cond = " && ".join(conds) if conds else "true"
                    stores.append(
                        f"    {{ const long long ij = ij_{ia}_{ib}, kl = kl_{ic}_{id_};\n"
                        f"      if ({cond} && (!same || ij >= kl)) "
                        f"out[packed_index(ij, kl)] = res[{x}]; }}")
    ij_code = "\n".join(f"    const long long ij_{ia}_{ib} = pair_index(ib_.z + {ia}, ib_.w + {ib});"
                        for ia in range(na) for ib in range(nb))
    kl_code = "\n".join(f"    const long long kl_{ic}_{id_} = pair_index(ik_.z + {ic}, ik_.w + {id_});"
                        for ic in range(nc) for id_ in range(nd))
    store_code = "\n".join(stores)
    schwarz = ""
    if X == Y and not rys and has_schwarz(X):
        diag = []
        for ia in range(na):
            for ib in range(nb):
                x = ((ia * nb + ib) * nc + ia) * nd + ib
                diag.append(f"    m = fmax(m, fabs(res[{x}]));")
        diag = "\n".join(diag)
        accdiag = "\n".join(f"        w = fmax(w, fabs(acc[{hp.acc_index[(a, a)]}]));" for a in hp.acc_a)
        schwarz = f"""
// Bounds of the pairs of one class.
// full == 0 (plan set-up): for every primitive pair k of pair p, from the diagonal primitive
//   quartet (a_k b_k | a_k b_k):
//     pbound[k].x = b_k = sqrt(max over components |(a_k b_k|a_k b_k)|)
//     pbound[k].y = w_k = sqrt(max over the VRR block |[e0|e0]_kk|), e = la..la+lb
//   By the Schwarz inequality b_k b_l bounds |(a_k b_k|c_l d_l)| and w_k w_l bounds every
//   entry of the VRR output block [e0|f0] that the HRR combines.
//   qmax[mol[p]]: the largest sum of b_k (in list order) over the molecule's pairs, as bits.
// full != 0: the contracted bound Q_p = sqrt(max |(ab|ab)|) into qout[p].
// A warp per pair, its lanes over the primitive pairs (one thread per pair, over up to 49 primitive
// pairs in turn, took 46 us for (ss) on B200).  The contracted bound takes one lane of it: pairs of unlike
// length then do not wait for one another (molints_plan_schwarz of 36 split-valence atoms 445 us, with
// a thread per pair 530; 24 polarised atoms 754 and 920).
__global__ void __launch_bounds__(128) schwarz_kernel_{tag}(PairTab P, BoysTab B, int p0, int np,
                                                          double2 *pbound, const int *mol,
                                                          unsigned long long *qmax, double *qout, int full) {{
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= np) return;
    const int p = p0 + t;
    const int4 in = __ldg(&P.info[p]);
    double res[{nout}];
    if (full) {{
        if (lane) return;
        quartet_{tag}<double>(P, B, p, p, 0, in.y, 0, in.y, res);
        double m = 0.0;
{diag}
        qout[p] = sqrt(m);
        return;
    }}
    double acc[{nacc}], q = 0.0;
    for (int k0 = 0; k0 < in.y; k0 += 32) {{
        const int k = k0 + lane;
        double m = 0.0, w = 0.0;
        if (k < in.y) {{
            quartet_{tag}<double>(P, B, p, p, k, k + 1, k, k + 1, res, acc);
{diag}
{accdiag}
            m = sqrt(m);
            pbound[in.x + k] = make_double2(m, sqrt(w));
        }}
        const int n = min(32, in.y - k0);
        for (int x = 0; x < n; ++x) q += __shfl_sync(0xffffffffu, m, x);
    }}
    // the sums are >= 0, so their bit patterns order like the values
    if (lane == 0) atomicMax(&qmax[__ldg(&mol[p])], (unsigned long long)__double_as_longlong(q));
}}

void launch_schwarz_{tag}(const PairTab &P, const BoysTab &B, int p0, int np, double2 *pbound,
                          const int *mol, unsigned long long *qmax, double *qout, int full, cudaStream_t s) {{
    if (np <= 0) return;
    schwarz_kernel_{tag}<<<(np + 3) / 4, 128, 0, s>>>(P, B, p0, np, pbound, mol, qmax, qout, full);
}}
"""
    if nout <= STAGE_MAX_OUT:
        sbytes = 4 * 32 * nout * 8
        mixed_attr = (f"        cudaFuncSetAttribute(eri_queue_{tag}<1, 0>, "
                      f"cudaFuncAttributeMaxDynamicSharedMemorySize, {sbytes});\n"
                      if has32 else "")
        stage_fn = (f"""
// The dynamic shared memory of the two-phase staging ({sbytes} bytes), allowed once per device
// (before any graph capture: the occupancy query of plan creation calls it first).
static void eri_prepare_{tag}() {{
    static bool done[64] = {{false}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {{
        cudaFuncSetAttribute(eri_queue_{tag}<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, {sbytes});
{mixed_attr}        done[dev] = true;
    }}
}}
""" if sbytes > 48 * 1024 else "")
        stage_prep = (f"    // two-phase plans stage the chunk's blocks in {sbytes} bytes of dynamic shared memory\n"
                      f"    const size_t smem = Q.scratch && !Q.jk.J ? {sbytes} : 0;" +
                      (f"\n    if (smem) eri_prepare_{tag}();" if sbytes > 48 * 1024 else ""))
        occ_prep = f"    eri_prepare_{tag}();" if sbytes > 48 * 1024 else ""
    else:
        stage_fn, occ_prep = "", ""
        stage_prep = "    constexpr size_t smem = 0;"
    if nout <= STAGE_MAX_OUT:
        scratch_store = f"""            // two-phase: the leaders' HRR writes the blocks of the chunk's quartets straight
            // into shared memory, where they lie as in the scratch (consecutive slots); the warp
            // then copies them out as one contiguous run
            extern __shared__ double stg[];  // 4 * 32 * {nout} doubles (launch_eri_{tag})
            double *sb = stg + (threadIdx.x >> 5) * (32 * {nout});
            if (lead) hrr_{tag}(Q.pairs, p, q, acc, sb + kq * {nout});
            __syncwarp();
            const int nlive = min(W, cnt - base);
            double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                (__ldg(&Q.chunk_slot[c]) + base) * (long long){nout};
            for (int t = lane; t < nlive * {nout}; t += 32) dst[t] = sb[t];
            __syncwarp();"""
    else:
        scratch_store = f"""            // two-phase: each leader stores its quartet's whole block at its slot
            if (lead) {{
                double res[{nout}];
                hrr_{tag}(Q.pairs, p, q, acc, res);
                double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                    (__ldg(&Q.chunk_slot[c]) + base + kq) * (long long){nout};
#pragma unroll
                for (int x = 0; x < {nout}; ++x) dst[x] = res[x];
            }}"""
    if has32:
        mixed_dispatch = ("    const bool jk = Q.jk.J != nullptr;\n"
                          "    if (mixed) {{ if (jk) eri_queue_{t}<1, 1><<<grid, 128, 0, s>>>(Q); "
                          "else eri_queue_{t}<1, 0><<<grid, 128, smem, s>>>(Q); }}\n"
                          "    else if (jk) eri_queue_{t}<0, 1><<<grid, 128, 0, s>>>(Q);\n"
                          "    else eri_queue_{t}<0, 0><<<grid, 128, smem, s>>>(Q);").format(t=tag)
        occ_dispatch = ("    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_{t}<1, 0>, 128, 0);\n"
                        "    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_{t}<0, 0>, 128, 0);").format(t=tag)
    else:
        mixed_dispatch = ("    (void)mixed;  // no FP32 variant for this class (MIXED_MIN_VRR)\n"
                          "    if (Q.jk.J) eri_queue_{t}<0, 1><<<grid, 128, 0, s>>>(Q);\n"
                          "    else eri_queue_{t}<0, 0><<<grid, 128, smem, s>>>(Q);").format(t=tag)
        occ_dispatch = ("    (void)mixed;\n"
                        "    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_{t}<0, 0>, 128, 0);").format(t=tag)
    if rys:
        nr = M // 2 + 1
        body = "\n".join(ind + "        " + ln for ln in rys_lane_lines(X, Y, hp))
        vrr_fn = f"""// The contracted [e0|f0] block of bra pair p and ket pair q into acc[{nacc}] by the {nr}-point Rys
// rule, summed over the bra primitive pairs i0, i0 + istep, ... < i1 and the ket primitive pairs
// j0, j0 + jstep, ... < j1; loop order and splits as in the HGP kernel of the class.
__device__ __forceinline__ void vrr_{tag}(const PairTab &P, const RysTab &R, int p, int q, int i0, int i1,
                                          int istep, int j0, int j1, int jstep, double *__restrict__ acc) {{
    const int4 ib_ = __ldg(&P.info[p]);
    const int4 ik_ = __ldg(&P.info[q]);
#pragma unroll
    for (int x = 0; x < {nacc}; ++x) acc[x] = 0.0;
    for (int j = j0; j < j1; j += jstep) {{
        const PrimPair ket = load_pp(P.pp, ik_.x + j);
        for (int i = i0; i < i1; i += istep) {{
            const PrimPair bra = load_pp(P.pp, ib_.x + i);
            const double r = rsqrt(bra.zeta + ket.zeta);
            const double r2 = r * r;
            const double PQx = bra.px - ket.px, PQy = bra.py - ket.py, PQz = bra.pz - ket.pz;
            const double T = bra.zeta * ket.zeta * r2 * (PQx * PQx + PQy * PQy + PQz * PQz);
            const double pref = bra.kab * ket.kab * r;
            const double ez = ket.zeta * r2, zz = bra.zeta * r2;
#pragma unroll 1
            for (int k = 0; k < {nr}; ++k) {{
                double u, w;
                rys_root<{nr}>(R, T, k, u, w);
                const double b10 = bra.oo2z * fma(-ez, u, 1.0), b01 = ket.oo2z * fma(-zz, u, 1.0), b00 = 0.5 * r2 * u;
                (void)b10; (void)b01; (void)b00;
{body}
            }}
        }}
    }}
}}"""
    else:
        vrr_fn = f"""// The contracted [e0|f0] block of bra pair p and ket pair q into acc[{nacc}], summed over
// the bra primitive pairs i0, i0 + istep, ... < i1 and the ket primitive pairs j0, j0 + jstep,
// ... < j1 of the two shell pairs.  VT is the VRR arithmetic type (double, or float for MIXED).
// The ket loop is outside: a warp shares its bra pair, so the inner bra loads are broadcasts
// and each lane's ket record is loaded once.  Steps above 1 split one quartet's primitive
// quartets over the lanes of a split group (their blocks are summed before the HRR).
template <typename VT>
__device__ __forceinline__ void vrr_{tag}(const PairTab &P, const BoysTab &B, int p, int q,
                                          int i0, int i1, int istep, int j0, int j1, int jstep,
                                          double *__restrict__ acc) {{
    const int4 ib_ = __ldg(&P.info[p]);
    const int4 ik_ = __ldg(&P.info[q]);
#pragma unroll
    for (int x = 0; x < {nacc}; ++x) acc[x] = 0.0;
    for (int j = j0; j < j1; j += jstep) {{
        const PrimPair ket = load_pp(P.pp, ik_.x + j);
        for (int i = i0; i < i1; i += istep) {{
            const PrimPair bra = load_pp(P.pp, ib_.x + i);
            const double PQx = bra.px - ket.px, PQy = bra.py - ket.py, PQz = bra.pz - ket.pz;
            // near (T below the switch): r = 1/sqrt(zeta+eta), r2 = r^2.  Far: the same recurrences with
            // r2 = 1/(zeta eta PQ^2) in the place of 1/(zeta+eta) and F_m T^m, constants, in that of
            // F_m -- each factor of r2 comes with one order of F -- so both take one square root
            // and a far lane no other work (boys_scaled)
            const double s = bra.zeta + ket.zeta, ze = bra.zeta * ket.zeta * (PQx * PQx + PQy * PQy + PQz * PQz);
            const bool far = !(ze < B.t_switch * s);
            const double r = rsqrt(far ? ze : s);
            const double r2 = r * r;
            const double ez = ket.zeta * r2, zz = bra.zeta * r2;
            const double pref = bra.kab * ket.kab * r;
            double F[{M + 1}];
            boys_scaled<{M}>(far, ze * r2, B, F);
            const VT PAx = (VT)bra.pax, PAy = (VT)bra.pay, PAz = (VT)bra.paz;
            const VT QCx = (VT)ket.pax, QCy = (VT)ket.pay, QCz = (VT)ket.paz;
            const VT WPx = (VT)(-ez * PQx), WPy = (VT)(-ez * PQy), WPz = (VT)(-ez * PQz);
            const VT WQx = (VT)(zz * PQx), WQy = (VT)(zz * PQy), WQz = (VT)(zz * PQz);
            const VT oo2z = (VT)bra.oo2z, oo2e = (VT)ket.oo2z, oo2ze = (VT)(0.5 * r2);
            const VT rho_z = (VT)ez, rho_e = (VT)zz;
            (void)PAx; (void)PAy; (void)PAz; (void)QCx; (void)QCy; (void)QCz;
            (void)WPx; (void)WPy; (void)WPz; (void)WQx; (void)WQy; (void)WQz;
            (void)oo2z; (void)oo2e; (void)oo2ze; (void)rho_z; (void)rho_e;
{vrr_code}
{acc_code}
        }}
    }}
}}"""
    quartet_fn = "" if rys else f"""// (ab|cd) over the bra primitive pairs [i0, i1) and ket primitive pairs [j0, j1) into
// res[{nout}]; the contracted block also into acc_out when given (the bound kernels).
template <typename VT>
__device__ __forceinline__ void quartet_{tag}(const PairTab &P, const BoysTab &B, int p, int q,
                                              int i0, int i1, int j0, int j1,
                                              double *__restrict__ res,
                                              double *__restrict__ acc_out = nullptr) {{
    double acc[{nacc}];
    vrr_{tag}<VT>(P, B, p, q, i0, i1, 1, j0, j1, 1, acc);
    if (acc_out) {{
#pragma unroll
        for (int x = 0; x < {nacc}; ++x) acc_out[x] = acc[x];
    }}
    hrr_{tag}(P, p, q, acc, res);
}}"""
    # J/K digestion: loops over A's components (unrolled for small blocks, so that res stays in
    # registers), the rest unrolled
    body = []
    for jb in range(nb):
        for ic in range(nc):
            for jd in range(nd):
                body += [f"        {{ const double v = f * res[(i * {nb} + {jb}) * {nc * nd} + {ic * nd + jd}];",
                         f"          jab[i * {nb} + {jb}] = fma(dcd[{ic * nd + jd}], v, jab[i * {nb} + {jb}]);",
                         f"          jcd[{ic * nd + jd}] = fma(dab[{jb}], v, jcd[{ic * nd + jd}]);",
                         f"          kac[{ic}] = fma(dbd[{jb * nd + jd}], v, kac[{ic}]);",
                         f"          kad[{jd}] = fma(dbc[{jb * nc + ic}], v, kad[{jd}]);",
                         f"          kbc[{jb * nc + ic}] = fma(dad[{jd}], v, kbc[{jb * nc + ic}]);",
                         f"          kbd[{jb * nd + jd}] = fma(dac[{ic}], v, kbd[{jb * nd + jd}]); }}"]
    jk_body = "\n".join(body)
    jk_fn = f"""// The quartet's share of J and K (molints_plan_jk, eri_common.cuh): every integral of the block,
// times f, into one orientation of each target; J_ab stays in the lane (one bra pair per chunk).
__device__ __forceinline__ void jk_{tag}(const JKOut &jk, const int4 ib_, const int4 ik_, double f,
                                         const double *__restrict__ res, double *__restrict__ jab) {{
    const long long n = jk.n;
    const double *__restrict__ D = jk.D;
    const double *__restrict__ Db = D + ib_.w * n, *__restrict__ Dc = D + ik_.z * n;
    double dcd[{nc * nd}], dbc[{nb * nc}], dbd[{nb * nd}], jcd[{nc * nd}], kbc[{nb * nc}], kbd[{nb * nd}];
#pragma unroll
    for (int k = 0; k < {nc}; ++k)
#pragma unroll
        for (int l = 0; l < {nd}; ++l) {{
            dcd[k * {nd} + l] = __ldg(&Dc[k * n + ik_.w + l]);
            jcd[k * {nd} + l] = 0.0;
        }}
#pragma unroll
    for (int j = 0; j < {nb}; ++j) {{
#pragma unroll
        for (int k = 0; k < {nc}; ++k) {{
            dbc[j * {nc} + k] = __ldg(&Db[j * n + ik_.z + k]);
            kbc[j * {nc} + k] = 0.0;
        }}
#pragma unroll
        for (int l = 0; l < {nd}; ++l) {{
            dbd[j * {nd} + l] = __ldg(&Db[j * n + ik_.w + l]);
            kbd[j * {nd} + l] = 0.0;
        }}
    }}
#pragma unroll {na if nout <= JK_UNROLL_MAX_OUT else 1}
    for (int i = 0; i < {na}; ++i) {{
        const double *__restrict__ Da = D + (ib_.z + i) * n;
        double dab[{nb}], dac[{nc}], dad[{nd}], kac[{nc}], kad[{nd}];
#pragma unroll
        for (int j = 0; j < {nb}; ++j) dab[j] = __ldg(&Da[ib_.w + j]);
#pragma unroll
        for (int k = 0; k < {nc}; ++k) {{ dac[k] = __ldg(&Da[ik_.z + k]); kac[k] = 0.0; }}
#pragma unroll
        for (int l = 0; l < {nd}; ++l) {{ dad[l] = __ldg(&Da[ik_.w + l]); kad[l] = 0.0; }}
{jk_body}
#pragma unroll
        for (int k = 0; k < {nc}; ++k) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.z + k], kac[k]);
#pragma unroll
        for (int l = 0; l < {nd}; ++l) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.w + l], kad[l]);
    }}
#pragma unroll
    for (int j = 0; j < {nb}; ++j) {{
#pragma unroll
        for (int k = 0; k < {nc}; ++k) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.z + k], kbc[j * {nc} + k]);
#pragma unroll
        for (int l = 0; l < {nd}; ++l) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.w + l], kbd[j * {nd} + l]);
    }}
#pragma unroll
    for (int k = 0; k < {nc}; ++k)
#pragma unroll
        for (int l = 0; l < {nd}; ++l) atomicAdd(&jk.J[(ik_.z + k) * n + ik_.w + l], 2.0 * jcd[k * {nd} + l]);
}}"""
    if rys:
        head = (f"// Generated by gen_rys.py -- Rys class ({tag[0]}{tag[1]}|{tag[2]}{tag[3]}).  Do not edit.\n"
                f"// roots {M // 2 + 1}, contracted block: {nacc}, outputs: {nout}: a lane-split kernel, the lanes' primitive quartets by\n"
                f"// Rys quadrature with the 2-D tables in registers.\n"
                f'#include "../rys_common.cuh"')
        vrr_call = f"vrr_{tag}(Q.pairs, Q.rys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);"
        launch_head = f"""void launch_rys_{tag_of(X, Y)}(const EriQueue &Q0, const RysTab &R, int mixed, int grid, cudaStream_t s) {{
    EriQueue Q = Q0;
    Q.rys = R;"""
        occ_head = f"int occupancy_rys_{tag_of(X, Y)}(int mixed) {{"
    else:
        head = (f"// Generated by gen_eri.py -- class ({'spdfg'[la]}{'spdfg'[lb]}|{'spdfg'[lc]}{'spdfg'[ld]}).  Do not edit.\n"
                f"// VRR entries: {len(entries)}, contracted block: {nacc}, HRR lines: {len(hp.lines)}, outputs: {nout}.\n"
                f'#include "../eri_common.cuh"')
        vrr_call = (f"if (MIXED && bp.y * bq.y < Q.fp32_cut)\n"
                    f"                vrr_{tag}<float>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);\n"
                    f"            else vrr_{tag}<double>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);")
        launch_head = f"void launch_eri_{tag}(const EriQueue &Q, int mixed, int grid, cudaStream_t s) {{"
        occ_head = f"int occupancy_eri_{tag}(int mixed) {{"
    return f"""{head}

namespace molints {{

{vrr_fn}

// Bra and ket HRR of the contracted block (src/HGP.jl:92-114), then the component norms:
// the normalised (ab|cd) of bra pair p and ket pair q into res[{nout}] (ma, mb, mc, md
// row-major).
__device__ __forceinline__ void hrr_{tag}(const PairTab &P, int p, int q, const double *__restrict__ acc,
                                          double *__restrict__ res) {{
    const double4 gb = ldg4(&P.geo[p]);
    const double4 gk = ldg4(&P.geo[q]);
    const double ABx = gb.x, ABy = gb.y, ABz = gb.z;
    const double CDx = gk.x, CDy = gk.y, CDz = gk.z;
    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;
{hrr_code}
{out_code}
}}

{quartet_fn}

__device__ __forceinline__ void store_{tag}(double *__restrict__ out, const int4 ib_, const int4 ik_,
                                            bool same, const double *__restrict__ res) {{
    const bool dab = ib_.z == ib_.w, dcd = ik_.z == ik_.w;
    (void)dab; (void)dcd;
{ij_code}
{kl_code}
{store_code}
}}

{jk_fn}

// Persistent work-queue kernel: each warp takes chunks (one bra pair, a run of consecutive
// ket pairs of one molecule) from a shared counter until the chunk list, ordered by
// decreasing estimated cost, is exhausted.  A chunk's count field carries the split in bits
// 16+: lg = log2 S (bits 16-18) and lgj = log2 Sj (bits 20-22).  S lanes share each quartet:
// lane l takes ket pair q0 + l % (32/S) (+ 32/S per round); its group rank s = l / (32/S)
// takes every Sj-th ket primitive from s % Sj and every (S/Sj)-th bra primitive from s / Sj.
// The S partial blocks are summed by a fixed butterfly (the result depends on the split
// alone, not on the chunk), and the group's first lane runs the HRR and stores.  Heavy
// quartets are split so that no single lane's serial primitive loop sets the kernel time.
// JK: digest into J and K (molints_plan_jk) instead of storing the packed integrals; a separate
// instantiation, so that the store kernels carry none of the digestion code.
template <int MIXED, int JK>
__global__ void __launch_bounds__(128{bounds}) eri_queue_{tag}(const EriQueue Q) {{
    const int lane = threadIdx.x & 31;
    for (;;) {{
        int c = 0;
        if (lane == 0) c = atomicAdd(Q.counter, 1);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= Q.nchunks) return;
        const int4 ch = __ldg(&Q.chunks[c]);
        const int p = ch.x, cnt = ch.z & 0xffff, lg = (ch.z >> 16) & 7, lgj = (ch.z >> 20) & 7;
        const int W = 32 >> lg, kq = lane & (W - 1), s = lane >> (5 - lg);
        const int js = s & ((1 << lgj) - 1), is = s >> lgj;
        double jab[JK ? {na * nb} : 1];  // J/K digestion: the bra pair's J, over the chunk
        if constexpr (JK) {{
#pragma unroll
            for (int x = 0; x < {na * nb}; ++x) jab[x] = 0.0;
        }}
        for (int base = 0; base < cnt; base += W) {{
        const int q = ch.y + base + kq;
        const bool live = base + kq < cnt;
        double acc[{nacc}];
        double2 bp = make_double2(0.0, 0.0), bq = bp;
        if (live) {{
            bp = __ldg(&Q.pairs.bnd[p]);
            bq = __ldg(&Q.pairs.bnd[q]);
        }}
        if (!live || bp.x * bq.x < Q.screen_cut) {{
#pragma unroll
            for (int x = 0; x < {nacc}; ++x) acc[x] = 0.0;
        }} else {{
            const int nb = __ldg(&Q.pairs.info[p]).y, nk = __ldg(&Q.pairs.info[q]).y;
            {vrr_call}
        }}
        if (lg) {{
            for (int off = W; off < 32; off <<= 1) {{
#pragma unroll
                for (int x = 0; x < {nacc}; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
            }}
        }}
        const bool lead = live && s == 0;
        if (!JK && Q.scratch) {{
{scratch_store}
        }} else if (lead) {{
            double res[{nout}];
            hrr_{tag}(Q.pairs, p, q, acc, res);
            if constexpr (JK) {{
                const int4 ib_ = __ldg(&Q.pairs.info[p]), ik_ = __ldg(&Q.pairs.info[q]);
                jk_{tag}(Q.jk, ib_, ik_, jk_weight(ib_.z == ib_.w, ik_.z == ik_.w, p == q), res, jab);
            }} else {{
                store_{tag}(Q.out + __ldg(&Q.mol_out[ch.w]), __ldg(&Q.pairs.info[p]), __ldg(&Q.pairs.info[q]),
                            p == q, res);
            }}
        }}
        }}
        if constexpr (JK) {{
            // one addition per J_ab and chunk
            const int4 ib_ = __ldg(&Q.pairs.info[p]);
#pragma unroll
            for (int x = 0; x < {na * nb}; ++x) {{
                double v = jab[x];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == 0) atomicAdd(&Q.jk.J[(long long)(ib_.z + x / {nb}) * Q.jk.n + ib_.w + x % {nb}], 2.0 * v);
            }}
        }}
    }}
}}

{stage_fn}
{launch_head}
    if (Q.nchunks <= 0 || grid <= 0) return;
{stage_prep}
{mixed_dispatch}
}}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
{occ_head}
{occ_prep}
    int n = 0;
{occ_dispatch}
    return n;
}}
{schwarz}
}}  // namespace molints
"""


def emit_dispatch(pairs):
    """eri_dispatch.h: launch tables over all pair classes up to f (gen_rys.LMAX).  HGP kernels
    exist for the class pairs of shells up to d; Rys kernels for every class pair."""
    cls = gen_rys.pair_classes()
    hgp = set(pairs)
    lines = ["// Generated by gen_eri.py.  Do not edit.", "#pragma once",
             '#include "eri_common.cuh"', "namespace molints {"]
    for X, Y in pairs:
        t = tag_of(X, Y)
        lines.append(f"void launch_eri_{t}(const EriQueue &Q, int mixed, int grid, cudaStream_t s);")
        lines.append(f"int occupancy_eri_{t}(int mixed);")
        if X == Y and has_schwarz(X):
            lines.append(f"void launch_schwarz_{t}(const PairTab &P, const BoysTab &B, int p0, int np, "
                         f"double2 *pbound, const int *mol, unsigned long long *qmax, double *qout, int full, "
                         f"cudaStream_t s);")
    for X, Y in gen_rys.class_pairs():
        t = tag_of(X, Y)
        lines.append(f"void launch_rys_{t}(const EriQueue &Q, const RysTab &R, int mixed, int grid, cudaStream_t s);")
        lines.append(f"int occupancy_rys_{t}(int mixed);")
        if X == Y and not has_schwarz(X):
            lines.append(f"void launch_rys_bound_{t}(const PairTab &P, const RysTab &R, int p0, int np, "
                         f"double2 *pbound, const int *mol, unsigned long long *qmax, double *qout, int full, "
                         f"cudaStream_t s);")
    lines.append("typedef void (*EriLauncher)(const EriQueue &, int, int, cudaStream_t);")
    lines.append("typedef int (*EriOccupancy)(int);")
    lines.append("typedef void (*SchwarzLauncher)(const PairTab &, const BoysTab &, int, int, double2 *, "
                 "const int *, unsigned long long *, double *, int, cudaStream_t);")
    lines.append("typedef void (*RysLauncher)(const EriQueue &, const RysTab &, int, int, cudaStream_t);")
    lines.append("typedef int (*RysOccupancy)(int);")
    lines.append("typedef void (*RysBoundLauncher)(const PairTab &, const RysTab &, int, int, double2 *, "
                 "const int *, unsigned long long *, double *, int, cudaStream_t);")
    lines.append(f"constexpr int kLmax = {gen_rys.LMAX};      // shells up to f (Rys)")
    lines.append(f"constexpr int kLmaxHgp = {LMAX_ALL_HGP};   // every class pair up to d has an HGP kernel")
    lines.append(f"constexpr int kNumPairClasses = {len(cls)};")
    lines.append("// pair class c = (kPairClassLa[c], kPairClassLb[c]), ordered by la+lb then la")
    lines.append("constexpr int kPairClassLa[] = {" + ", ".join(str(c[0]) for c in cls) + "};")
    lines.append("constexpr int kPairClassLb[] = {" + ", ".join(str(c[1]) for c in cls) + "};")
    n = len(cls)

    def table(ctype, name, fmt, cond=lambda X, Y: True):
        lines.append(f"static const {ctype} {name}[{n}][{n}] = {{")
        for i, X in enumerate(cls):
            row = [fmt(X, Y) if (j <= i and cond(X, Y)) else "nullptr" for j, Y in enumerate(cls)]
            lines.append("    {" + ", ".join(row) + "},")
        lines.append("};")

    lines.append("// [x][y], x >= y (bra class x, ket class y); nullptr where no HGP kernel exists")
    table("EriLauncher", "kEriLaunchers", lambda X, Y: f"launch_eri_{tag_of(X, Y)}", lambda X, Y: (X, Y) in hgp)
    table("EriOccupancy", "kEriOccupancy", lambda X, Y: f"occupancy_eri_{tag_of(X, Y)}", lambda X, Y: (X, Y) in hgp)
    table("char *const", "kEriNames", lambda X, Y: f'"eri_{tag_of(X, Y)}"', lambda X, Y: (X, Y) in hgp)
    lines.append("// relative cost of one primitive quartet of the HGP kernel, 1 + VRR entries / 4 (the")
    lines.append("// (ss|ss) quartet ~ 1); sizes the lane split of heavy quartets; 0 where no HGP kernel")
    lines.append(f"static const float kEriPrimCost[{n}][{n}] = {{")
    for i, X in enumerate(cls):
        row = []
        for j, Y in enumerate(cls):
            if j <= i and (X, Y) in hgp:
                (la, lb), (lc, ld) = X, Y
                row.append(f"{1.0 + len(vrr_entries(la, la + lb, lc, lc + ld)) / 4.0!r}f")
            else:
                row.append("0.0f")
        lines.append("    {" + ", ".join(row) + "},")
    lines.append("};")
    lines.append("// the same of the Rys kernel where its queue is lane-split like an HGP kernel's (gen_rys.is_lane):")
    lines.append("// a root's two series cost about what twelve VRR entries do; 0 where a group computes whole quartets")
    lines.append(f"static const float kRysPrimCost[{n}][{n}] = {{")
    for i, X in enumerate(cls):
        row = []
        for j, Y in enumerate(cls):
            if j <= i and gen_rys.is_lane(X, Y):
                nr = (sum(X) + sum(Y)) // 2 + 1
                row.append(f"{1.0 + nr * (12 + gen_rys.class_tables(X, Y)['nblk']) / 4.0!r}f")
            else:
                row.append("0.0f")
        lines.append("    {" + ", ".join(row) + "},")
    lines.append("};")
    lines.append("// 1 where the class pair's kernel has an FP32 variant for MIXED quartets (HGP: at least")
    lines.append(f"// {MIXED_MIN_VRR} VRR entries; Rys: {gen_rys.MIXED_MIN_NBLK} to {gen_rys.MIXED_MAX_NBLK} block entries), else 0")
    for name, has in (("kEriHasFp32", lambda X, Y: (X, Y) in hgp and
                       len(vrr_entries(X[0], X[0] + X[1], Y[0], Y[0] + Y[1])) >= MIXED_MIN_VRR),
                      ("kRysHasFp32", lambda X, Y: gen_rys.class_tables(X, Y)["mixed"])):
        lines.append(f"static const unsigned char {name}[{n}][{n}] = {{")
        for i, X in enumerate(cls):
            lines.append("    {" + ", ".join("1" if (j <= i and has(X, Y)) else "0"
                                             for j, Y in enumerate(cls)) + "},")
        lines.append("};")
    table("RysLauncher", "kRysLaunchers", lambda X, Y: f"launch_rys_{tag_of(X, Y)}")
    table("RysOccupancy", "kRysOccupancy", lambda X, Y: f"occupancy_rys_{tag_of(X, Y)}")
    table("char *const", "kRysNames", lambda X, Y: f'"rys_{tag_of(X, Y)}"')
    lines.append(f"static const char *const kSchwarzNames[{n}] = {{")
    lines.append("    " + ", ".join(f'"schwarz_{tag_of(X, X)[:2]}"' for X in cls))
    lines.append("};")
    lines.append(f"static const SchwarzLauncher kSchwarzLaunchers[{n}] = {{")
    lines.append("    " + ", ".join(f"launch_schwarz_{tag_of(X, X)}" if has_schwarz(X) else "nullptr" for X in cls))
    lines.append("};")
    lines.append(f"static const RysBoundLauncher kRysBoundLaunchers[{n}] = {{")
    lines.append("    " + ", ".join("nullptr" if has_schwarz(X) else f"launch_rys_bound_{tag_of(X, X)}" for X in cls))
    lines.append("};")
    lines.append("}  // namespace molints")
    return "\n".join(lines) + "\n"


def emit_class_table(path: Path):
    """class_table.h: the default per-class-pair method table of MOLINTS_METHOD_AUTO, from the
    class tuner's result kept in data/class_table_<gpu>.json (the classes it found faster with
    Rys, those of them whose Rys kernel follows the Boys mode under AUTO, and those whose FP32 variant
    it found faster than FP64)."""
    import json
    d = json.loads(path.read_text())
    cls = gen_rys.pair_classes()
    lv = {"s": 0, "p": 1, "d": 2, "f": 3}

    def idx(t):
        return cls.index((lv[t[0]], lv[t[1]])), cls.index((lv[t[2]], lv[t[3]]))
    n = len(cls)
    tab = [[0] * n for _ in range(n)]
    for x in range(n):
        for y in range(x + 1):
            tab[x][y] = 1 | 4  # MOLINTS_METHOD_HGP | MOLINTS_CLASS_NO_FP32
    for t in d["rys"]:
        x, y = idx(t)
        tab[x][y] = 2 | (tab[x][y] & 4)
    for t in d["fp32"]:
        x, y = idx(t)
        tab[x][y] &= 3
    lines = [f"// Generated by gen_eri.py from data/{path.name}.  Do not edit.",
             "// Default MOLINTS_METHOD_AUTO table of contexts on the device named below:",
             f"// {d['source']}.",
             "// Entries: 1 HGP, 2 Rys, | 4 (MOLINTS_CLASS_NO_FP32) where MIXED runs the FP64 kernel.",
             "#pragma once", "#include <stdint.h>", "namespace molints {",
             f'constexpr const char *kTunedDevice = "{d["device"]}";',
             f"static const int32_t kTunedClassMethods[{n}][{n}] = {{"]
    for x in range(n):
        lines.append("    {" + ", ".join(str(v) for v in tab[x]) + "},")
    follow = {idx(t) for t in d["follow_boys"]}
    assert not any(gen_rys.is_lane(cls[x], cls[y]) for x, y in follow), "lane-split kernels do not read xmax"
    lines += ["};",
              "// 1 where an AUTO plan's Rys kernel follows the Boys mode as the HGP kernel of the class pair does",
              "// (RysTab::xmax = 30 in the reference mode): (dp|dp), (fp|pp) and (dd|dd) evaluate the exact function",
              "// in either mode, and so do the class pairs without an HGP kernel.  For nine polarised atoms with f",
              "// shells the two forms differ by up to 7.4e-12 in (dd|pp), 1.3e-12 in (dd|ps).",
              f"static const unsigned char kRysFollowsBoys[{n}][{n}] = {{"]
    for x in range(n):
        lines.append("    {" + ", ".join(str(int((x, y) in follow)) for y in range(n)) + "},")
    # work-queue schedule (molints_schedule: lane_cost, hgp_widen, rys_chunks, rys_max_width,
    # gather_blocks), the built-in values where the tuner's result has none
    sc = dict({"lane_cost": 80.0, "hgp_widen": 1, "rys_chunks": 4096, "rys_max_width": 8, "gather_blocks": 5},
              **d.get("schedule", {}))
    keys = ("lane_cost", "hgp_widen", "rys_chunks", "rys_max_width", "gather_blocks")
    lines += ["};",
              "// work-queue schedule: " + ", ".join(keys)
              + (f" ({d['schedule_source']})" if "schedule_source" in d else " (built-in values)"),
              f"static const double kTunedSchedule[{len(keys)}] = {{" +
              ", ".join(repr(float(sc[k])) for k in keys) + "};",
              "}  // namespace molints", ""]
    return "\n".join(lines)


def generate(out_dir: Path = OUT_DIR):
    out_dir.mkdir(parents=True, exist_ok=True)
    pairs = class_pairs()
    written = []
    for X, Y in pairs:
        p = out_dir / f"eri_{tag_of(X, Y)}.cu"
        src = emit_class_pair(X, Y)
        if not p.exists() or p.read_text() != src:
            p.write_text(src)
        written.append(p)
    written += gen_rys.generate(out_dir)
    d = HERE / "eri_dispatch.h"
    src = emit_dispatch(pairs)
    if not d.exists() or d.read_text() != src:
        d.write_text(src)
    t = HERE / "class_table.h"
    src = emit_class_table(HERE.parent / "data" / "class_table_b200.json")
    if not t.exists() or t.read_text() != src:
        t.write_text(src)
    return written


if __name__ == "__main__":
    files = generate()
    print(f"{len(files)} class-pair kernels in {OUT_DIR}", file=sys.stderr)
