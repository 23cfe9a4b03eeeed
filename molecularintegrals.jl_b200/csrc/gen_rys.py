"""Generate the Rys-quadrature class kernels (CUDA C for sm_100a).

This is the engine's counterpart of the reference's Rys driver (coulomb_rys and Int1d,
src/Rys.jl:27-156), reorganised for the GPU as Rys VRR + HGP HRR:

  * per primitive quartet and root t_r^2 = u_r of the NR = (e+f)/2 + 1 point Rys rule
    (nodes and weights from the tables of gen_rys_tables.py), the 2-D integrals
    I_x(a, c), I_y, I_z for a <= e = la+lb, c <= f = lc+ld by the Rys recurrences
        I(a+1, c) = C00 I(a, c) + a B10 I(a-1, c) + c B00 I(a, c-1)
        I(a, c+1) = D00 I(a, c) + c B01 I(a, c-1) + a B00 I(a-1, c)
    (C00 = PA + (W-P) u, D00 = QC + (W-Q) u, B10 = (1 - eta u/(zeta+eta)) / 2 zeta,
    B01 = (1 - zeta u/(zeta+eta)) / 2 eta, B00 = u / 2(zeta+eta)), the same recurrences as
    Recur (src/Rys.jl:86-120) written in u instead of t^2/(1-t^2);
  * the [e0|f0] block of the class (rows: the cartesian components of l = la..e, columns:
    l = lc..f) as sum_r W_r I_x I_y I_z, contracted over the primitive quartets in FP64;
  * the horizontal recurrence on the contracted block in closed form (the binomial
    transfer of Shift, src/Rys.jl:122-135, applied once per side after contraction):
        (a b| = sum_{k <= b} C(b_x,k_x) C(b_y,k_y) C(b_z,k_z) AB^(b-k) (a+k, 0|
    bra side first, then ket side;
  * component norms and the packed iindex store, as in the HGP kernels.

A group of G threads (32, 64 or 128; a block of 128 threads holds 128/G groups) takes W ket
pairs of one bra pair at a time (W > 1 where the block has few columns).  Stage 1 of a primitive
batch: one thread per (ket pair, primitive quartet, root) evaluates the root and builds the three
2-D tables into shared memory; stage 2: one thread per (ket pair, block column) loads the column's
table columns once per root and updates all row accumulators of the column in registers.  The bra
HRR then runs in that thread's registers, the ket HRR one thread per bra component pair on a row
in shared memory, both as unrolled recurrences (up to 351 steps, (ff|, without spills).

The class-specific code (column update, the two HRR sides) and data (column components, norms) are
emitted per class; the kernel body is the template in rys_common.cuh.  class_tables also states
the block's table offsets and the HRR in closed form, which the tests evaluate.
"""
from __future__ import annotations

import math
from pathlib import Path

HERE = Path(__file__).resolve().parent
OUT_DIR = HERE / "generated"
LMAX = 3             # shells up to f
NMONO = 20           # monomials AB^(px,py,pz), px+py+pz <= 3
# Classes of this many block entries get an FP32 variant for MIXED quartets (stage-2 products summed in
# FP32 per batch): all but the smallest and (ff|df), (ff|fd), (ff|ff).
MIXED_MIN_NBLK, MIXED_MAX_NBLK = 32, 3072


def shell_components(l):
    """src/Basis.jl:269-279 order (x-power descending, then y), l=3 with xzz before xyz."""
    comps = [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]
    if l == 3:
        comps[4], comps[5] = comps[5], comps[4]
    return comps


def ncart(l):
    return (l + 1) * (l + 2) // 2


# Mirrored pair classes (la < lb): a pair (f, d) whose d shell is the tighter one is computed
# as (d f|, so that the HRR moves angular momentum away from the tight shell (P near A); the
# other orientation loses up to 1e-11 Eh to cancellation.  (For lb <= 1 the loss stays at
# rounding level, and equal-L pairs are reoriented within their class.)
MIRRORED = [(2, 3)]


def pair_classes(lmax=LMAX):
    """Shell-pair classes (la, lb): la >= lb, plus MIRRORED; ordered by la+lb then la."""
    cls = [(la, lb) for la in range(lmax + 1) for lb in range(la + 1)]
    cls += [c for c in MIRRORED if max(c) <= lmax]
    return sorted(cls, key=lambda c: (c[0] + c[1], c[0]))


def class_pairs(lmax=LMAX):
    cls = pair_classes(lmax)
    return [(X, cls[j]) for i, X in enumerate(cls) for j in range(i + 1)]


def tag_of(X, Y):
    L = "spdfg"
    return f"{L[X[0]]}{L[X[1]]}{L[Y[0]]}{L[Y[1]]}"


MONOS = [(px, py, d - px - py) for d in range(4) for px in range(d, -1, -1) for py in range(d - px, -1, -1)]
MONO_INDEX = {m: i for i, m in enumerate(MONOS)}
assert len(MONOS) == NMONO


def dfact2(n):
    r = 1
    while n > 1:
        r *= n
        n -= 2
    return r


def comp_norm(c):
    return 1.0 / math.sqrt(dfact2(2 * c[0] - 1) * dfact2(2 * c[1] - 1) * dfact2(2 * c[2] - 1))


def block_components(l0, l1):
    """Components of the block rows (or columns): l = l0..l1, each shell in reference order."""
    out = []
    for l in range(l0, l1 + 1):
        out.extend(shell_components(l))
    return out


def hrr_terms(lx, ly, rows_index):
    """Closed-form HRR (a b| = sum_k C(b,k) AB^(b-k) (a+k, 0| for a in shell lx, b in shell ly.
    Returns per output r = ia * ncart(ly) + ib the list of (block index, monomial, binomial)."""
    out = []
    for a in shell_components(lx):
        for b in shell_components(ly):
            terms = []
            for kx in range(b[0] + 1):
                for ky in range(b[1] + 1):
                    for kz in range(b[2] + 1):
                        src = rows_index[(a[0] + kx, a[1] + ky, a[2] + kz)]
                        mono = MONO_INDEX[(b[0] - kx, b[1] - ky, b[2] - kz)]
                        binom = math.comb(b[0], kx) * math.comb(b[1], ky) * math.comb(b[2], kz)
                        terms.append((src, mono, binom))
            out.append(terms)
    return out


class HrrSide:
    """Unrolled horizontal recurrence of one side, (a b| = (a+1 b-1| + AB (a b-1| (src/HGP.jl:92-114):
    from the side's (a 0| entries in[] to every (a b|, a in shell lx, b in shell ly."""

    def __init__(self, lx, ly, index):
        self.index, self.lines, self.done = index, [], {}
        self.out = [self.term(a, b) for a in shell_components(lx) for b in shell_components(ly)]

    def term(self, a, b):
        if sum(b) == 0:
            return f"in[{self.index[a]}]"
        if (a, b) not in self.done:
            i = max(range(3), key=lambda t: (b[t], -t))
            bm = tuple(b[t] - (t == i) for t in range(3))
            ap = tuple(a[t] + (t == i) for t in range(3))
            hi, lo = self.term(ap, bm), self.term(a, bm)
            name = f"h{len(self.lines)}"
            self.lines.append(f"const double {name} = fma({'xyz'[i]}, {lo}, {hi});")
            self.done[(a, b)] = name
        return self.done[(a, b)]


def class_tables(X, Y):
    """Everything the kernel of class pair (X|Y) needs, as Python data."""
    (la, lb), (lc, ld) = X, Y
    e, f = la + lb, lc + ld
    nr = (e + f) // 2 + 1
    rows = block_components(la, e)
    cols = block_components(lc, f)
    rows_index = {c: i for i, c in enumerate(rows)}
    cols_index = {c: i for i, c in enumerate(cols)}
    S = (e + 1) * (f + 1)
    blk = []
    for a in rows:
        for c in cols:
            offs = [a[t] * (f + 1) + c[t] for t in range(3)]
            blk.append(offs)
    bra = hrr_terms(la, lb, rows_index)
    ket = hrr_terms(lc, ld, cols_index)
    norm_ab = [comp_norm(a) * comp_norm(b) for a in shell_components(la) for b in shell_components(lb)]
    norm_cd = [comp_norm(c) * comp_norm(d) for c in shell_components(lc) for d in shell_components(ld)]
    na, nc = len(rows), len(cols)
    nblk = na * nc
    nab, ncd = ncart(la) * ncart(lb), ncart(lc) * ncart(ld)
    # threads: a column of the block each
    G = 32 * ((nc + 31) // 32)
    G = 128 if G > 64 else G
    bra_lines, ket_lines = HrrSide(la, lb, rows_index), HrrSide(lc, ld, cols_index)
    # odd row strides: a warp reading a column of rows meets no bank twice
    ncp, ncdp = nc | 1, ncd | 1
    # ket pairs per group and round: as many as have columns and a root each, with their HRR
    # buffers in about 19 KB
    # (blocks of one or three columns: H threads share a column, each every H-th (quartet, root))
    H = {1: 8, 3: 2}.get(nc, 1)
    W = max(1, min(G // (nc * H), 32 // nr, 8)) if G == 32 else 1
    while W > 1 and W * nab * (ncp + ncdp) > 2400:
        W -= 1
    hrr_room = W * nab * (ncp + ncdp)
    # primitive quartets per ket pair and batch: one stage-1 thread per (ket pair, quartet, root);
    # the batch's 2-D tables (an odd stride per item) may use the HRR buffers' room
    si = (3 * S) | 1
    pb = max(1, min(G // (W * nr), max(hrr_room, 1536 * (G // 32)) // (W * nr * si)))
    npb = W * pb
    smem_group = max(npb * nr * si, hrr_room)
    mixed = MIXED_MIN_NBLK <= nblk <= MIXED_MAX_NBLK
    return dict(la=la, lb=lb, lc=lc, ld=ld, e=e, f=f, nr=nr, rows=rows, cols=cols, S=S, SI=si,
                blk=blk, bra=bra, ket=ket, norm_ab=norm_ab, norm_cd=norm_cd, na=na, nc=nc,
                nblk=nblk, nab=nab, ncd=ncd, ncp=ncp, ncdp=ncdp, G=G, W=W, H=H, pb=pb, npb=npb, nslot=1,
                acc=na, smem_group=smem_group, mixed=mixed, col=False,
                bra_side=bra_lines, ket_side=ket_lines)


def _arr(vals, fmt=str, per=12):
    vals = list(vals)
    lines = []
    for i in range(0, len(vals), per):
        lines.append("    " + ", ".join(fmt(v) for v in vals[i:i + per]) + ",")
    return "\n".join(lines) if lines else "    0,"


def is_lane(X, Y):
    """Class pairs of small blocks (below the FP32 variant's bound) run a lane-split kernel, the HGP
    kernel's frame with the lanes' primitive quartets by Rys quadrature: a group of threads per
    quartet leaves most of them idle (one to thirty block entries) and serialises long contractions.
    On B200, (ss|ss) of a 60-function molecule (300,949 primitive quartets): group form 342 us."""
    return class_tables(X, Y)["nblk"] < MIXED_MIN_NBLK


def emit_class_pair(X, Y):
    if is_lane(X, Y):
        import gen_eri
        return gen_eri.emit_class_pair(X, Y, rys=True)
    t = class_tables(X, Y)
    tag = tag_of(X, Y)
    smem_block = (128 // t["G"]) * t["smem_group"] * 8
    assert smem_block <= 227 * 1024, (tag, smem_block)
    import gen_eri
    diag = X == Y and not gen_eri.has_schwarz(X)
    bound_kernel = bound_launch = ""
    if diag:
        bound_kernel = f"""
__global__ void __launch_bounds__(128) rys_bound_kernel_{tag}(PairTab P, RysTab R, int p0, int np,
                                                              double2 *pbound, const int *mol,
                                                              unsigned long long *qmax, double *qout, int full) {{
    rys_bound_body<C_{tag}>(P, R, tabs_{tag}(), p0, np, pbound, mol, qmax, qout, full);
}}
"""
        bound_launch = f"""
void launch_rys_bound_{tag}(const PairTab &P, const RysTab &R, int p0, int np, double2 *pbound,
                            const int *mol, unsigned long long *qmax, double *qout, int full, cudaStream_t s) {{
    if (np <= 0) return;
    rys_prepare_{tag}();
    constexpr int ng = 128 / C_{tag}::G;
    rys_bound_kernel_{tag}<<<(np + ng - 1) / ng, 128, {smem_block}, s>>>(P, R, p0, np, pbound, mol, qmax, qout,
                                                                             full);
}}
"""
    if t["mixed"]:
        mixed_dispatch = (f"    if (mixed) rys_queue_{tag}<1><<<grid, 128, {smem_block}, s>>>(Q, R);\n"
                          f"    else rys_queue_{tag}<0><<<grid, 128, {smem_block}, s>>>(Q, R);")
        occ_dispatch = (f"    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_{tag}<1>, 128, {smem_block});\n"
                        f"    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_{tag}<0>, 128, {smem_block});")
    else:
        mixed_dispatch = (f"    (void)mixed;  // no FP32 variant for this class\n"
                          f"    rys_queue_{tag}<0><<<grid, 128, {smem_block}, s>>>(Q, R);")
        occ_dispatch = (f"    (void)mixed;\n"
                        f"    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_{tag}<0>, 128, {smem_block});")
    # stage 2: one block column's row accumulators from its three table columns
    col_code = ("    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns\n"
                "    template <typename T, typename A>\n"
                "    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {\n"
                + "\n".join(f"        acc[{ia}] = fma(x[{a[0]}] * y[{a[1]}], z[{a[2]}], acc[{ia}]);"
                            for ia, a in enumerate(t["rows"])) + "\n    }")
    colpow = ", ".join(str(c[0] | (c[1] << 4) | (c[2] << 8)) for c in t["cols"])
    col_tab = f"\n// column components cx | cy << 4 | cz << 8\n__device__ const uint16_t kCol_{tag}[{t['nc']}] = {{ {colpow} }};\n"

    def side_code(name, side, scale, stride):
        head = (f"    __device__ __forceinline__ static void {name}(const double *__restrict__ in, double x, double y, "
                f"double z, double nrm, double *__restrict__ out) {{\n")
        body = "".join(f"        {ln}\n" for ln in side.lines)
        outs = "".join(f"        out[{r * stride}] = {e}{scale(r)};\n" for r, e in enumerate(side.out))
        return head + "        (void)x; (void)y; (void)z; (void)nrm;\n" + body + outs + "    }"
    hrr_code = ("    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms\n" +
                side_code("bra_hrr", t["bra_side"], lambda r: "", t["ncp"]) + "\n" +
                side_code("ket_hrr", t["ket_side"], lambda r: f" * (nrm * {t['norm_cd'][r]!r})", 1))
    return f"""// Generated by gen_rys.py -- Rys class ({tag[0]}{tag[1]}|{tag[2]}{tag[3]}).  Do not edit.
// roots {t['nr']}, block {t['na']} x {t['nc']}, outputs {t['nab']} x {t['ncd']}, group {t['G']} threads, {t['W']} ket pairs a round,
// {t['pb']} primitive quartets per ket pair and batch, {smem_block} B shared per block.
#include "../rys_common.cuh"

namespace molints {{

struct C_{tag} {{
    static constexpr int LA = {t['la']}, LB = {t['lb']}, LC = {t['lc']}, LD = {t['ld']};
    static constexpr int E = {t['e']}, F = {t['f']}, NR = {t['nr']};
    static constexpr int NA = {t['na']}, NC = {t['nc']}, NBLK = {t['nblk']};
    static constexpr int NB = {ncart(t['lb'])}, ND = {ncart(t['ld'])};
    static constexpr int NAB = {t['nab']}, NCD = {t['ncd']};
    static constexpr int G = {t['G']}, W = {t['W']}, H = {t['H']}, PB = {t['pb']};
    static constexpr int S = {t['S']}, SI = {t['SI']}, NCP = {t['ncp']}, NCDP = {t['ncdp']};
    static constexpr int SMEM_GROUP = {t['smem_group']};
{col_code}
{hrr_code}
}};

__device__ const double kNormAB_{tag}[{len(t['norm_ab'])}] = {{
{_arr(t['norm_ab'], repr, 4)}
}};
{col_tab}
__device__ __forceinline__ RysClassTabs tabs_{tag}() {{
    return RysClassTabs{{kNormAB_{tag}, kCol_{tag}}};
}}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_{tag}(const EriQueue Q, const RysTab R) {{
    rys_queue_body<C_{tag}, MIXED>(Q, R, tabs_{tag}());
}}
{bound_kernel}
static void rys_prepare_{tag}() {{
    static bool done[64] = {{false}};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {{
        cudaFuncSetAttribute(rys_queue_{tag}<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, {smem_block});
{"        cudaFuncSetAttribute(rys_queue_" + tag + "<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, " + str(smem_block) + ");" if t["mixed"] else ""}
{"        cudaFuncSetAttribute(rys_bound_kernel_" + tag + ", cudaFuncAttributeMaxDynamicSharedMemorySize, " + str(smem_block) + ");" if diag else ""}
        done[dev] = true;
    }}
}}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_{tag}(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {{
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_{tag}();
    constexpr int ng = 128 / C_{tag}::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
{mixed_dispatch}
}}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_{tag}(int mixed) {{
    rys_prepare_{tag}();
    int n = 0;
{occ_dispatch}
    return n;
}}
{bound_launch}
}}  // namespace molints
"""


def generate(out_dir: Path = OUT_DIR):
    out_dir.mkdir(parents=True, exist_ok=True)
    written = []
    for X, Y in class_pairs():
        p = out_dir / f"rys_{tag_of(X, Y)}.cu"
        src = emit_class_pair(X, Y)
        if not p.exists() or p.read_text() != src:
            p.write_text(src)
        written.append(p)
    return written
