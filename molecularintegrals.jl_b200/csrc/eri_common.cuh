// eri_common.cuh -- device data layout and shared device functions of the ERI engine.
//
// Layout in HBM (all arrays are owned by a plan, see molints.cu):
//   * shell pairs, canonical orientation (L_A >= L_B), sorted by pair class and then by
//     contraction length; structure of arrays:
//       info[p] = {first primitive pair, number of primitive pairs, first function of A,
//                  first function of B}                      (int4, 16 B)
//       geo[p]  = {A-B (x,y,z), unused}                    (double4, 32 B)
//       bnd[p]  = {Qabs_p, R_p}: bounds for screening and for FP32 quartets (double2)
//   * primitive pairs, 80 B each (5 x 16 B vector loads): PrimPair below;
//   * the Boys tables (T = 0..40 step 1/32), 32 bytes per order and point;
//   * the packed output vector, 0-based iindex order (src/Utils.jl:14-19).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace molints {

constexpr int kBoysRows = 1281;           // T_n = n/32, n = 0..1280 (T up to 40)
constexpr int kBoysTaylor = 7;            // Taylor terms about T_n; |T - T_n| <= 1/64
constexpr double kBoysStepInv = 32.0;
constexpr double kBoysStep = 0.03125;
constexpr double kBoysTableMax = 40.0;    // exact-mode switch to the asymptotic form
constexpr int kBoysMaxM1 = 16;            // tables exist for M = 0..15
// Two tables of 16-byte rows per M: {F_M(T_n), e^-T_n} and {F_{M+6}(T_n)/6!, F_{M+3}(T_n)/3!}
constexpr int kBoysHalf = 2 * kBoysRows;  // doubles of one of them
constexpr double kBoysReferenceSwitch = 30.0;  // farray's Tmax, src/Boys.jl:19

// Record of one primitive pair (a, b) of a canonical shell pair (A, B):
//   zeta = a + b
//   kab  = sqrt(2) pi^(5/4) c_a c_b exp(-a b |A-B|^2 / zeta) / zeta, with c_a, c_b the
//          fully normalised contraction coefficients (radial primitive norm x CGBF norm)
//   oo2z = 1 / (2 zeta)
//   P    = (a A + b B) / zeta (gaussian_product_center, src/OneInts.jl:78-83)
//   PA   = P - A
//   b    = sqrt(max |(ab|ab)|) of this primitive pair (its Schwarz bound; 0 before the plan's
//          bound pass)
// so that kab_bra * kab_ket / sqrt(zeta+eta) is the [00|00] prefactor of HGP eq. 12,
// 2 pi^(5/2) / (zeta eta sqrt(zeta+eta)) x exp(...) x coefficients.
struct PrimPair {
    double zeta, kab, px, py, pz, oo2z, pax, pay, paz, b;  // what (ss| needs comes first
};
static_assert(sizeof(PrimPair) == 80, "PrimPair is 5 x 16 bytes");

struct PairTab {
    const int4 *info;
    const double4 *geo;   // A - B (w unused)
    const PrimPair *pp;
    const double2 *bnd;   // x: Qabs_p = sum_k b_k, y: R_p = (1+|AB|)^lb sum_k w_k (kept prims)
};

struct BoysTab {
    const double *tab;     // [kBoysMaxM1][2][kBoysRows][2] (fill_boys_table)
    double t_switch;       // asymptotic form at T >= t_switch
};

// Rys quadrature tables (generated/rys_tables.cu): for n = 1..7 roots, Chebyshev series of
// the nodes u_i = t_i^2 and weights W_i on unit intervals of X < 100, and the Gauss-Hermite
// limits x_i = h_i^2 / X, W_i = g_i / sqrt(X) above.  The moments of the limits are the asymptotic
// family of the Boys function, so a kernel with xmax = 30 evaluates the reference mode
// (kRysFollowsBoys, class_table.h) and one with xmax = 100 the exact function.
struct RysTab {
    const double *cheb;     // [n][interval j < 100][2n functions][16 coefficients]
    const double *herm_x2;  // h_i^2 of the 2n-point Gauss-Hermite rule, n at n(n-1)/2
    const double *herm_w;   // g_i, same layout
    double xmax = 100.0;    // the group kernels take the limits from here on (at most 100)
};
int rys_tables(RysTab *t);  // device addresses on the current device; 0 on success

// Coulomb and exchange digestion (molints_plan_jk): J_pq = sum_rs D_rs (pq|rs) and
// K_pr = sum_qs D_qs (pq|rs), full n x n row-major: J = X + X^T, K = Y + Y^T with X, Y accumulated
// with FP64 atomics (jk_weight below).
struct JKOut {
    const double *D;   // symmetric density, n x n
    double *J, *K;     // X and Y, zeroed before the execute
    int n;
};

// The chunk queue of one class pair: chunk c = {bra pair, first ket pair, ket count |
// split << 16, molecule}.  HGP kernels and the lane-split Rys ones: split = lg | lgj << 4, S = 2^lg
// lanes share each quartet and lane l of the warp that takes the chunk computes its share of
// (bra | first + l % (32/S) + (32/S) i), the ket primitives split over 2^lgj lanes and the bra
// primitives over the rest (split 0: one lane per quartet).  Chunks of the Rys kernels with a group of
// threads per quartet have split 0.  Chunks never cross a bra pair, a
// molecule or, when bra and ket class coincide, the triangle q <= p.
struct EriQueue {
    PairTab pairs;
    BoysTab boys;
    RysTab rys;                   // lane-split Rys kernels
    JKOut jk;                     // jk.J != nullptr: digest into J and K instead of storing
    double *out;                  // packed outputs of all molecules (device)
    const long long *mol_out;     // offset of each molecule's packed vector in out
    const int4 *chunks;
    int nchunks;
    int *counter;                 // next chunk; zero at launch
    double screen_cut;            // Qabs_p Qabs_q below this: written as 0
    double fp32_cut;              // R_p R_q below this (MIXED kernels): FP32 VRR
    // two-phase output (scratch != nullptr): quartet (p, q0 + t) of chunk c (molecule m = its
    // w field) has slot u = chunk_slot[c] + t of its class pair's region for molecule m,
    // region[m * kRegionFields ..] = {offset, first bra, first ket, kets}: its whole block
    // (ma, mb, mc, md row-major) goes to scratch[offset + u * block size].  A gather pass
    // writes the packed vector from the scratch afterwards.
    double *scratch;
    const long long *chunk_slot;
    const long long *region;
};
constexpr int kRegionFields = 4;

__device__ __forceinline__ PrimPair load_pp(const PrimPair *__restrict__ base, int k) {
    const double2 *v = reinterpret_cast<const double2 *>(base + k);
    const double2 a = __ldg(v), b = __ldg(v + 1), c = __ldg(v + 2), d = __ldg(v + 3),
                  e = __ldg(v + 4);
    PrimPair r;
    r.zeta = a.x; r.kab = a.y; r.px = b.x; r.py = b.y; r.pz = c.x; r.oo2z = c.y;
    r.pax = d.x; r.pay = d.y; r.paz = e.x; r.b = e.y;
    return r;
}

// F_0..F_M at T: the farray structure of src/Boys.jl:19-27.
//   T <  t_switch: F_M by a 7-term Taylor expansion about the nearest table point,
//                  F_M(T_n - d) = sum_k c_k d^k, c_k = F_{M+k}(T_n)/k!, then e^-T = e^-T_n e^d and
//                  the downward recursion F_m = (2T F_{m+1} + e^-T) / (2m+1).  Of the c_k only c_0,
//                  c_3 and c_6 are read; the others follow by the same recursion at T_n (all terms
//                  positive, and what rounding it adds comes times d <= 1/64).  A warp's lanes read
//                  rows at random, so every 16 bytes of a row cost about eight passes of the L1
//                  data pipe, which was what bound the (ss|ss) and (ps|ss) kernels (78-83 % busy
//                  with all of c_0 .. c_7 read, in 80-byte rows; the FP64 pipe 40-54 %): over 1.17e9
//                  integrals on B200 (ss|ss) 930 -> 884 us, (ps|ps) 458 -> 409.
//   T >= t_switch: the asymptotic family F_m = (2m-1)!! / (2T)^m * sqrt(pi/T)/2, the values
//                  farray's Fm_asymp top order and e^-T-free recursion produce.
// The table index is rounded with the 1.5*2^52 trick: T*32 + 1.5*2^52 holds round(T*32) in
// its low mantissa bits, and subtracting the constant back gives T_n*32 exactly.
// The near part: T at most the tables' end.
template <int M>
__device__ __forceinline__ void boys_near(double T, const BoysTab &bt, double *F) {
    static_assert(M < kBoysMaxM1, "Boys order beyond the tables");
    constexpr double kMagic = 6755399441055744.0;  // 1.5 * 2^52
    const double t32 = fma(T, kBoysStepInv, kMagic);
    // (exponents near the ends of the double range can make T a NaN: the row stays in the table)
    const unsigned n = min((unsigned)__double2loint(t32), (unsigned)(kBoysRows - 1));
    const double tn = (t32 - kMagic) * kBoysStep, d = tn - T;
    const double2 *__restrict__ tab = reinterpret_cast<const double2 *>(bt.tab + (size_t)M * (2 * kBoysHalf)) + n;
    const double2 fe = __ldg(tab), c63 = __ldg(tab + kBoysRows);
    // c_k = T_n c_{k+1} 2(k+1)/(2(M+k)+1) + e^-T_n / (k! (2(M+k)+1))
    const double c5 = fma(tn * c63.x, 12.0 / (2 * M + 11), fe.y * (1.0 / (120.0 * (2 * M + 11))));
    const double c2 = fma(tn * c63.y, 6.0 / (2 * M + 5), fe.y * (1.0 / (2.0 * (2 * M + 5))));
    const double c4 = fma(tn * c5, 10.0 / (2 * M + 9), fe.y * (1.0 / (24.0 * (2 * M + 9))));
    const double c1 = fma(tn * c2, 4.0 / (2 * M + 3), fe.y * (1.0 / (2 * M + 3)));
    double f = fma(c63.x, d, c5);
    f = fma(f, d, c4);
    f = fma(f, d, c63.y);
    f = fma(f, d, c2);
    f = fma(f, d, c1);
    f = fma(f, d, fe.x);
    F[M] = f;
    if (M > 0) {
        // e^d for |d| <= 1/64 by its Taylor polynomial to d^6
        double ed = fma(d, 1.0 / 720, 1.0 / 120);
        ed = fma(ed, d, 1.0 / 24);
        ed = fma(ed, d, 1.0 / 6);
        ed = fma(ed, d, 0.5);
        ed = fma(ed, d, 1.0);
        ed = fma(ed, d, 1.0);
        const double emt = fe.y * ed;
        const double t2 = 2.0 * T;
#pragma unroll
        for (int m = M - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], emt) * (1.0 / (2 * m + 1));
    }
}

template <int M>
__device__ __forceinline__ void boys_fm(double T, const BoysTab &bt, double *F) {
    if (T < bt.t_switch) {
        boys_near<M>(T, bt, F);
    } else {
        const double r = rsqrt(T);
        F[0] = 0.88622692545275801365 * r;  // sqrt(pi)/2
        const double oo2t = 0.5 * r * r;
#pragma unroll
        for (int m = 1; m <= M; ++m) F[m] = F[m - 1] * ((2 * m - 1) * oo2t);
    }
}

// What the class kernels take: F_0..F_M at T below the switch; far (T at or above it) the asymptotic
// family times T^(m + 1/2), (2m-1)!! / 2^m * sqrt(pi)/2 (the caller's r and r2 carry the powers of T).
// (With the asymptotic branch of boys_fm, its own square root included, most warps ran both branches:
// over 1.17e9 integrals on B200 (ss|ss) 884 us against 833, (ps|ss) 1032 against 961.)
template <int M>
__device__ __forceinline__ void boys_scaled(bool far, double T, const BoysTab &bt, double *F) {
    if (!far) {
        boys_near<M>(T, bt, F);
    } else {
        F[0] = 0.88622692545275801365;  // sqrt(pi)/2
#pragma unroll
        for (int m = 1; m <= M; ++m) F[m] = F[m - 1] * (m - 0.5);
    }
}

__device__ __forceinline__ double4 ldg4(const double4 *p) {
    const double2 *v = reinterpret_cast<const double2 *>(p);
    const double2 a = __ldg(v), b = __ldg(v + 1);
    return make_double4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ long long tri_ll(long long i) { return i * (i + 1) / 2; }

// J/K digestion (the Fock-build contraction that make2JmK, src/ERI.jl:114-128, performs on the
// packed vector).  An integral (ab|cd) adds D_cd v to J_ab and D_bd v to K_ac, and the same for its
// other index permutations.  A shell quartet's whole block is digested, duplicates of same-shell
// pairs included, with the weight f = (distinct permutations of its shells) / 8:
//   J_ab += 2 f D_cd v, J_cd += 2 f D_ab v, K_ac += f D_bd v, K_ad += f D_bc v, K_bc += f D_ad v,
//   K_bd += f D_ac v
// into one orientation of each target, sums over the block first, so a quartet makes one addition
// per target (ab, cd, ac, ad, bc, bd) instead of six per integral; molints_plan_jk adds the
// transposes.  (Six additions per unique integral: 0.71 ms for 24 atoms of split valence, 3.5 ms
// for 15 polarised atoms on B200, most of it FP64 atomics.)
__device__ __forceinline__ double jk_weight(bool same_ab, bool same_cd, bool same_pq) {
    return (same_ab ? 0.5 : 1.0) * (same_cd ? 0.5 : 1.0) * (same_pq ? 0.5 : 1.0);
}

// 0-based packed index of the function-pair indices ij, kl (iindex, src/Utils.jl:19).
__device__ __forceinline__ long long packed_index(long long ij, long long kl) {
    return ij >= kl ? tri_ll(ij) + kl : tri_ll(kl) + ij;
}
__device__ __forceinline__ long long pair_index(int i, int j) {
    return i >= j ? tri_ll(i) + j : tri_ll(j) + i;
}

}  // namespace molints
