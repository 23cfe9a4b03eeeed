// rys_common.cuh -- device templates of the Rys class kernels (generated/rys_*.cu).
//
// One group of C::G threads (32 for most classes) evaluates C::W contracted shell quartets
// (ab|cd) of one bra pair at a time, W > 1 where the [e0|f0] block has few columns:
//   1. rys_contract: the primitive quartets in batches of C::PB per ket pair.  Stage 1, one thread
//      per (ket pair, primitive quartet, root): the Rys node u and weight W of that root, then the
//      three 2-D tables I(a, c), a <= E, c <= F (the x table carries the prefactor and W) into
//      shared memory.  Stage 2, one thread per (ket pair, block column): per primitive quartet and
//      root the column's 3 (E+1) table values in registers and all NA row accumulators of the
//      column, in FP64 registers.
//   2. HRR: the bra side in the column's thread (registers in, [r][column] of shared memory out),
//      the ket side one thread per row r, times the component norms, into shared memory; both
//      unrolled recurrences.
//   3. The quartets' outputs leave shared memory as one contiguous run (two-phase scratch), or to
//      their packed positions, or into J and K.
// These kernels have few primitive quartets per quartet (one to three), so the per-quartet work
// -- roots, tables, HRR -- is what counts: they are bound by the latency of these steps at 8 to 16
// warps per SM.  Measured on B200, eight molecules (1.17e9 integrals), against a form with a thread
// per block entry and the HRR's terms from tables: (dp|dp) 178 -> 59 us, (dd|dp) 180 -> 45,
// (dd|dd) 52 -> 13; an 11-atom molecule with f shells: (fd|dd) 74 -> 27, (ff|ff) 96 -> 25,
// (df|df) 43 -> 23.
// Recurrences: Rys, Dupuis and King's 2-D integrals in the Head-Gordon/Pople variables, with
// u = t^2 the root (see gen_rys.py); MolecularIntegrals.jl states the same method in
// src/Rys.jl:59-156.
#pragma once
#include <algorithm>
#include <type_traits>

#include "eri_common.cuh"

namespace molints {

constexpr int kRysXmax = 100;   // Chebyshev fits on [0, 100)
constexpr int kRysNcheb = 16;

// Class tables emitted by gen_rys.py.
struct RysClassTabs {
    const double *norm_ab;     // [NAB] component norms of a and b
    const uint16_t *col;       // [NC] column components cx | cy << 4 | cz << 8
};

// The HRR's closed form, by which gen_rys.class_tables states the transfer term by term, takes the
// monomials AB^(px,py,pz) in the order, packed px | py << 2 | pz << 4,
//   kRysMonoPow[kRysNmono] = {
//    0x00, 0x01, 0x04, 0x10, 0x02, 0x05, 0x11, 0x08, 0x14, 0x20,
//    0x03, 0x06, 0x12, 0x09, 0x15, 0x21, 0x0c, 0x18, 0x24, 0x30};
// The kernels run the recurrence (C::bra_hrr, C::ket_hrr); the tests compare the two.

// sum_k c_k T_k(s) for 16 coefficients by Clenshaw's recurrence.
__device__ __forceinline__ double clenshaw16(const double *__restrict__ c, double s) {
    const double2 *v = reinterpret_cast<const double2 *>(c);
    double2 q[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) q[k] = __ldg(v + k);
    const double s2 = 2.0 * s;
    double b1 = 0.0, b2 = 0.0;
#pragma unroll
    for (int k = 15; k >= 1; --k) {
        const double ck = (k & 1) ? q[k >> 1].y : q[k >> 1].x;
        const double t = fma(s2, b1, ck - b2);
        b2 = b1;
        b1 = t;
    }
    return fma(s, b1, q[0].x - b2);
}

// Node u_r = t_r^2 and weight W_r of the NR-point Rys rule at X >= 0: sum_r W_r u_r^m = F_m(X) for
// m < 2 NR, from X = xmax on the asymptotic form of F_m (Gauss-Hermite limit).  The kernels with a group
// of threads per quartet pass R.xmax; of the lane-split ones none follows the Boys mode.
template <int NR>
__device__ __forceinline__ void rys_root(const RysTab &R, double X, int r, double &u, double &w,
                                         double xmax = kRysXmax) {
    if (X < xmax) {
        const int j = (int)X;
        const double s = 2.0 * (X - (double)j) - 1.0;
        const double *c = R.cheb + (size_t)kRysXmax * kRysNcheb * NR * (NR - 1) +
                          ((size_t)j * 2 * NR + r) * kRysNcheb;
        u = clenshaw16(c, s);
        w = clenshaw16(c + NR * kRysNcheb, s);
    } else {
        const int o = NR * (NR - 1) / 2 + r;
        const double ox = 1.0 / X;
        u = __ldg(R.herm_x2 + o) * ox;
        w = __ldg(R.herm_w + o) * sqrt(ox);
    }
}

// Barrier over the G threads of group gid (named barrier gid+1 for 64-thread groups).
template <int G>
__device__ __forceinline__ void group_sync(int gid) {
    if constexpr (G == 32) {
        __syncwarp();
    } else if constexpr (G >= 128) {
        __syncthreads();
    } else {
        asm volatile("bar.sync %0, %1;" ::"r"(gid + 1), "r"(G) : "memory");
    }
}

template <int G>
__device__ __forceinline__ double group_max(double v, double *red, int gid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if constexpr (G == 32) {
        return v;
    } else {
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
        group_sync<G>(gid);
        double r = 0.0;
#pragma unroll
        for (int w = 0; w < G / 32; ++w) r = fmax(r, red[gid * (G / 32) + w]);
        group_sync<G>(gid);
        return r;
    }
}

// The three 2-D tables of root tr of one primitive quartet into tab (axis stride C::S).
template <class C, typename TT>
__device__ __forceinline__ void rys_tables_of(const RysTab &R, const PrimPair &bra, const PrimPair &ket, int tr,
                                              TT *__restrict__ tabs) {
    constexpr int S = C::S, F1 = C::F + 1, NR = C::NR, E = C::E, F = C::F;
    const double rz = rsqrt(bra.zeta + ket.zeta);
    const double r2 = rz * rz;
    const double PQv[3] = {bra.px - ket.px, bra.py - ket.py, bra.pz - ket.pz};
    const double X = bra.zeta * ket.zeta * r2 * (PQv[0] * PQv[0] + PQv[1] * PQv[1] + PQv[2] * PQv[2]);
    double u, w;
    rys_root<NR>(R, X, tr, u, w, R.xmax);
    const double ez = ket.zeta * r2, zz = bra.zeta * r2;
    const double PAv[3] = {bra.pax, bra.pay, bra.paz}, QCv[3] = {ket.pax, ket.pay, ket.paz};
    const double b10 = bra.oo2z * fma(-ez, u, 1.0);
    const double b01 = ket.oo2z * fma(-zz, u, 1.0);
    const double b00 = 0.5 * r2 * u;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const double c00 = fma(-ez * PQv[ax], u, PAv[ax]);
        const double d00 = fma(zz * PQv[ax], u, QCv[ax]);
        TT *tab = tabs + ax * S;
        // column c = 0 by the a-recurrence, then column c+1 from columns c and c-1
        double cur[E + 1], prev[E + 1];
        cur[0] = ax == 0 ? bra.kab * ket.kab * rz * w : 1.0;
        if (E > 0) cur[1] = c00 * cur[0];
#pragma unroll
        for (int a = 1; a < E; ++a) cur[a + 1] = fma(c00, cur[a], (double)a * b10 * cur[a - 1]);
#pragma unroll
        for (int a = 0; a <= E; ++a) {
            tab[a * F1] = (TT)cur[a];
            prev[a] = 0.0;
        }
#pragma unroll
        for (int c = 0; c < F; ++c) {
            double nxt[E + 1];
#pragma unroll
            for (int a = 0; a <= E; ++a) {
                double v = d00 * cur[a];
                if (c > 0) v = fma((double)c * b01, prev[a], v);
                if (a > 0) v = fma((double)a * b00, cur[a - 1], v);
                nxt[a] = v;
            }
#pragma unroll
            for (int a = 0; a <= E; ++a) {
                prev[a] = cur[a];
                cur[a] = nxt[a];
                tab[a * F1 + c + 1] = (TT)nxt[a];
            }
        }
    }
}

// A thread's parts in a round of W ket pairs: (w1, b1, r1) in stage 1, (w2, c2) in stage 2, there
// with every H-th (primitive quartet, root) from h; a thread without a part has w = W.
template <class C>
struct RysPart {
    int w1, b1, r1, w2, h, c2, cx, cy, cz;
    __device__ __forceinline__ RysPart(const RysClassTabs &T, int lane) {
        constexpr int NI = C::PB * C::NR;
        w1 = min(lane / NI, C::W);
        b1 = (lane - w1 * NI) / C::NR;
        r1 = lane - w1 * NI - b1 * C::NR;
        w2 = min(lane / (C::H * C::NC), C::W);
        h = w2 < C::W ? lane / C::NC - w2 * C::H : 0;
        c2 = w2 < C::W ? lane - (w2 * C::H + h) * C::NC : 0;
        const unsigned cp = __ldg(&T.col[c2]);
        cx = cp & 15u;
        cy = (cp >> 4) & 15u;
        cz = cp >> 8;
    }
};

// Primitive quartets of a quartet whose pairs keep nb and nk primitive pairs.  Unsigned: shells have up to
// 255 primitives, and 255^4 + 128 (a kernel's step) is below 2^32 where 216^4 is above 2^31.
__host__ __device__ __forceinline__ unsigned rys_prim_count(int nb, int nk) { return (unsigned)nb * (unsigned)nk; }

// Of a quartet of nq primitive quartets, those in the batch of pb that starts at g0.
__host__ __device__ __forceinline__ int rys_batch(unsigned nq, unsigned g0, int pb) {
    const unsigned left = nq - (nq < g0 ? nq : g0);
    return (int)(left < (unsigned)pb ? left : (unsigned)pb);
}

// One round's ket pairs as a thread sees them.
struct RysKets {
    int kx;              // stage 1: first ket primitive pair of w1
    unsigned nq1, nq2;   // primitive quartets of w1's and of w2's quartet (0: none, or no part)
    unsigned nqmax;      // the round's largest count, the same in every thread of the group
    bool f1, f2;    // MIXED: w1's / w2's quartet below the FP32 cutoff
};

// Stages 1 and 2: the contracted column c2 of w2's quartet into acc[NA].  All G threads of the
// group call it; it ends with a barrier (the tables in work are dead).  bx, nbp: the bra pair's
// first primitive pair and their count.  MIXED quartets below the FP32 cutoff: the 2-D tables are
// stored in FP32 and a batch's products are summed in FP32, then added to the FP64 accumulators
// (roots, weights and the recurrences stay FP64).
template <class C, int MIXED>
__device__ __forceinline__ void rys_contract(const PairTab &P, const RysTab &R, const RysPart<C> &L, int bx, int nbp,
                                             const RysKets &K, double *__restrict__ work, double *__restrict__ acc,
                                             int gid) {
    constexpr int S = C::S, F1 = C::F + 1, NR = C::NR, E = C::E, NA = C::NA, PB = C::PB, SI = C::SI;
#pragma unroll
    for (int a = 0; a < NA; ++a) acc[a] = 0.0;
    for (unsigned g0 = 0; g0 < K.nqmax; g0 += PB) {
        if (g0 + L.b1 < K.nq1) {
            const unsigned g = g0 + L.b1, gj = g / (unsigned)nbp;
            const PrimPair bra = load_pp(P.pp, bx + (int)(g - gj * nbp));
            const PrimPair ket = load_pp(P.pp, K.kx + (int)gj);
            double *tab = work + ((L.w1 * PB + L.b1) * NR + L.r1) * SI;
            if (MIXED && K.f1) rys_tables_of<C, float>(R, bra, ket, L.r1, reinterpret_cast<float *>(tab));
            else rys_tables_of<C, double>(R, bra, ket, L.r1, tab);
        }
        group_sync<C::G>(gid);
        const int ni = rys_batch(K.nq2, g0, PB) * NR;  // this quartet's (primitive quartet, root) items
        const double *__restrict__ t0 = work + L.w2 * PB * NR * SI;
        if (MIXED && K.f2) {
            float bacc[NA];
#pragma unroll
            for (int a = 0; a < NA; ++a) bacc[a] = 0.0f;
#pragma unroll 1
            for (int i = L.h; i < ni; i += C::H) {
                const float *__restrict__ t = reinterpret_cast<const float *>(t0 + i * SI);
                float x[E + 1], y[E + 1], z[E + 1];
#pragma unroll
                for (int a = 0; a <= E; ++a) {
                    x[a] = t[a * F1 + L.cx];
                    y[a] = t[S + a * F1 + L.cy];
                    z[a] = t[2 * S + a * F1 + L.cz];
                }
                C::col_update(x, y, z, bacc);
            }
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[a] += (double)bacc[a];
        } else {
#pragma unroll 1
            for (int i = L.h; i < ni; i += C::H) {
                const double *__restrict__ t = t0 + i * SI;
                double x[E + 1], y[E + 1], z[E + 1];
#pragma unroll
                for (int a = 0; a <= E; ++a) {
                    x[a] = t[a * F1 + L.cx];
                    y[a] = t[S + a * F1 + L.cy];
                    z[a] = t[2 * S + a * F1 + L.cz];
                }
                C::col_update(x, y, z, acc);
            }
        }
        group_sync<C::G>(gid);
    }
    if constexpr (C::H > 1) {  // a fixed butterfly over the column's H threads
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int bit = 1; bit < C::H; bit <<= 1) {
            const int from = L.w2 < C::W ? lane + ((L.h & bit) ? -bit : bit) * C::NC : lane;
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[a] += __shfl_sync(0xffffffffu, acc[a], from);
        }
    }
}

// HRR of the round's nlive quartets (ket pairs q0 ..) from the columns' accumulators to the
// normalised outputs (w, r, s) at the returned buffer's [(w NAB + r) NCDP + s].  Ends with a barrier.
template <class C>
__device__ __forceinline__ double *rys_hrr(const PairTab &P, const RysClassTabs &T, const RysPart<C> &L,
                                           const double *__restrict__ acc, const double4 gb, int q0, int nlive,
                                           double *__restrict__ work, int lane, int gid) {
    constexpr int NAB = C::NAB, NCP = C::NCP;
    double *__restrict__ mid = work, *__restrict__ stg = work + C::W * NAB * NCP;
    if (L.w2 < nlive && L.h == 0) C::bra_hrr(acc, gb.x, gb.y, gb.z, 1.0, mid + L.w2 * NAB * NCP + L.c2);
    group_sync<C::G>(gid);
    for (int row = lane; row < nlive * NAB; row += C::G) {
        const int w = row / NAB;
        const double4 gk = ldg4(&P.geo[q0 + w]);
        C::ket_hrr(mid + row * NCP, gk.x, gk.y, gk.z, __ldg(&T.norm_ab[row - w * NAB]), stg + row * C::NCDP);
    }
    group_sync<C::G>(gid);
    return stg;
}

// The round's quartets into J and K (jk_weight, eri_common.cuh): a thread per target (J_ab, J_cd,
// K_ac, K_ad, K_bc, K_bd) sums its terms of the block in shared memory and adds once.
template <class C>
__device__ __noinline__ void rys_digest(const JKOut jk, const int4 *__restrict__ info, const int4 ib, int p, int q0,
                                        int nlive, const double *__restrict__ stg, int lane) {
    constexpr int NB = C::NB, ND = C::ND, NA1 = C::NAB / NB, NC1 = C::NCD / ND;
    constexpr int T0 = C::NAB, T1 = T0 + C::NCD, T2 = T1 + NA1 * NC1, T3 = T2 + NA1 * ND, T4 = T3 + NB * NC1,
                  T5 = T4 + NB * ND;
    const double *__restrict__ D = jk.D;
    const long long n = jk.n;
    for (int t = lane; t < nlive * T5; t += C::G) {
        const int w = t / T5, k = t - w * T5;
        const int4 ik = __ldg(&info[q0 + w]);
        const double f = jk_weight(ib.z == ib.w, ik.z == ik.w, p == q0 + w);
        const double *__restrict__ v = stg + w * C::NAB * C::NCDP;  // v[(a NB + b) NCDP + c ND + d]
        double s = 0.0;
        if (k < T0) {
            const int a = k / NB, b = k - a * NB;
            for (int c = 0; c < NC1; ++c)
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    s = fma(__ldg(&D[(ik.z + c) * n + ik.w + d]), v[k * C::NCDP + c * ND + d], s);
            atomicAdd(&jk.J[(ib.z + a) * n + ib.w + b], 2.0 * f * s);
        } else if (k < T1) {
            const int x = k - T0, c = x / ND, d = x - c * ND;
            for (int a = 0; a < NA1; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    s = fma(__ldg(&D[(ib.z + a) * n + ib.w + b]), v[(a * NB + b) * C::NCDP + x], s);
            atomicAdd(&jk.J[(ik.z + c) * n + ik.w + d], 2.0 * f * s);
        } else if (k < T2) {
            const int x = k - T1, a = x / NC1, c = x - a * NC1;
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    s = fma(__ldg(&D[(ib.w + b) * n + ik.w + d]), v[(a * NB + b) * C::NCDP + c * ND + d], s);
            atomicAdd(&jk.K[(ib.z + a) * n + ik.z + c], f * s);
        } else if (k < T3) {
            const int x = k - T2, a = x / ND, d = x - a * ND;
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int c = 0; c < NC1; ++c)
                    s = fma(__ldg(&D[(ib.w + b) * n + ik.z + c]), v[(a * NB + b) * C::NCDP + c * ND + d], s);
            atomicAdd(&jk.K[(ib.z + a) * n + ik.w + d], f * s);
        } else if (k < T4) {
            const int x = k - T3, b = x / NC1, c = x - b * NC1;
            for (int a = 0; a < NA1; ++a)
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    s = fma(__ldg(&D[(ib.z + a) * n + ik.w + d]), v[(a * NB + b) * C::NCDP + c * ND + d], s);
            atomicAdd(&jk.K[(ib.w + b) * n + ik.z + c], f * s);
        } else {
            const int x = k - T4, b = x / ND, d = x - b * ND;
            for (int a = 0; a < NA1; ++a)
#pragma unroll
                for (int c = 0; c < NC1; ++c)
                    s = fma(__ldg(&D[(ib.z + a) * n + ik.z + c]), v[(a * NB + b) * C::NCDP + c * ND + d], s);
            atomicAdd(&jk.K[(ib.w + b) * n + ik.w + d], f * s);
        }
    }
}

// Persistent work-queue kernel body: each group takes chunks (one bra pair, a run of ket pairs
// of one molecule) from the class pair's counter and computes their quartets W at a time.
template <class C, int MIXED = 0>
__device__ __forceinline__ void rys_queue_body(const EriQueue &Q, const RysTab &R, const RysClassTabs &T) {
    extern __shared__ __align__(16) double rys_smem[];
    __shared__ int s_chunk[128 / C::G];
    constexpr int NAB = C::NAB, NCD = C::NCD, NOUT = NAB * NCD;
    const int gid = threadIdx.x / C::G, lane = threadIdx.x - gid * C::G;
    double *work = rys_smem + gid * C::SMEM_GROUP;
    const RysPart<C> L(T, lane);
    for (;;) {
        int c;
        if constexpr (C::G == 32) {
            c = lane == 0 ? atomicAdd(Q.counter, 1) : 0;
            c = __shfl_sync(0xffffffffu, c, 0);
        } else {
            if (lane == 0) s_chunk[gid] = atomicAdd(Q.counter, 1);
            group_sync<C::G>(gid);
            c = s_chunk[gid];
            group_sync<C::G>(gid);
        }
        if (c >= Q.nchunks) return;
        const int4 ch = __ldg(&Q.chunks[c]);
        const int p = ch.x;
        const int4 ib = __ldg(&Q.pairs.info[p]);
        const double2 bp = __ldg(&Q.pairs.bnd[p]);
        const double4 gb = ldg4(&Q.pairs.geo[p]);
        for (int base = 0; base < ch.z; base += C::W) {
            const int q0 = ch.y + base, nlive = min(C::W, ch.z - base);
            RysKets K{0, 0, 0, 0, false, false};
            // (one ket pair a round: every thread reads it, so that the count is the group's)
            if (C::W == 1 || L.w1 < nlive) {
                const int q = C::W == 1 ? q0 : q0 + L.w1;
                const int4 ik = __ldg(&Q.pairs.info[q]);
                const double2 bq = __ldg(&Q.pairs.bnd[q]);
                K.kx = ik.x;
                K.nq1 = (bp.x * bq.x < Q.screen_cut) ? 0 : rys_prim_count(ib.y, ik.y);  // screened: written as 0
                K.f1 = MIXED && bp.y * bq.y < Q.fp32_cut;
            }
            if constexpr (C::W == 1) {
                K.nqmax = K.nq1;
                K.nq2 = L.w2 == 0 ? K.nq1 : 0;
                K.f2 = K.f1;
                if (L.w1 != 0) K.nq1 = 0;
            } else {
                if (L.w2 < nlive) {
                    const int q = q0 + L.w2;
                    const int4 ik = __ldg(&Q.pairs.info[q]);
                    const double2 bq = __ldg(&Q.pairs.bnd[q]);
                    K.nq2 = (bp.x * bq.x < Q.screen_cut) ? 0 : rys_prim_count(ib.y, ik.y);
                    K.f2 = MIXED && bp.y * bq.y < Q.fp32_cut;
                }
                K.nqmax = __reduce_max_sync(0xffffffffu, K.nq1);
            }
            double acc[C::NA];
            rys_contract<C, MIXED>(Q.pairs, R, L, ib.x, ib.y, K, work, acc, gid);
            const double *__restrict__ stg = rys_hrr<C>(Q.pairs, T, L, acc, gb, q0, nlive, work, lane, gid);
            if (Q.scratch && !Q.jk.J) {
                // two-phase output: the quartets' whole blocks, (bra component, ket component)
                // row-major, in consecutive slots
                double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                    (__ldg(&Q.chunk_slot[c]) + base) * (long long)NOUT;
                for (int x = lane; x < nlive * NOUT; x += C::G) {
                    const int row = x / NCD;
                    dst[x] = stg[row * C::NCDP + (x - row * NCD)];
                }
            } else if (Q.jk.J) {
                rys_digest<C>(Q.jk, Q.pairs.info, ib, p, q0, nlive, stg, lane);
            } else {
                double *__restrict__ out = Q.out + __ldg(&Q.mol_out[ch.w]);
                const bool dab = ib.z == ib.w;
                for (int x = lane; x < nlive * NOUT; x += C::G) {
                    const int row = x / NCD, s = x - row * NCD, w = row / NAB, r = row - w * NAB;
                    const int4 ik = __ldg(&Q.pairs.info[q0 + w]);
                    const int ia = r / C::NB, jb = r - ia * C::NB, ic = s / C::ND, jd = s - ic * C::ND;
                    if ((dab && ia < jb) || (ik.z == ik.w && ic < jd)) continue;
                    const long long ij = pair_index(ib.z + ia, ib.w + jb), kl = pair_index(ik.z + ic, ik.w + jd);
                    if (p == q0 + w && ij < kl) continue;
                    out[packed_index(ij, kl)] = stg[row * C::NCDP + s];
                }
            }
            group_sync<C::G>(gid);
        }
    }
}

// Bounds of the pairs [p0, p0+np) of a pair class (bra class == ket class), one group per pair:
// full == 0: for every primitive pair k, from the diagonal primitive quartet,
//   pbound[k] = {sqrt(max |(a_k b_k|a_k b_k)|), sqrt(max |[e0|e0]_kk|)},
//   qmax[mol[p]]: the largest sum of the first over the molecule's pairs, as bits;
// full != 0: the contracted Q_p = sqrt(max |(ab|ab)|) into qout[p].
template <class C>
__device__ __forceinline__ void rys_bound_body(const PairTab &P, const RysTab &R, const RysClassTabs &T,
                                               int p0, int np, double2 *pbound, const int *mol,
                                               unsigned long long *qmax, double *qout, int full) {
    extern __shared__ __align__(16) double rys_smem[];
    __shared__ double s_red[4];
    constexpr int NG = 128 / C::G;
    const int gid = threadIdx.x / C::G, lane = threadIdx.x - gid * C::G;
    const int t = blockIdx.x * NG + gid;
    if (t >= np) return;
    double *work = rys_smem + gid * C::SMEM_GROUP;
    const RysPart<C> L(T, lane);
    const int p = p0 + t;
    const int4 in = __ldg(&P.info[p]);
    const double4 g = ldg4(&P.geo[p]);
    const int nk = full ? 1 : in.y;
    double q = 0.0;  // sum of b_k in list order
    for (int k = 0; k < nk; ++k) {
        const int i0 = full ? 0 : k, n = full ? in.y : 1;
        const unsigned nq = rys_prim_count(n, n);
        const RysKets K{in.x + i0, L.w1 == 0 ? nq : 0, L.w2 == 0 ? nq : 0, nq, false, false};
        double acc[C::NA];
        rys_contract<C, 0>(P, R, L, in.x + i0, n, K, work, acc, gid);
        double wmax = 0.0, m = 0.0;
#pragma unroll
        for (int a = 0; a < C::NA; ++a)
            if (L.w2 == 0 && a == L.c2) wmax = fabs(acc[a]);
        const double *__restrict__ stg = rys_hrr<C>(P, T, L, acc, g, p, 1, work, lane, gid);
        for (int r = lane; r < C::NAB; r += C::G) m = fmax(m, fabs(stg[r * C::NCDP + r]));
        m = group_max<C::G>(m, s_red, gid);
        wmax = group_max<C::G>(wmax, s_red, gid);
        if (lane == 0) {
            if (full) qout[p] = sqrt(m);
            else pbound[in.x + k] = make_double2(sqrt(m), sqrt(wmax));
        }
        q += sqrt(m);
        group_sync<C::G>(gid);
    }
    // the sums are >= 0, so their bit patterns order like the values
    if (!full && lane == 0) atomicMax(&qmax[__ldg(&mol[p])], (unsigned long long)__double_as_longlong(q));
}

}  // namespace molints
