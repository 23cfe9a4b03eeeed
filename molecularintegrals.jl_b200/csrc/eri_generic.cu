// eri_generic.cu -- the shell quartets with a g shell (l = 4): a thread block per tile of a contracted
// quartet's outputs, Rys quadrature with up to nine roots, any angular momentum up to (gg|gg).
//
// The generated class kernels cover every class pair up to (ff|ff).  The reference's tables stop
// at l = 4 (shell_indices, src/Basis.jl:269-279) and its Huzinaga driver, all_twoe_ints
// (src/ERI.jl:15-112), accepts such shells; this kernel is their drop-in.  It follows
// coulomb_rys (src/Rys.jl:46-83) per primitive quartet -- roots and weights at X = rho |PQ|^2,
// the 1-D integrals of Int1d/Recur (src/Rys.jl:86-125) and the binomial transfer of Shift
// (src/Rys.jl:128-135) -- with the contracted-function norms applied (the reference driver
// leaves them out), and the outputs accumulated over primitive quartets in FP64:
//
//   G(i, k) per axis and root, i <= la+lb, k <= lc+ld, from G(0,0) = 1 and
//     G(i+1, k) = C00 G(i, k) + i B10 G(i-1, k) + k B00 G(i, k-1)
//     G(i, k+1) = D00 G(i, k) + k B01 G(i, k-1) + i B00 G(i-1, k)
//   with u the root (t^2), B00 = u / 2(z+e), B10 = (1 - e u/(z+e)) / 2z,
//   B01 = (1 - z u/(z+e)) / 2e, C00 = PA + e (Q-P) u/(z+e), D00 = QC + z (P-Q) u/(z+e);
//   H(ia, ib, k) = sum_s C(ib, s) AB^(ib-s) G(ia+s, k)   (bra transfer, AB = A - B);
//   I(ia, ib, ic, id) = sum_t C(id, t) CD^(id-t) H(ia, ib, ic+t);
//   (ab|cd) += c_a c_b c_c c_d 2 pi^(5/2) / (z e sqrt(z+e)) exp(-ab/z AB^2 - cd/e CD^2)
//              sum_r W_r Ix Iy Iz.
//
// A thread block takes one unit -- a tile of up to kGenTile outputs of one quartet -- at a time
// from a queue.  The quartet's items (primitive quartet, root) are set up together, a thread each
// (node, weight, recurrence coefficients), then go through shared memory in batches: a thread per
// (item, axis) forms the columns of G in registers and transfers each to H; a thread per row of H
// transfers it to I(ia, ib, ic, id); last every thread adds the batch's I_x I_y I_z to its outputs'
// registers.  The transfers are paid once per 1-D entry ((gg|gg): 1875 per item) instead of once
// per output (50,625), and most quartets (up to 4096 outputs: (gd|gp), (gg|gs)) are one tile and build
// their tables once; a larger one builds them once a tile.  Bound by the latency of a unit's phases (46 us for a (gg|gg) tile alone
// on the device, half of it the FP64 divisions, exponentials and root series of the set-up).
// Measured on B200, two centres with an s, p, d, f and g shell each (70 functions, 874 quartets
// here): 0.185 ms, against 15.9 ms for a form that built G with one thread per axis and
// transferred per output; kernels of 128 registers and two blocks per SM 0.185, three blocks of 80
// registers (spilling) 0.34 against 0.31 ms with index tables instead of the register transfers.
#include <cuda_runtime.h>

#include "../../include/molints.h"
#include "eri_common.cuh"
#include "eri_generic.cuh"

namespace molints {

constexpr int kGenThreads = 256;
constexpr int kGenAcc = 16;                       // outputs per thread and tile
static_assert(kGenTile == kGenThreads * kGenAcc, "a tile is one register accumulator per thread and output");
constexpr int kGenL = 4;                          // highest shell angular momentum
constexpr int kGenE = 2 * kGenL;                  // la + lb
constexpr int kGenRysXmax = 100;
constexpr int kGenNcheb = 16;
constexpr int kGenItems = 96;                     // (primitive quartet, root) items set up at once, at most
// doubles of each of the two table regions (H and I): the 1-D tables of three (gg|gg) items
// (3 * 5^4 doubles each), more items of smaller quartets.  Two blocks per SM.
constexpr int kGenRegion = 5760;
constexpr int kGenBatch = 64;                     // items whose tables are built at once, at most
constexpr int kGenPar = 10;                       // per item: C00 x 3, D00 x 3, B00, B10, B01, weight
constexpr int kGenPairs = 225;                    // component pairs of a (gg) shell pair

// Cartesian components of l = 0..4 in the reference's shell_indices order, flat (35 entries):
// x | y << 4 | z << 8, those of shell l starting at c_gen_comp_off[l].
__constant__ unsigned short c_gen_comp[35] = {0x0, 0x1, 0x10, 0x100, 0x2, 0x11, 0x101, 0x20, 0x110, 0x200, 0x3, 0x12, 0x102, 0x21, 0x201, 0x111, 0x30, 0x120, 0x210, 0x300, 0x4, 0x13, 0x103, 0x22, 0x112, 0x202, 0x31, 0x121, 0x211, 0x301, 0x40, 0x130, 0x220, 0x310, 0x400};
// 1/sqrt((2I-1)!!(2J-1)!!(2K-1)!!) of each component
__constant__ double c_gen_norm[35] = {0x1.0000000000000p+0, 0x1.0000000000000p+0, 0x1.0000000000000p+0, 0x1.0000000000000p+0, 0x1.279a74590331dp-1, 0x1.0000000000000p+0, 0x1.0000000000000p+0, 0x1.279a74590331dp-1, 0x1.0000000000000p+0, 0x1.279a74590331dp-1, 0x1.08654a2d4f6dap-2, 0x1.279a74590331dp-1, 0x1.279a74590331dp-1, 0x1.279a74590331dp-1, 0x1.279a74590331dp-1, 0x1.0000000000000p+0, 0x1.08654a2d4f6dap-2, 0x1.279a74590331dp-1, 0x1.279a74590331dp-1, 0x1.08654a2d4f6dap-2, 0x1.8fba8a1bf6f97p-4, 0x1.08654a2d4f6dap-2, 0x1.08654a2d4f6dap-2, 0x1.5555555555555p-2, 0x1.279a74590331dp-1, 0x1.5555555555555p-2, 0x1.08654a2d4f6dap-2, 0x1.279a74590331dp-1, 0x1.279a74590331dp-1, 0x1.08654a2d4f6dap-2, 0x1.8fba8a1bf6f97p-4, 0x1.08654a2d4f6dap-2, 0x1.5555555555555p-2, 0x1.08654a2d4f6dap-2, 0x1.8fba8a1bf6f97p-4};
__constant__ int c_gen_comp_off[kGenL + 2] = {0, 1, 4, 10, 20, 35};

// Node u_r and weight W_r of the n-point Rys rule at X (the tables of rys_root<NR> in
// rys_common.cuh, n a run-time value).
__device__ __forceinline__ double gen_clenshaw(const double *__restrict__ c, double s) {
    double b1 = 0.0, b2 = 0.0;
    for (int k = kGenNcheb - 1; k >= 1; --k) {
        const double t = fma(2.0 * s, b1, __ldg(c + k) - b2);
        b2 = b1;
        b1 = t;
    }
    return fma(s, b1, __ldg(c) - b2);
}

__device__ void gen_root(const RysTab &R, int n, double X, int r, double &u, double &w) {
    if (X < (double)kGenRysXmax) {
        const int j = (int)X;
        const double s = 2.0 * (X - (double)j) - 1.0;
        const double *c = R.cheb + (size_t)kGenRysXmax * kGenNcheb * n * (n - 1) +
                          ((size_t)j * 2 * n + r) * kGenNcheb;
        u = gen_clenshaw(c, s);
        w = gen_clenshaw(c + (size_t)n * kGenNcheb, s);
    } else {
        const int o = n * (n - 1) / 2 + r;
        const double ox = 1.0 / X;
        u = __ldg(R.herm_x2 + o) * ox;
        w = __ldg(R.herm_w + o) * sqrt(ox);
    }
}

// Transfer of one 1-D column v[0 .. l0 + l1] (AB = the shells' distance on the axis): out[i *
// (l1 + 1) * stride + j * stride] for i <= l0, j <= l1, by v_(j+1)[i] = v_j[i + 1] + AB v_j[i].
__device__ __forceinline__ void gen_transfer(double *v, int l0, int l1, double AB, double *__restrict__ out,
                                             int stride) {
    const int si = (l1 + 1) * stride;
    for (int j = 0;; ++j) {
#pragma unroll
        for (int i = 0; i <= kGenL; ++i)
            if (i <= l0) out[i * si + j * stride] = v[i];
        if (j == l1) break;
#pragma unroll
        for (int i = 0; i < kGenE; ++i) v[i] = fma(AB, v[i], v[i + 1]);  // beyond l0 + l1 - j: unused
    }
}

__global__ void __launch_bounds__(kGenThreads, 2) eri_generic_kernel(const GenQuartets Gq) {
    extern __shared__ __align__(16) double gen_smem[];
    double *const tabI = gen_smem, *const tabH = gen_smem + kGenRegion;
    __shared__ double sPar[kGenItems][kGenPar];
    // per component pair of the bra and of the ket: offsets in the x, y and z tables (10 bits each,
    // the bra's and the ket's add up: IS <= 625), function-pair index (-1: a duplicate), norm
    __shared__ unsigned sOff[2][kGenPairs];
    __shared__ int sFn[2][kGenPairs];
    __shared__ double sNorm[2][kGenPairs];
    __shared__ int s_unit;
    const int tid = threadIdx.x;
    for (;;) {
        __syncthreads();  // the previous unit's readers are done
        if (tid == 0) s_unit = atomicAdd(Gq.counter, 1);
        __syncthreads();
        if (s_unit >= Gq.n) return;
        // the list is in reference order, where the shells of high l tend to come last in each
        // atom: taken from its end, the heavy quartets start first
        const long long qi = Gq.n - 1 - s_unit;
        const int4 q = __ldg(&Gq.quartet[qi]);
        const int2 mt = __ldg(&Gq.mol_tile[qi]);
        const int sh[4] = {q.x, q.y, q.z, q.w};
        int l[4], np[4], po[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            l[t] = __ldg(&Gq.L[sh[t]]);
            np[t] = __ldg(&Gq.nprim[sh[t]]);
            po[t] = __ldg(&Gq.poff[sh[t]]);
        }
        const int nc[4] = {(l[0] + 1) * (l[0] + 2) / 2, (l[1] + 1) * (l[1] + 2) / 2,
                           (l[2] + 1) * (l[2] + 2) / 2, (l[3] + 1) * (l[3] + 2) / 2};
        const int E = l[0] + l[1], F = l[2] + l[3], nr = (E + F) / 2 + 1;
        const int nab = nc[0] * nc[1], ncd = nc[2] * nc[3], nout = nab * ncd;
        const int F1 = F + 1, AB2 = (l[0] + 1) * (l[1] + 1), CD2 = (l[2] + 1) * (l[3] + 1);
        const int HS = AB2 * F1, IS = AB2 * CD2;
        const int t0 = mt.y * kGenTile, tn = min(kGenTile, nout - t0);
        const int nj = (tn + kGenThreads - 1) / kGenThreads;  // outputs of a thread
        // the unit's component-pair tables
        for (int w = tid; w < 2 * kGenPairs; w += kGenThreads) {
            const int side = w >= kGenPairs, x = w - side * kGenPairs;
            const int l0 = l[2 * side], l1 = l[2 * side + 1], n1 = nc[2 * side + 1];
            if (x < nc[2 * side] * n1) {
                const int i0 = x / n1, i1 = x - i0 * n1;
                const int c0 = c_gen_comp_off[l0] + i0, c1 = c_gen_comp_off[l1] + i1;
                const unsigned m0 = c_gen_comp[c0], m1 = c_gen_comp[c1];
                unsigned off = 0;
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    off |= ((((m0 >> (4 * k)) & 15) * (l1 + 1) + ((m1 >> (4 * k)) & 15)) * (side ? 1 : CD2)) << (10 * k);
                const int f0 = __ldg(&Gq.fn_off[sh[2 * side]]) + i0, f1 = __ldg(&Gq.fn_off[sh[2 * side + 1]]) + i1;
                sOff[side][x] = off;
                // same-shell pairs: the larger component first; nbf <= 46000, so the index fits
                sFn[side][x] = (sh[2 * side] == sh[2 * side + 1] && f0 < f1) ? -1 : (int)pair_index(f0, f1);
                sNorm[side][x] = c_gen_norm[c0] * c_gen_norm[c1];
            }
        }
        __syncthreads();
        // this thread's outputs: component pairs (bra | ket << 8) and table offsets
        unsigned off[kGenAcc];
        double acc[kGenAcc];
#pragma unroll
        for (int j = 0; j < kGenAcc; ++j) {
            acc[j] = 0.0;
            const int o = j * kGenThreads + tid;
            const int ab = o < tn ? (t0 + o) / ncd : 0, cd = o < tn ? t0 + o - ab * ncd : 0;
            off[j] = sOff[0][ab] + sOff[1][cd];
        }
        const unsigned nquart = gen_prim_count(np);
        const int per = kGenItems / nr;  // primitive quartets set up at once
        const int batch = min(kGenBatch, kGenRegion / (3 * IS));  // HS <= IS
        for (unsigned g0 = 0; g0 < nquart; g0 += per) {
            const int ng = (int)min((unsigned)per, nquart - g0) * nr;
            if (tid < ng) {
                // item: primitive quartet and root.  The previous items' readers (the H phase) are done:
                // a barrier follows every H phase.
                const int pq = tid / nr, r = tid - pq * nr;
                const GenPrims k4 = gen_prim(g0 + pq, np);
                const double a = __ldg(&Gq.expn[po[0] + k4.a]), b = __ldg(&Gq.expn[po[1] + k4.b]);
                const double c = __ldg(&Gq.expn[po[2] + k4.c]), d = __ldg(&Gq.expn[po[3] + k4.d]);
                const double z = a + b, e = c + d, ze = z + e;
                double ab2 = 0.0, cd2 = 0.0, pq2 = 0.0, PA[3], QC[3], QP[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const double A = __ldg(&Gq.xyz[3 * sh[0] + k]), B = __ldg(&Gq.xyz[3 * sh[1] + k]);
                    const double C = __ldg(&Gq.xyz[3 * sh[2] + k]), D = __ldg(&Gq.xyz[3 * sh[3] + k]);
                    const double P = (a * A + b * B) / z, Q = (c * C + d * D) / e;
                    ab2 += (A - B) * (A - B);
                    cd2 += (C - D) * (C - D);
                    PA[k] = P - A;
                    QC[k] = Q - C;
                    QP[k] = Q - P;
                    pq2 += (P - Q) * (P - Q);
                }
                const double coef = __ldg(&Gq.ncoef[po[0] + k4.a]) * __ldg(&Gq.ncoef[po[1] + k4.b]) *
                                    __ldg(&Gq.ncoef[po[2] + k4.c]) * __ldg(&Gq.ncoef[po[3] + k4.d]);
                const double pref = 2.0 * 17.493418327624862 /* pi^2.5 */ / (z * e * sqrt(ze)) *
                                    exp(-a * b / z * ab2 - c * d / e * cd2) * coef;
                double u, w;
                gen_root(Gq.rys, nr, z * e / ze * pq2, r, u, w);
                const double uze = u / ze;
                double *par = sPar[tid];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    par[k] = PA[k] + e * QP[k] * uze;
                    par[3 + k] = QC[k] - z * QP[k] * uze;
                }
                par[6] = 0.5 * uze;
                par[7] = (1.0 - e * uze) / (2.0 * z);
                par[8] = (1.0 - z * uze) / (2.0 * e);
                par[9] = pref * w;
            }
            for (int b0 = 0; b0 < ng; b0 += batch) {
                const int nb = min(batch, ng - b0);
                __syncthreads();  // the items are set up; the previous batch's readers of H are done
                // G of every (item, axis) column by column in registers (the x tables carry the
                // weight), each column transferred to H(ia, ib, k) as it is formed
                for (int ga = tid; ga < 3 * nb; ga += kGenThreads) {
                    const int it = ga / 3, ax = ga - 3 * it;
                    const double *par = sPar[b0 + it];
                    const double C00 = par[ax], D00 = par[3 + ax], B00 = par[6], B10 = par[7], B01 = par[8];
                    const double AB = __ldg(&Gq.xyz[3 * sh[0] + ax]) - __ldg(&Gq.xyz[3 * sh[1] + ax]);
                    double *__restrict__ h = tabH + ga * HS;
                    double cur[kGenE + 1], prev[kGenE + 1];
                    cur[0] = ax == 0 ? par[9] : 1.0;
                    cur[1] = C00 * cur[0];
                    prev[0] = prev[1] = 0.0;
#pragma unroll
                    for (int i = 1; i < kGenE; ++i) {
                        cur[i + 1] = i < E ? C00 * cur[i] + (double)i * B10 * cur[i - 1] : 0.0;
                        prev[i + 1] = 0.0;
                    }
                    for (int k = 0;; ++k) {
                        double v[kGenE + 1];
#pragma unroll
                        for (int i = 0; i <= kGenE; ++i) v[i] = cur[i];
                        gen_transfer(v, l[0], l[1], AB, h + k, F1);
                        if (k == F) break;
#pragma unroll
                        for (int i = 0; i <= kGenE; ++i) {
                            v[i] = D00 * cur[i] + (double)k * B01 * prev[i];
                            if (i > 0) v[i] += (double)i * B00 * cur[i - 1];
                        }
#pragma unroll
                        for (int i = 0; i <= kGenE; ++i) {
                            prev[i] = cur[i];
                            cur[i] = v[i];
                        }
                    }
                }
                __syncthreads();
                // ket transfer: I(ia, ib, ic, id) of every (item, axis, ia, ib)
                for (int w = tid; w < 3 * nb * AB2; w += kGenThreads) {
                    const int ax = (w / AB2) % 3;
                    const double CD = __ldg(&Gq.xyz[3 * sh[2] + ax]) - __ldg(&Gq.xyz[3 * sh[3] + ax]);
                    const double *__restrict__ h = tabH + w * F1;
                    double v[kGenE + 1];
#pragma unroll
                    for (int k = 0; k <= kGenE; ++k) v[k] = k <= F ? h[k] : 0.0;
                    gen_transfer(v, l[2], l[3], CD, tabI + w * CD2, 1);
                }
                __syncthreads();
                for (int it = 0; it < nb; ++it) {
                    const double *__restrict__ X = tabI + it * 3 * IS, *__restrict__ Y = X + IS, *__restrict__ Z = Y + IS;
#pragma unroll
                    for (int j = 0; j < kGenAcc; ++j) {
                        if (j >= nj) break;
                        const unsigned o = off[j];
                        acc[j] = fma(X[o & 1023u] * Y[(o >> 10) & 1023u], Z[o >> 20], acc[j]);
                    }
                }
            }
        }
        // the tile's unique integrals, normalised, at their iindex positions
        const bool same_pq = q.x == q.z && q.y == q.w;
        double *__restrict__ out = Gq.out + __ldg(&Gq.mol_out[mt.x]);
#pragma unroll
        for (int j = 0; j < kGenAcc; ++j) {
            const int o = j * kGenThreads + tid;
            if (o >= tn) break;
            const int ab = (t0 + o) / ncd, cd = t0 + o - ab * ncd;
            const int ij = sFn[0][ab], kl = sFn[1][cd];
            if (ij < 0 || kl < 0 || (same_pq && ij < kl)) continue;
            out[packed_index(ij, kl)] = acc[j] * (sNorm[0][ab] * sNorm[1][cd]);
        }
    }
}

constexpr int kGenSmem = 2 * kGenRegion * (int)sizeof(double);

void launch_eri_generic(const GenQuartets &G, int num_sms, cudaStream_t s) {
    if (G.n <= 0 || num_sms <= 0) return;
    // (above 48 KB: allowed per function and device; plain state of the function, no queue work)
    cudaFuncSetAttribute(eri_generic_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kGenSmem);
    const long long grid = G.n < 2LL * num_sms ? G.n : 2LL * num_sms;  // two resident blocks per SM
    eri_generic_kernel<<<(int)grid, kGenThreads, kGenSmem, s>>>(G);
}

}  // namespace molints
