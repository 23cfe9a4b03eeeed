// Generated by gen_eri.py -- class (dd|ps).  Do not edit.
// VRR entries: 198, contracted block: 93, HRR lines: 237, outputs: 108.
#include "../eri_common.cuh"

namespace molints {

// The contracted [e0|f0] block of bra pair p and ket pair q into acc[93], summed over
// the bra primitive pairs i0, i0 + istep, ... < i1 and the ket primitive pairs j0, j0 + jstep,
// ... < j1 of the two shell pairs.  VT is the VRR arithmetic type (double, or float for MIXED).
// The ket loop is outside: a warp shares its bra pair, so the inner bra loads are broadcasts
// and each lane's ket record is loaded once.  Steps above 1 split one quartet's primitive
// quartets over the lanes of a split group (their blocks are summed before the HRR).
template <typename VT>
__device__ __forceinline__ void vrr_ddps(const PairTab &P, const BoysTab &B, int p, int q,
                                          int i0, int i1, int istep, int j0, int j1, int jstep,
                                          double *__restrict__ acc) {
    const int4 ib_ = __ldg(&P.info[p]);
    const int4 ik_ = __ldg(&P.info[q]);
#pragma unroll
    for (int x = 0; x < 93; ++x) acc[x] = 0.0;
    for (int j = j0; j < j1; j += jstep) {
        const PrimPair ket = load_pp(P.pp, ik_.x + j);
        for (int i = i0; i < i1; i += istep) {
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
            double F[6];
            boys_scaled<5>(far, ze * r2, B, F);
            const VT PAx = (VT)bra.pax, PAy = (VT)bra.pay, PAz = (VT)bra.paz;
            const VT QCx = (VT)ket.pax, QCy = (VT)ket.pay, QCz = (VT)ket.paz;
            const VT WPx = (VT)(-ez * PQx), WPy = (VT)(-ez * PQy), WPz = (VT)(-ez * PQz);
            const VT WQx = (VT)(zz * PQx), WQy = (VT)(zz * PQy), WQz = (VT)(zz * PQz);
            const VT oo2z = (VT)bra.oo2z, oo2e = (VT)ket.oo2z, oo2ze = (VT)(0.5 * r2);
            const VT rho_z = (VT)ez, rho_e = (VT)zz;
            (void)PAx; (void)PAy; (void)PAz; (void)QCx; (void)QCy; (void)QCz;
            (void)WPx; (void)WPy; (void)WPz; (void)WQx; (void)WQy; (void)WQz;
            (void)oo2z; (void)oo2e; (void)oo2ze; (void)rho_z; (void)rho_e;
            const VT v0_0_0 = (VT)(pref * F[0]);
            const VT v0_0_1 = (VT)(pref * F[1]);
            const VT v0_0_2 = (VT)(pref * F[2]);
            const VT v0_0_3 = (VT)(pref * F[3]);
            const VT v0_0_4 = (VT)(pref * F[4]);
            const VT v0_0_5 = (VT)(pref * F[5]);
            const VT v1_0_0 = PAx * v0_0_0 + WPx * v0_0_1;
            const VT v1_0_1 = PAx * v0_0_1 + WPx * v0_0_2;
            const VT v1_0_2 = PAx * v0_0_2 + WPx * v0_0_3;
            const VT v1_0_3 = PAx * v0_0_3 + WPx * v0_0_4;
            const VT v1_0_4 = PAx * v0_0_4 + WPx * v0_0_5;
            const VT v2_0_0 = PAy * v0_0_0 + WPy * v0_0_1;
            const VT v2_0_1 = PAy * v0_0_1 + WPy * v0_0_2;
            const VT v2_0_2 = PAy * v0_0_2 + WPy * v0_0_3;
            const VT v2_0_3 = PAy * v0_0_3 + WPy * v0_0_4;
            const VT v2_0_4 = PAy * v0_0_4 + WPy * v0_0_5;
            const VT v3_0_0 = PAz * v0_0_0 + WPz * v0_0_1;
            const VT v3_0_1 = PAz * v0_0_1 + WPz * v0_0_2;
            const VT v3_0_2 = PAz * v0_0_2 + WPz * v0_0_3;
            const VT v3_0_3 = PAz * v0_0_3 + WPz * v0_0_4;
            const VT v3_0_4 = PAz * v0_0_4 + WPz * v0_0_5;
            const VT v4_0_0 = PAx * v1_0_0 + WPx * v1_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v4_0_1 = PAx * v1_0_1 + WPx * v1_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v4_0_2 = PAx * v1_0_2 + WPx * v1_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v4_0_3 = PAx * v1_0_3 + WPx * v1_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v5_0_0 = PAx * v2_0_0 + WPx * v2_0_1;
            const VT v5_0_1 = PAx * v2_0_1 + WPx * v2_0_2;
            const VT v5_0_2 = PAx * v2_0_2 + WPx * v2_0_3;
            const VT v5_0_3 = PAx * v2_0_3 + WPx * v2_0_4;
            const VT v6_0_0 = PAx * v3_0_0 + WPx * v3_0_1;
            const VT v6_0_1 = PAx * v3_0_1 + WPx * v3_0_2;
            const VT v6_0_2 = PAx * v3_0_2 + WPx * v3_0_3;
            const VT v6_0_3 = PAx * v3_0_3 + WPx * v3_0_4;
            const VT v7_0_0 = PAy * v2_0_0 + WPy * v2_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v7_0_1 = PAy * v2_0_1 + WPy * v2_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v7_0_2 = PAy * v2_0_2 + WPy * v2_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v7_0_3 = PAy * v2_0_3 + WPy * v2_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v8_0_0 = PAy * v3_0_0 + WPy * v3_0_1;
            const VT v8_0_1 = PAy * v3_0_1 + WPy * v3_0_2;
            const VT v8_0_2 = PAy * v3_0_2 + WPy * v3_0_3;
            const VT v8_0_3 = PAy * v3_0_3 + WPy * v3_0_4;
            const VT v9_0_0 = PAz * v3_0_0 + WPz * v3_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v9_0_1 = PAz * v3_0_1 + WPz * v3_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v9_0_2 = PAz * v3_0_2 + WPz * v3_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v9_0_3 = PAz * v3_0_3 + WPz * v3_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v10_0_0 = PAx * v4_0_0 + WPx * v4_0_1 + (VT)2.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v10_0_1 = PAx * v4_0_1 + WPx * v4_0_2 + (VT)2.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v10_0_2 = PAx * v4_0_2 + WPx * v4_0_3 + (VT)2.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v11_0_0 = PAx * v5_0_0 + WPx * v5_0_1 + (VT)1.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v11_0_1 = PAx * v5_0_1 + WPx * v5_0_2 + (VT)1.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v11_0_2 = PAx * v5_0_2 + WPx * v5_0_3 + (VT)1.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v12_0_0 = PAx * v6_0_0 + WPx * v6_0_1 + (VT)1.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v12_0_1 = PAx * v6_0_1 + WPx * v6_0_2 + (VT)1.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v12_0_2 = PAx * v6_0_2 + WPx * v6_0_3 + (VT)1.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v13_0_0 = PAy * v5_0_0 + WPy * v5_0_1 + (VT)1.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v13_0_1 = PAy * v5_0_1 + WPy * v5_0_2 + (VT)1.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v13_0_2 = PAy * v5_0_2 + WPy * v5_0_3 + (VT)1.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v14_0_0 = PAz * v6_0_0 + WPz * v6_0_1 + (VT)1.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v14_0_1 = PAz * v6_0_1 + WPz * v6_0_2 + (VT)1.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v14_0_2 = PAz * v6_0_2 + WPz * v6_0_3 + (VT)1.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v15_0_0 = PAx * v8_0_0 + WPx * v8_0_1;
            const VT v15_0_1 = PAx * v8_0_1 + WPx * v8_0_2;
            const VT v15_0_2 = PAx * v8_0_2 + WPx * v8_0_3;
            const VT v16_0_0 = PAy * v7_0_0 + WPy * v7_0_1 + (VT)2.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v16_0_1 = PAy * v7_0_1 + WPy * v7_0_2 + (VT)2.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v16_0_2 = PAy * v7_0_2 + WPy * v7_0_3 + (VT)2.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v17_0_0 = PAy * v8_0_0 + WPy * v8_0_1 + (VT)1.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v17_0_1 = PAy * v8_0_1 + WPy * v8_0_2 + (VT)1.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v17_0_2 = PAy * v8_0_2 + WPy * v8_0_3 + (VT)1.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v18_0_0 = PAz * v8_0_0 + WPz * v8_0_1 + (VT)1.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v18_0_1 = PAz * v8_0_1 + WPz * v8_0_2 + (VT)1.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v18_0_2 = PAz * v8_0_2 + WPz * v8_0_3 + (VT)1.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v19_0_0 = PAz * v9_0_0 + WPz * v9_0_1 + (VT)2.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v19_0_1 = PAz * v9_0_1 + WPz * v9_0_2 + (VT)2.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v19_0_2 = PAz * v9_0_2 + WPz * v9_0_3 + (VT)2.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v20_0_0 = PAx * v10_0_0 + WPx * v10_0_1 + (VT)3.0 * oo2z * (v4_0_0 - rho_z * v4_0_1);
            const VT v20_0_1 = PAx * v10_0_1 + WPx * v10_0_2 + (VT)3.0 * oo2z * (v4_0_1 - rho_z * v4_0_2);
            const VT v21_0_0 = PAx * v11_0_0 + WPx * v11_0_1 + (VT)2.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v21_0_1 = PAx * v11_0_1 + WPx * v11_0_2 + (VT)2.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v22_0_0 = PAx * v12_0_0 + WPx * v12_0_1 + (VT)2.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v22_0_1 = PAx * v12_0_1 + WPx * v12_0_2 + (VT)2.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v23_0_0 = PAx * v13_0_0 + WPx * v13_0_1 + (VT)1.0 * oo2z * (v7_0_0 - rho_z * v7_0_1);
            const VT v23_0_1 = PAx * v13_0_1 + WPx * v13_0_2 + (VT)1.0 * oo2z * (v7_0_1 - rho_z * v7_0_2);
            const VT v24_0_0 = PAx * v15_0_0 + WPx * v15_0_1 + (VT)1.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v24_0_1 = PAx * v15_0_1 + WPx * v15_0_2 + (VT)1.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v25_0_0 = PAx * v14_0_0 + WPx * v14_0_1 + (VT)1.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v25_0_1 = PAx * v14_0_1 + WPx * v14_0_2 + (VT)1.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            const VT v26_0_0 = PAy * v13_0_0 + WPy * v13_0_1 + (VT)2.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v26_0_1 = PAy * v13_0_1 + WPy * v13_0_2 + (VT)2.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v27_0_0 = PAy * v15_0_0 + WPy * v15_0_1 + (VT)1.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v27_0_1 = PAy * v15_0_1 + WPy * v15_0_2 + (VT)1.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v28_0_0 = PAz * v15_0_0 + WPz * v15_0_1 + (VT)1.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v28_0_1 = PAz * v15_0_1 + WPz * v15_0_2 + (VT)1.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v29_0_0 = PAz * v14_0_0 + WPz * v14_0_1 + (VT)2.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v29_0_1 = PAz * v14_0_1 + WPz * v14_0_2 + (VT)2.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v30_0_0 = PAy * v16_0_0 + WPy * v16_0_1 + (VT)3.0 * oo2z * (v7_0_0 - rho_z * v7_0_1);
            const VT v30_0_1 = PAy * v16_0_1 + WPy * v16_0_2 + (VT)3.0 * oo2z * (v7_0_1 - rho_z * v7_0_2);
            const VT v31_0_0 = PAy * v17_0_0 + WPy * v17_0_1 + (VT)2.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v31_0_1 = PAy * v17_0_1 + WPy * v17_0_2 + (VT)2.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v32_0_0 = PAy * v18_0_0 + WPy * v18_0_1 + (VT)1.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v32_0_1 = PAy * v18_0_1 + WPy * v18_0_2 + (VT)1.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            const VT v33_0_0 = PAz * v18_0_0 + WPz * v18_0_1 + (VT)2.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v33_0_1 = PAz * v18_0_1 + WPz * v18_0_2 + (VT)2.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v34_0_0 = PAz * v19_0_0 + WPz * v19_0_1 + (VT)3.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v34_0_1 = PAz * v19_0_1 + WPz * v19_0_2 + (VT)3.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            if constexpr (sizeof(VT) == 8) {
                acc[0] = fma(QCx, v4_0_0, fma(WQx, v4_0_1, fma(2.0 * oo2ze, v1_0_1, acc[0])));
                acc[1] = fma(QCy, v4_0_0, fma(WQy, v4_0_1, acc[1]));
                acc[2] = fma(QCz, v4_0_0, fma(WQz, v4_0_1, acc[2]));
                acc[3] = fma(QCx, v5_0_0, fma(WQx, v5_0_1, fma(1.0 * oo2ze, v2_0_1, acc[3])));
                acc[4] = fma(QCy, v5_0_0, fma(WQy, v5_0_1, fma(1.0 * oo2ze, v1_0_1, acc[4])));
                acc[5] = fma(QCz, v5_0_0, fma(WQz, v5_0_1, acc[5]));
                acc[6] = fma(QCx, v6_0_0, fma(WQx, v6_0_1, fma(1.0 * oo2ze, v3_0_1, acc[6])));
                acc[7] = fma(QCy, v6_0_0, fma(WQy, v6_0_1, acc[7]));
                acc[8] = fma(QCz, v6_0_0, fma(WQz, v6_0_1, fma(1.0 * oo2ze, v1_0_1, acc[8])));
                acc[9] = fma(QCx, v7_0_0, fma(WQx, v7_0_1, acc[9]));
                acc[10] = fma(QCy, v7_0_0, fma(WQy, v7_0_1, fma(2.0 * oo2ze, v2_0_1, acc[10])));
                acc[11] = fma(QCz, v7_0_0, fma(WQz, v7_0_1, acc[11]));
                acc[12] = fma(QCx, v8_0_0, fma(WQx, v8_0_1, acc[12]));
                acc[13] = fma(QCy, v8_0_0, fma(WQy, v8_0_1, fma(1.0 * oo2ze, v3_0_1, acc[13])));
                acc[14] = fma(QCz, v8_0_0, fma(WQz, v8_0_1, fma(1.0 * oo2ze, v2_0_1, acc[14])));
                acc[15] = fma(QCx, v9_0_0, fma(WQx, v9_0_1, acc[15]));
                acc[16] = fma(QCy, v9_0_0, fma(WQy, v9_0_1, acc[16]));
                acc[17] = fma(QCz, v9_0_0, fma(WQz, v9_0_1, fma(2.0 * oo2ze, v3_0_1, acc[17])));
                acc[18] = fma(QCx, v10_0_0, fma(WQx, v10_0_1, fma(3.0 * oo2ze, v4_0_1, acc[18])));
                acc[19] = fma(QCy, v10_0_0, fma(WQy, v10_0_1, acc[19]));
                acc[20] = fma(QCz, v10_0_0, fma(WQz, v10_0_1, acc[20]));
                acc[21] = fma(QCx, v11_0_0, fma(WQx, v11_0_1, fma(2.0 * oo2ze, v5_0_1, acc[21])));
                acc[22] = fma(QCy, v11_0_0, fma(WQy, v11_0_1, fma(1.0 * oo2ze, v4_0_1, acc[22])));
                acc[23] = fma(QCz, v11_0_0, fma(WQz, v11_0_1, acc[23]));
                acc[24] = fma(QCx, v12_0_0, fma(WQx, v12_0_1, fma(2.0 * oo2ze, v6_0_1, acc[24])));
                acc[25] = fma(QCy, v12_0_0, fma(WQy, v12_0_1, acc[25]));
                acc[26] = fma(QCz, v12_0_0, fma(WQz, v12_0_1, fma(1.0 * oo2ze, v4_0_1, acc[26])));
                acc[27] = fma(QCx, v13_0_0, fma(WQx, v13_0_1, fma(1.0 * oo2ze, v7_0_1, acc[27])));
                acc[28] = fma(QCy, v13_0_0, fma(WQy, v13_0_1, fma(2.0 * oo2ze, v5_0_1, acc[28])));
                acc[29] = fma(QCz, v13_0_0, fma(WQz, v13_0_1, acc[29]));
                acc[30] = fma(QCx, v14_0_0, fma(WQx, v14_0_1, fma(1.0 * oo2ze, v9_0_1, acc[30])));
                acc[31] = fma(QCy, v14_0_0, fma(WQy, v14_0_1, acc[31]));
                acc[32] = fma(QCz, v14_0_0, fma(WQz, v14_0_1, fma(2.0 * oo2ze, v6_0_1, acc[32])));
                acc[33] = fma(QCx, v15_0_0, fma(WQx, v15_0_1, fma(1.0 * oo2ze, v8_0_1, acc[33])));
                acc[34] = fma(QCy, v15_0_0, fma(WQy, v15_0_1, fma(1.0 * oo2ze, v6_0_1, acc[34])));
                acc[35] = fma(QCz, v15_0_0, fma(WQz, v15_0_1, fma(1.0 * oo2ze, v5_0_1, acc[35])));
                acc[36] = fma(QCx, v16_0_0, fma(WQx, v16_0_1, acc[36]));
                acc[37] = fma(QCy, v16_0_0, fma(WQy, v16_0_1, fma(3.0 * oo2ze, v7_0_1, acc[37])));
                acc[38] = fma(QCz, v16_0_0, fma(WQz, v16_0_1, acc[38]));
                acc[39] = fma(QCx, v17_0_0, fma(WQx, v17_0_1, acc[39]));
                acc[40] = fma(QCy, v17_0_0, fma(WQy, v17_0_1, fma(2.0 * oo2ze, v8_0_1, acc[40])));
                acc[41] = fma(QCz, v17_0_0, fma(WQz, v17_0_1, fma(1.0 * oo2ze, v7_0_1, acc[41])));
                acc[42] = fma(QCx, v18_0_0, fma(WQx, v18_0_1, acc[42]));
                acc[43] = fma(QCy, v18_0_0, fma(WQy, v18_0_1, fma(1.0 * oo2ze, v9_0_1, acc[43])));
                acc[44] = fma(QCz, v18_0_0, fma(WQz, v18_0_1, fma(2.0 * oo2ze, v8_0_1, acc[44])));
                acc[45] = fma(QCx, v19_0_0, fma(WQx, v19_0_1, acc[45]));
                acc[46] = fma(QCy, v19_0_0, fma(WQy, v19_0_1, acc[46]));
                acc[47] = fma(QCz, v19_0_0, fma(WQz, v19_0_1, fma(3.0 * oo2ze, v9_0_1, acc[47])));
                acc[48] = fma(QCx, v20_0_0, fma(WQx, v20_0_1, fma(4.0 * oo2ze, v10_0_1, acc[48])));
                acc[49] = fma(QCy, v20_0_0, fma(WQy, v20_0_1, acc[49]));
                acc[50] = fma(QCz, v20_0_0, fma(WQz, v20_0_1, acc[50]));
                acc[51] = fma(QCx, v21_0_0, fma(WQx, v21_0_1, fma(3.0 * oo2ze, v11_0_1, acc[51])));
                acc[52] = fma(QCy, v21_0_0, fma(WQy, v21_0_1, fma(1.0 * oo2ze, v10_0_1, acc[52])));
                acc[53] = fma(QCz, v21_0_0, fma(WQz, v21_0_1, acc[53]));
                acc[54] = fma(QCx, v22_0_0, fma(WQx, v22_0_1, fma(3.0 * oo2ze, v12_0_1, acc[54])));
                acc[55] = fma(QCy, v22_0_0, fma(WQy, v22_0_1, acc[55]));
                acc[56] = fma(QCz, v22_0_0, fma(WQz, v22_0_1, fma(1.0 * oo2ze, v10_0_1, acc[56])));
                acc[57] = fma(QCx, v23_0_0, fma(WQx, v23_0_1, fma(2.0 * oo2ze, v13_0_1, acc[57])));
                acc[58] = fma(QCy, v23_0_0, fma(WQy, v23_0_1, fma(2.0 * oo2ze, v11_0_1, acc[58])));
                acc[59] = fma(QCz, v23_0_0, fma(WQz, v23_0_1, acc[59]));
                acc[60] = fma(QCx, v24_0_0, fma(WQx, v24_0_1, fma(2.0 * oo2ze, v15_0_1, acc[60])));
                acc[61] = fma(QCy, v24_0_0, fma(WQy, v24_0_1, fma(1.0 * oo2ze, v12_0_1, acc[61])));
                acc[62] = fma(QCz, v24_0_0, fma(WQz, v24_0_1, fma(1.0 * oo2ze, v11_0_1, acc[62])));
                acc[63] = fma(QCx, v25_0_0, fma(WQx, v25_0_1, fma(2.0 * oo2ze, v14_0_1, acc[63])));
                acc[64] = fma(QCy, v25_0_0, fma(WQy, v25_0_1, acc[64]));
                acc[65] = fma(QCz, v25_0_0, fma(WQz, v25_0_1, fma(2.0 * oo2ze, v12_0_1, acc[65])));
                acc[66] = fma(QCx, v26_0_0, fma(WQx, v26_0_1, fma(1.0 * oo2ze, v16_0_1, acc[66])));
                acc[67] = fma(QCy, v26_0_0, fma(WQy, v26_0_1, fma(3.0 * oo2ze, v13_0_1, acc[67])));
                acc[68] = fma(QCz, v26_0_0, fma(WQz, v26_0_1, acc[68]));
                acc[69] = fma(QCx, v27_0_0, fma(WQx, v27_0_1, fma(1.0 * oo2ze, v17_0_1, acc[69])));
                acc[70] = fma(QCy, v27_0_0, fma(WQy, v27_0_1, fma(2.0 * oo2ze, v15_0_1, acc[70])));
                acc[71] = fma(QCz, v27_0_0, fma(WQz, v27_0_1, fma(1.0 * oo2ze, v13_0_1, acc[71])));
                acc[72] = fma(QCx, v28_0_0, fma(WQx, v28_0_1, fma(1.0 * oo2ze, v18_0_1, acc[72])));
                acc[73] = fma(QCy, v28_0_0, fma(WQy, v28_0_1, fma(1.0 * oo2ze, v14_0_1, acc[73])));
                acc[74] = fma(QCz, v28_0_0, fma(WQz, v28_0_1, fma(2.0 * oo2ze, v15_0_1, acc[74])));
                acc[75] = fma(QCx, v29_0_0, fma(WQx, v29_0_1, fma(1.0 * oo2ze, v19_0_1, acc[75])));
                acc[76] = fma(QCy, v29_0_0, fma(WQy, v29_0_1, acc[76]));
                acc[77] = fma(QCz, v29_0_0, fma(WQz, v29_0_1, fma(3.0 * oo2ze, v14_0_1, acc[77])));
                acc[78] = fma(QCx, v30_0_0, fma(WQx, v30_0_1, acc[78]));
                acc[79] = fma(QCy, v30_0_0, fma(WQy, v30_0_1, fma(4.0 * oo2ze, v16_0_1, acc[79])));
                acc[80] = fma(QCz, v30_0_0, fma(WQz, v30_0_1, acc[80]));
                acc[81] = fma(QCx, v31_0_0, fma(WQx, v31_0_1, acc[81]));
                acc[82] = fma(QCy, v31_0_0, fma(WQy, v31_0_1, fma(3.0 * oo2ze, v17_0_1, acc[82])));
                acc[83] = fma(QCz, v31_0_0, fma(WQz, v31_0_1, fma(1.0 * oo2ze, v16_0_1, acc[83])));
                acc[84] = fma(QCx, v32_0_0, fma(WQx, v32_0_1, acc[84]));
                acc[85] = fma(QCy, v32_0_0, fma(WQy, v32_0_1, fma(2.0 * oo2ze, v18_0_1, acc[85])));
                acc[86] = fma(QCz, v32_0_0, fma(WQz, v32_0_1, fma(2.0 * oo2ze, v17_0_1, acc[86])));
                acc[87] = fma(QCx, v33_0_0, fma(WQx, v33_0_1, acc[87]));
                acc[88] = fma(QCy, v33_0_0, fma(WQy, v33_0_1, fma(1.0 * oo2ze, v19_0_1, acc[88])));
                acc[89] = fma(QCz, v33_0_0, fma(WQz, v33_0_1, fma(3.0 * oo2ze, v18_0_1, acc[89])));
                acc[90] = fma(QCx, v34_0_0, fma(WQx, v34_0_1, acc[90]));
                acc[91] = fma(QCy, v34_0_0, fma(WQy, v34_0_1, acc[91]));
                acc[92] = fma(QCz, v34_0_0, fma(WQz, v34_0_1, fma(4.0 * oo2ze, v19_0_1, acc[92])));
            } else {
                const VT v4_1_0 = QCx * v4_0_0 + WQx * v4_0_1 + (VT)2.0 * oo2ze * v1_0_1;
                acc[0] += (double)v4_1_0;
                const VT v4_2_0 = QCy * v4_0_0 + WQy * v4_0_1;
                acc[1] += (double)v4_2_0;
                const VT v4_3_0 = QCz * v4_0_0 + WQz * v4_0_1;
                acc[2] += (double)v4_3_0;
                const VT v5_1_0 = QCx * v5_0_0 + WQx * v5_0_1 + (VT)1.0 * oo2ze * v2_0_1;
                acc[3] += (double)v5_1_0;
                const VT v5_2_0 = QCy * v5_0_0 + WQy * v5_0_1 + (VT)1.0 * oo2ze * v1_0_1;
                acc[4] += (double)v5_2_0;
                const VT v5_3_0 = QCz * v5_0_0 + WQz * v5_0_1;
                acc[5] += (double)v5_3_0;
                const VT v6_1_0 = QCx * v6_0_0 + WQx * v6_0_1 + (VT)1.0 * oo2ze * v3_0_1;
                acc[6] += (double)v6_1_0;
                const VT v6_2_0 = QCy * v6_0_0 + WQy * v6_0_1;
                acc[7] += (double)v6_2_0;
                const VT v6_3_0 = QCz * v6_0_0 + WQz * v6_0_1 + (VT)1.0 * oo2ze * v1_0_1;
                acc[8] += (double)v6_3_0;
                const VT v7_1_0 = QCx * v7_0_0 + WQx * v7_0_1;
                acc[9] += (double)v7_1_0;
                const VT v7_2_0 = QCy * v7_0_0 + WQy * v7_0_1 + (VT)2.0 * oo2ze * v2_0_1;
                acc[10] += (double)v7_2_0;
                const VT v7_3_0 = QCz * v7_0_0 + WQz * v7_0_1;
                acc[11] += (double)v7_3_0;
                const VT v8_1_0 = QCx * v8_0_0 + WQx * v8_0_1;
                acc[12] += (double)v8_1_0;
                const VT v8_2_0 = QCy * v8_0_0 + WQy * v8_0_1 + (VT)1.0 * oo2ze * v3_0_1;
                acc[13] += (double)v8_2_0;
                const VT v8_3_0 = QCz * v8_0_0 + WQz * v8_0_1 + (VT)1.0 * oo2ze * v2_0_1;
                acc[14] += (double)v8_3_0;
                const VT v9_1_0 = QCx * v9_0_0 + WQx * v9_0_1;
                acc[15] += (double)v9_1_0;
                const VT v9_2_0 = QCy * v9_0_0 + WQy * v9_0_1;
                acc[16] += (double)v9_2_0;
                const VT v9_3_0 = QCz * v9_0_0 + WQz * v9_0_1 + (VT)2.0 * oo2ze * v3_0_1;
                acc[17] += (double)v9_3_0;
                const VT v10_1_0 = QCx * v10_0_0 + WQx * v10_0_1 + (VT)3.0 * oo2ze * v4_0_1;
                acc[18] += (double)v10_1_0;
                const VT v10_2_0 = QCy * v10_0_0 + WQy * v10_0_1;
                acc[19] += (double)v10_2_0;
                const VT v10_3_0 = QCz * v10_0_0 + WQz * v10_0_1;
                acc[20] += (double)v10_3_0;
                const VT v11_1_0 = QCx * v11_0_0 + WQx * v11_0_1 + (VT)2.0 * oo2ze * v5_0_1;
                acc[21] += (double)v11_1_0;
                const VT v11_2_0 = QCy * v11_0_0 + WQy * v11_0_1 + (VT)1.0 * oo2ze * v4_0_1;
                acc[22] += (double)v11_2_0;
                const VT v11_3_0 = QCz * v11_0_0 + WQz * v11_0_1;
                acc[23] += (double)v11_3_0;
                const VT v12_1_0 = QCx * v12_0_0 + WQx * v12_0_1 + (VT)2.0 * oo2ze * v6_0_1;
                acc[24] += (double)v12_1_0;
                const VT v12_2_0 = QCy * v12_0_0 + WQy * v12_0_1;
                acc[25] += (double)v12_2_0;
                const VT v12_3_0 = QCz * v12_0_0 + WQz * v12_0_1 + (VT)1.0 * oo2ze * v4_0_1;
                acc[26] += (double)v12_3_0;
                const VT v13_1_0 = QCx * v13_0_0 + WQx * v13_0_1 + (VT)1.0 * oo2ze * v7_0_1;
                acc[27] += (double)v13_1_0;
                const VT v13_2_0 = QCy * v13_0_0 + WQy * v13_0_1 + (VT)2.0 * oo2ze * v5_0_1;
                acc[28] += (double)v13_2_0;
                const VT v13_3_0 = QCz * v13_0_0 + WQz * v13_0_1;
                acc[29] += (double)v13_3_0;
                const VT v14_1_0 = QCx * v14_0_0 + WQx * v14_0_1 + (VT)1.0 * oo2ze * v9_0_1;
                acc[30] += (double)v14_1_0;
                const VT v14_2_0 = QCy * v14_0_0 + WQy * v14_0_1;
                acc[31] += (double)v14_2_0;
                const VT v14_3_0 = QCz * v14_0_0 + WQz * v14_0_1 + (VT)2.0 * oo2ze * v6_0_1;
                acc[32] += (double)v14_3_0;
                const VT v15_1_0 = QCx * v15_0_0 + WQx * v15_0_1 + (VT)1.0 * oo2ze * v8_0_1;
                acc[33] += (double)v15_1_0;
                const VT v15_2_0 = QCy * v15_0_0 + WQy * v15_0_1 + (VT)1.0 * oo2ze * v6_0_1;
                acc[34] += (double)v15_2_0;
                const VT v15_3_0 = QCz * v15_0_0 + WQz * v15_0_1 + (VT)1.0 * oo2ze * v5_0_1;
                acc[35] += (double)v15_3_0;
                const VT v16_1_0 = QCx * v16_0_0 + WQx * v16_0_1;
                acc[36] += (double)v16_1_0;
                const VT v16_2_0 = QCy * v16_0_0 + WQy * v16_0_1 + (VT)3.0 * oo2ze * v7_0_1;
                acc[37] += (double)v16_2_0;
                const VT v16_3_0 = QCz * v16_0_0 + WQz * v16_0_1;
                acc[38] += (double)v16_3_0;
                const VT v17_1_0 = QCx * v17_0_0 + WQx * v17_0_1;
                acc[39] += (double)v17_1_0;
                const VT v17_2_0 = QCy * v17_0_0 + WQy * v17_0_1 + (VT)2.0 * oo2ze * v8_0_1;
                acc[40] += (double)v17_2_0;
                const VT v17_3_0 = QCz * v17_0_0 + WQz * v17_0_1 + (VT)1.0 * oo2ze * v7_0_1;
                acc[41] += (double)v17_3_0;
                const VT v18_1_0 = QCx * v18_0_0 + WQx * v18_0_1;
                acc[42] += (double)v18_1_0;
                const VT v18_2_0 = QCy * v18_0_0 + WQy * v18_0_1 + (VT)1.0 * oo2ze * v9_0_1;
                acc[43] += (double)v18_2_0;
                const VT v18_3_0 = QCz * v18_0_0 + WQz * v18_0_1 + (VT)2.0 * oo2ze * v8_0_1;
                acc[44] += (double)v18_3_0;
                const VT v19_1_0 = QCx * v19_0_0 + WQx * v19_0_1;
                acc[45] += (double)v19_1_0;
                const VT v19_2_0 = QCy * v19_0_0 + WQy * v19_0_1;
                acc[46] += (double)v19_2_0;
                const VT v19_3_0 = QCz * v19_0_0 + WQz * v19_0_1 + (VT)3.0 * oo2ze * v9_0_1;
                acc[47] += (double)v19_3_0;
                const VT v20_1_0 = QCx * v20_0_0 + WQx * v20_0_1 + (VT)4.0 * oo2ze * v10_0_1;
                acc[48] += (double)v20_1_0;
                const VT v20_2_0 = QCy * v20_0_0 + WQy * v20_0_1;
                acc[49] += (double)v20_2_0;
                const VT v20_3_0 = QCz * v20_0_0 + WQz * v20_0_1;
                acc[50] += (double)v20_3_0;
                const VT v21_1_0 = QCx * v21_0_0 + WQx * v21_0_1 + (VT)3.0 * oo2ze * v11_0_1;
                acc[51] += (double)v21_1_0;
                const VT v21_2_0 = QCy * v21_0_0 + WQy * v21_0_1 + (VT)1.0 * oo2ze * v10_0_1;
                acc[52] += (double)v21_2_0;
                const VT v21_3_0 = QCz * v21_0_0 + WQz * v21_0_1;
                acc[53] += (double)v21_3_0;
                const VT v22_1_0 = QCx * v22_0_0 + WQx * v22_0_1 + (VT)3.0 * oo2ze * v12_0_1;
                acc[54] += (double)v22_1_0;
                const VT v22_2_0 = QCy * v22_0_0 + WQy * v22_0_1;
                acc[55] += (double)v22_2_0;
                const VT v22_3_0 = QCz * v22_0_0 + WQz * v22_0_1 + (VT)1.0 * oo2ze * v10_0_1;
                acc[56] += (double)v22_3_0;
                const VT v23_1_0 = QCx * v23_0_0 + WQx * v23_0_1 + (VT)2.0 * oo2ze * v13_0_1;
                acc[57] += (double)v23_1_0;
                const VT v23_2_0 = QCy * v23_0_0 + WQy * v23_0_1 + (VT)2.0 * oo2ze * v11_0_1;
                acc[58] += (double)v23_2_0;
                const VT v23_3_0 = QCz * v23_0_0 + WQz * v23_0_1;
                acc[59] += (double)v23_3_0;
                const VT v24_1_0 = QCx * v24_0_0 + WQx * v24_0_1 + (VT)2.0 * oo2ze * v15_0_1;
                acc[60] += (double)v24_1_0;
                const VT v24_2_0 = QCy * v24_0_0 + WQy * v24_0_1 + (VT)1.0 * oo2ze * v12_0_1;
                acc[61] += (double)v24_2_0;
                const VT v24_3_0 = QCz * v24_0_0 + WQz * v24_0_1 + (VT)1.0 * oo2ze * v11_0_1;
                acc[62] += (double)v24_3_0;
                const VT v25_1_0 = QCx * v25_0_0 + WQx * v25_0_1 + (VT)2.0 * oo2ze * v14_0_1;
                acc[63] += (double)v25_1_0;
                const VT v25_2_0 = QCy * v25_0_0 + WQy * v25_0_1;
                acc[64] += (double)v25_2_0;
                const VT v25_3_0 = QCz * v25_0_0 + WQz * v25_0_1 + (VT)2.0 * oo2ze * v12_0_1;
                acc[65] += (double)v25_3_0;
                const VT v26_1_0 = QCx * v26_0_0 + WQx * v26_0_1 + (VT)1.0 * oo2ze * v16_0_1;
                acc[66] += (double)v26_1_0;
                const VT v26_2_0 = QCy * v26_0_0 + WQy * v26_0_1 + (VT)3.0 * oo2ze * v13_0_1;
                acc[67] += (double)v26_2_0;
                const VT v26_3_0 = QCz * v26_0_0 + WQz * v26_0_1;
                acc[68] += (double)v26_3_0;
                const VT v27_1_0 = QCx * v27_0_0 + WQx * v27_0_1 + (VT)1.0 * oo2ze * v17_0_1;
                acc[69] += (double)v27_1_0;
                const VT v27_2_0 = QCy * v27_0_0 + WQy * v27_0_1 + (VT)2.0 * oo2ze * v15_0_1;
                acc[70] += (double)v27_2_0;
                const VT v27_3_0 = QCz * v27_0_0 + WQz * v27_0_1 + (VT)1.0 * oo2ze * v13_0_1;
                acc[71] += (double)v27_3_0;
                const VT v28_1_0 = QCx * v28_0_0 + WQx * v28_0_1 + (VT)1.0 * oo2ze * v18_0_1;
                acc[72] += (double)v28_1_0;
                const VT v28_2_0 = QCy * v28_0_0 + WQy * v28_0_1 + (VT)1.0 * oo2ze * v14_0_1;
                acc[73] += (double)v28_2_0;
                const VT v28_3_0 = QCz * v28_0_0 + WQz * v28_0_1 + (VT)2.0 * oo2ze * v15_0_1;
                acc[74] += (double)v28_3_0;
                const VT v29_1_0 = QCx * v29_0_0 + WQx * v29_0_1 + (VT)1.0 * oo2ze * v19_0_1;
                acc[75] += (double)v29_1_0;
                const VT v29_2_0 = QCy * v29_0_0 + WQy * v29_0_1;
                acc[76] += (double)v29_2_0;
                const VT v29_3_0 = QCz * v29_0_0 + WQz * v29_0_1 + (VT)3.0 * oo2ze * v14_0_1;
                acc[77] += (double)v29_3_0;
                const VT v30_1_0 = QCx * v30_0_0 + WQx * v30_0_1;
                acc[78] += (double)v30_1_0;
                const VT v30_2_0 = QCy * v30_0_0 + WQy * v30_0_1 + (VT)4.0 * oo2ze * v16_0_1;
                acc[79] += (double)v30_2_0;
                const VT v30_3_0 = QCz * v30_0_0 + WQz * v30_0_1;
                acc[80] += (double)v30_3_0;
                const VT v31_1_0 = QCx * v31_0_0 + WQx * v31_0_1;
                acc[81] += (double)v31_1_0;
                const VT v31_2_0 = QCy * v31_0_0 + WQy * v31_0_1 + (VT)3.0 * oo2ze * v17_0_1;
                acc[82] += (double)v31_2_0;
                const VT v31_3_0 = QCz * v31_0_0 + WQz * v31_0_1 + (VT)1.0 * oo2ze * v16_0_1;
                acc[83] += (double)v31_3_0;
                const VT v32_1_0 = QCx * v32_0_0 + WQx * v32_0_1;
                acc[84] += (double)v32_1_0;
                const VT v32_2_0 = QCy * v32_0_0 + WQy * v32_0_1 + (VT)2.0 * oo2ze * v18_0_1;
                acc[85] += (double)v32_2_0;
                const VT v32_3_0 = QCz * v32_0_0 + WQz * v32_0_1 + (VT)2.0 * oo2ze * v17_0_1;
                acc[86] += (double)v32_3_0;
                const VT v33_1_0 = QCx * v33_0_0 + WQx * v33_0_1;
                acc[87] += (double)v33_1_0;
                const VT v33_2_0 = QCy * v33_0_0 + WQy * v33_0_1 + (VT)1.0 * oo2ze * v19_0_1;
                acc[88] += (double)v33_2_0;
                const VT v33_3_0 = QCz * v33_0_0 + WQz * v33_0_1 + (VT)3.0 * oo2ze * v18_0_1;
                acc[89] += (double)v33_3_0;
                const VT v34_1_0 = QCx * v34_0_0 + WQx * v34_0_1;
                acc[90] += (double)v34_1_0;
                const VT v34_2_0 = QCy * v34_0_0 + WQy * v34_0_1;
                acc[91] += (double)v34_2_0;
                const VT v34_3_0 = QCz * v34_0_0 + WQz * v34_0_1 + (VT)4.0 * oo2ze * v19_0_1;
                acc[92] += (double)v34_3_0;
            }
        }
    }
}

// Bra and ket HRR of the contracted block (src/HGP.jl:92-114), then the component norms:
// the normalised (ab|cd) of bra pair p and ket pair q into res[108] (ma, mb, mc, md
// row-major).
__device__ __forceinline__ void hrr_ddps(const PairTab &P, int p, int q, const double *__restrict__ acc,
                                          double *__restrict__ res) {
    const double4 gb = ldg4(&P.geo[p]);
    const double4 gk = ldg4(&P.geo[q]);
    const double ABx = gb.x, ABy = gb.y, ABz = gb.z;
    const double CDx = gk.x, CDy = gk.y, CDz = gk.z;
    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;
    const double h10_1_1 = acc[48] + ABx * acc[18];
    const double h4_1_1 = acc[18] + ABx * acc[0];
    const double h4_4_1 = h10_1_1 + ABx * h4_1_1;
    const double h10_1_2 = acc[49] + ABx * acc[19];
    const double h4_1_2 = acc[19] + ABx * acc[1];
    const double h4_4_2 = h10_1_2 + ABx * h4_1_2;
    const double h10_1_3 = acc[50] + ABx * acc[20];
    const double h4_1_3 = acc[20] + ABx * acc[2];
    const double h4_4_3 = h10_1_3 + ABx * h4_1_3;
    const double h10_2_1 = acc[51] + ABy * acc[18];
    const double h4_2_1 = acc[21] + ABy * acc[0];
    const double h4_5_1 = h10_2_1 + ABx * h4_2_1;
    const double h10_2_2 = acc[52] + ABy * acc[19];
    const double h4_2_2 = acc[22] + ABy * acc[1];
    const double h4_5_2 = h10_2_2 + ABx * h4_2_2;
    const double h10_2_3 = acc[53] + ABy * acc[20];
    const double h4_2_3 = acc[23] + ABy * acc[2];
    const double h4_5_3 = h10_2_3 + ABx * h4_2_3;
    const double h10_3_1 = acc[54] + ABz * acc[18];
    const double h4_3_1 = acc[24] + ABz * acc[0];
    const double h4_6_1 = h10_3_1 + ABx * h4_3_1;
    const double h10_3_2 = acc[55] + ABz * acc[19];
    const double h4_3_2 = acc[25] + ABz * acc[1];
    const double h4_6_2 = h10_3_2 + ABx * h4_3_2;
    const double h10_3_3 = acc[56] + ABz * acc[20];
    const double h4_3_3 = acc[26] + ABz * acc[2];
    const double h4_6_3 = h10_3_3 + ABx * h4_3_3;
    const double h11_2_1 = acc[57] + ABy * acc[21];
    const double h4_7_1 = h11_2_1 + ABy * h4_2_1;
    const double h11_2_2 = acc[58] + ABy * acc[22];
    const double h4_7_2 = h11_2_2 + ABy * h4_2_2;
    const double h11_2_3 = acc[59] + ABy * acc[23];
    const double h4_7_3 = h11_2_3 + ABy * h4_2_3;
    const double h11_3_1 = acc[60] + ABz * acc[21];
    const double h4_8_1 = h11_3_1 + ABy * h4_3_1;
    const double h11_3_2 = acc[61] + ABz * acc[22];
    const double h4_8_2 = h11_3_2 + ABy * h4_3_2;
    const double h11_3_3 = acc[62] + ABz * acc[23];
    const double h4_8_3 = h11_3_3 + ABy * h4_3_3;
    const double h12_3_1 = acc[63] + ABz * acc[24];
    const double h4_9_1 = h12_3_1 + ABz * h4_3_1;
    const double h12_3_2 = acc[64] + ABz * acc[25];
    const double h4_9_2 = h12_3_2 + ABz * h4_3_2;
    const double h12_3_3 = acc[65] + ABz * acc[26];
    const double h4_9_3 = h12_3_3 + ABz * h4_3_3;
    const double h11_1_1 = acc[51] + ABx * acc[21];
    const double h5_1_1 = acc[21] + ABx * acc[3];
    const double h5_4_1 = h11_1_1 + ABx * h5_1_1;
    const double h11_1_2 = acc[52] + ABx * acc[22];
    const double h5_1_2 = acc[22] + ABx * acc[4];
    const double h5_4_2 = h11_1_2 + ABx * h5_1_2;
    const double h11_1_3 = acc[53] + ABx * acc[23];
    const double h5_1_3 = acc[23] + ABx * acc[5];
    const double h5_4_3 = h11_1_3 + ABx * h5_1_3;
    const double h5_2_1 = acc[27] + ABy * acc[3];
    const double h5_5_1 = h11_2_1 + ABx * h5_2_1;
    const double h5_2_2 = acc[28] + ABy * acc[4];
    const double h5_5_2 = h11_2_2 + ABx * h5_2_2;
    const double h5_2_3 = acc[29] + ABy * acc[5];
    const double h5_5_3 = h11_2_3 + ABx * h5_2_3;
    const double h5_3_1 = acc[33] + ABz * acc[3];
    const double h5_6_1 = h11_3_1 + ABx * h5_3_1;
    const double h5_3_2 = acc[34] + ABz * acc[4];
    const double h5_6_2 = h11_3_2 + ABx * h5_3_2;
    const double h5_3_3 = acc[35] + ABz * acc[5];
    const double h5_6_3 = h11_3_3 + ABx * h5_3_3;
    const double h13_2_1 = acc[66] + ABy * acc[27];
    const double h5_7_1 = h13_2_1 + ABy * h5_2_1;
    const double h13_2_2 = acc[67] + ABy * acc[28];
    const double h5_7_2 = h13_2_2 + ABy * h5_2_2;
    const double h13_2_3 = acc[68] + ABy * acc[29];
    const double h5_7_3 = h13_2_3 + ABy * h5_2_3;
    const double h13_3_1 = acc[69] + ABz * acc[27];
    const double h5_8_1 = h13_3_1 + ABy * h5_3_1;
    const double h13_3_2 = acc[70] + ABz * acc[28];
    const double h5_8_2 = h13_3_2 + ABy * h5_3_2;
    const double h13_3_3 = acc[71] + ABz * acc[29];
    const double h5_8_3 = h13_3_3 + ABy * h5_3_3;
    const double h15_3_1 = acc[72] + ABz * acc[33];
    const double h5_9_1 = h15_3_1 + ABz * h5_3_1;
    const double h15_3_2 = acc[73] + ABz * acc[34];
    const double h5_9_2 = h15_3_2 + ABz * h5_3_2;
    const double h15_3_3 = acc[74] + ABz * acc[35];
    const double h5_9_3 = h15_3_3 + ABz * h5_3_3;
    const double h12_1_1 = acc[54] + ABx * acc[24];
    const double h6_1_1 = acc[24] + ABx * acc[6];
    const double h6_4_1 = h12_1_1 + ABx * h6_1_1;
    const double h12_1_2 = acc[55] + ABx * acc[25];
    const double h6_1_2 = acc[25] + ABx * acc[7];
    const double h6_4_2 = h12_1_2 + ABx * h6_1_2;
    const double h12_1_3 = acc[56] + ABx * acc[26];
    const double h6_1_3 = acc[26] + ABx * acc[8];
    const double h6_4_3 = h12_1_3 + ABx * h6_1_3;
    const double h12_2_1 = acc[60] + ABy * acc[24];
    const double h6_2_1 = acc[33] + ABy * acc[6];
    const double h6_5_1 = h12_2_1 + ABx * h6_2_1;
    const double h12_2_2 = acc[61] + ABy * acc[25];
    const double h6_2_2 = acc[34] + ABy * acc[7];
    const double h6_5_2 = h12_2_2 + ABx * h6_2_2;
    const double h12_2_3 = acc[62] + ABy * acc[26];
    const double h6_2_3 = acc[35] + ABy * acc[8];
    const double h6_5_3 = h12_2_3 + ABx * h6_2_3;
    const double h6_3_1 = acc[30] + ABz * acc[6];
    const double h6_6_1 = h12_3_1 + ABx * h6_3_1;
    const double h6_3_2 = acc[31] + ABz * acc[7];
    const double h6_6_2 = h12_3_2 + ABx * h6_3_2;
    const double h6_3_3 = acc[32] + ABz * acc[8];
    const double h6_6_3 = h12_3_3 + ABx * h6_3_3;
    const double h15_2_1 = acc[69] + ABy * acc[33];
    const double h6_7_1 = h15_2_1 + ABy * h6_2_1;
    const double h15_2_2 = acc[70] + ABy * acc[34];
    const double h6_7_2 = h15_2_2 + ABy * h6_2_2;
    const double h15_2_3 = acc[71] + ABy * acc[35];
    const double h6_7_3 = h15_2_3 + ABy * h6_2_3;
    const double h6_8_1 = h15_3_1 + ABy * h6_3_1;
    const double h6_8_2 = h15_3_2 + ABy * h6_3_2;
    const double h6_8_3 = h15_3_3 + ABy * h6_3_3;
    const double h14_3_1 = acc[75] + ABz * acc[30];
    const double h6_9_1 = h14_3_1 + ABz * h6_3_1;
    const double h14_3_2 = acc[76] + ABz * acc[31];
    const double h6_9_2 = h14_3_2 + ABz * h6_3_2;
    const double h14_3_3 = acc[77] + ABz * acc[32];
    const double h6_9_3 = h14_3_3 + ABz * h6_3_3;
    const double h13_1_1 = acc[57] + ABx * acc[27];
    const double h7_1_1 = acc[27] + ABx * acc[9];
    const double h7_4_1 = h13_1_1 + ABx * h7_1_1;
    const double h13_1_2 = acc[58] + ABx * acc[28];
    const double h7_1_2 = acc[28] + ABx * acc[10];
    const double h7_4_2 = h13_1_2 + ABx * h7_1_2;
    const double h13_1_3 = acc[59] + ABx * acc[29];
    const double h7_1_3 = acc[29] + ABx * acc[11];
    const double h7_4_3 = h13_1_3 + ABx * h7_1_3;
    const double h7_2_1 = acc[36] + ABy * acc[9];
    const double h7_5_1 = h13_2_1 + ABx * h7_2_1;
    const double h7_2_2 = acc[37] + ABy * acc[10];
    const double h7_5_2 = h13_2_2 + ABx * h7_2_2;
    const double h7_2_3 = acc[38] + ABy * acc[11];
    const double h7_5_3 = h13_2_3 + ABx * h7_2_3;
    const double h7_3_1 = acc[39] + ABz * acc[9];
    const double h7_6_1 = h13_3_1 + ABx * h7_3_1;
    const double h7_3_2 = acc[40] + ABz * acc[10];
    const double h7_6_2 = h13_3_2 + ABx * h7_3_2;
    const double h7_3_3 = acc[41] + ABz * acc[11];
    const double h7_6_3 = h13_3_3 + ABx * h7_3_3;
    const double h16_2_1 = acc[78] + ABy * acc[36];
    const double h7_7_1 = h16_2_1 + ABy * h7_2_1;
    const double h16_2_2 = acc[79] + ABy * acc[37];
    const double h7_7_2 = h16_2_2 + ABy * h7_2_2;
    const double h16_2_3 = acc[80] + ABy * acc[38];
    const double h7_7_3 = h16_2_3 + ABy * h7_2_3;
    const double h16_3_1 = acc[81] + ABz * acc[36];
    const double h7_8_1 = h16_3_1 + ABy * h7_3_1;
    const double h16_3_2 = acc[82] + ABz * acc[37];
    const double h7_8_2 = h16_3_2 + ABy * h7_3_2;
    const double h16_3_3 = acc[83] + ABz * acc[38];
    const double h7_8_3 = h16_3_3 + ABy * h7_3_3;
    const double h17_3_1 = acc[84] + ABz * acc[39];
    const double h7_9_1 = h17_3_1 + ABz * h7_3_1;
    const double h17_3_2 = acc[85] + ABz * acc[40];
    const double h7_9_2 = h17_3_2 + ABz * h7_3_2;
    const double h17_3_3 = acc[86] + ABz * acc[41];
    const double h7_9_3 = h17_3_3 + ABz * h7_3_3;
    const double h15_1_1 = acc[60] + ABx * acc[33];
    const double h8_1_1 = acc[33] + ABx * acc[12];
    const double h8_4_1 = h15_1_1 + ABx * h8_1_1;
    const double h15_1_2 = acc[61] + ABx * acc[34];
    const double h8_1_2 = acc[34] + ABx * acc[13];
    const double h8_4_2 = h15_1_2 + ABx * h8_1_2;
    const double h15_1_3 = acc[62] + ABx * acc[35];
    const double h8_1_3 = acc[35] + ABx * acc[14];
    const double h8_4_3 = h15_1_3 + ABx * h8_1_3;
    const double h8_2_1 = acc[39] + ABy * acc[12];
    const double h8_5_1 = h15_2_1 + ABx * h8_2_1;
    const double h8_2_2 = acc[40] + ABy * acc[13];
    const double h8_5_2 = h15_2_2 + ABx * h8_2_2;
    const double h8_2_3 = acc[41] + ABy * acc[14];
    const double h8_5_3 = h15_2_3 + ABx * h8_2_3;
    const double h8_3_1 = acc[42] + ABz * acc[12];
    const double h8_6_1 = h15_3_1 + ABx * h8_3_1;
    const double h8_3_2 = acc[43] + ABz * acc[13];
    const double h8_6_2 = h15_3_2 + ABx * h8_3_2;
    const double h8_3_3 = acc[44] + ABz * acc[14];
    const double h8_6_3 = h15_3_3 + ABx * h8_3_3;
    const double h17_2_1 = acc[81] + ABy * acc[39];
    const double h8_7_1 = h17_2_1 + ABy * h8_2_1;
    const double h17_2_2 = acc[82] + ABy * acc[40];
    const double h8_7_2 = h17_2_2 + ABy * h8_2_2;
    const double h17_2_3 = acc[83] + ABy * acc[41];
    const double h8_7_3 = h17_2_3 + ABy * h8_2_3;
    const double h8_8_1 = h17_3_1 + ABy * h8_3_1;
    const double h8_8_2 = h17_3_2 + ABy * h8_3_2;
    const double h8_8_3 = h17_3_3 + ABy * h8_3_3;
    const double h18_3_1 = acc[87] + ABz * acc[42];
    const double h8_9_1 = h18_3_1 + ABz * h8_3_1;
    const double h18_3_2 = acc[88] + ABz * acc[43];
    const double h8_9_2 = h18_3_2 + ABz * h8_3_2;
    const double h18_3_3 = acc[89] + ABz * acc[44];
    const double h8_9_3 = h18_3_3 + ABz * h8_3_3;
    const double h14_1_1 = acc[63] + ABx * acc[30];
    const double h9_1_1 = acc[30] + ABx * acc[15];
    const double h9_4_1 = h14_1_1 + ABx * h9_1_1;
    const double h14_1_2 = acc[64] + ABx * acc[31];
    const double h9_1_2 = acc[31] + ABx * acc[16];
    const double h9_4_2 = h14_1_2 + ABx * h9_1_2;
    const double h14_1_3 = acc[65] + ABx * acc[32];
    const double h9_1_3 = acc[32] + ABx * acc[17];
    const double h9_4_3 = h14_1_3 + ABx * h9_1_3;
    const double h14_2_1 = acc[72] + ABy * acc[30];
    const double h9_2_1 = acc[42] + ABy * acc[15];
    const double h9_5_1 = h14_2_1 + ABx * h9_2_1;
    const double h14_2_2 = acc[73] + ABy * acc[31];
    const double h9_2_2 = acc[43] + ABy * acc[16];
    const double h9_5_2 = h14_2_2 + ABx * h9_2_2;
    const double h14_2_3 = acc[74] + ABy * acc[32];
    const double h9_2_3 = acc[44] + ABy * acc[17];
    const double h9_5_3 = h14_2_3 + ABx * h9_2_3;
    const double h9_3_1 = acc[45] + ABz * acc[15];
    const double h9_6_1 = h14_3_1 + ABx * h9_3_1;
    const double h9_3_2 = acc[46] + ABz * acc[16];
    const double h9_6_2 = h14_3_2 + ABx * h9_3_2;
    const double h9_3_3 = acc[47] + ABz * acc[17];
    const double h9_6_3 = h14_3_3 + ABx * h9_3_3;
    const double h18_2_1 = acc[84] + ABy * acc[42];
    const double h9_7_1 = h18_2_1 + ABy * h9_2_1;
    const double h18_2_2 = acc[85] + ABy * acc[43];
    const double h9_7_2 = h18_2_2 + ABy * h9_2_2;
    const double h18_2_3 = acc[86] + ABy * acc[44];
    const double h9_7_3 = h18_2_3 + ABy * h9_2_3;
    const double h9_8_1 = h18_3_1 + ABy * h9_3_1;
    const double h9_8_2 = h18_3_2 + ABy * h9_3_2;
    const double h9_8_3 = h18_3_3 + ABy * h9_3_3;
    const double h19_3_1 = acc[90] + ABz * acc[45];
    const double h9_9_1 = h19_3_1 + ABz * h9_3_1;
    const double h19_3_2 = acc[91] + ABz * acc[46];
    const double h9_9_2 = h19_3_2 + ABz * h9_3_2;
    const double h19_3_3 = acc[92] + ABz * acc[47];
    const double h9_9_3 = h19_3_3 + ABz * h9_3_3;
    res[0] = h4_4_1 * 0.3333333333333334;
    res[1] = h4_4_2 * 0.3333333333333334;
    res[2] = h4_4_3 * 0.3333333333333334;
    res[3] = h4_5_1 * 0.5773502691896258;
    res[4] = h4_5_2 * 0.5773502691896258;
    res[5] = h4_5_3 * 0.5773502691896258;
    res[6] = h4_6_1 * 0.5773502691896258;
    res[7] = h4_6_2 * 0.5773502691896258;
    res[8] = h4_6_3 * 0.5773502691896258;
    res[9] = h4_7_1 * 0.3333333333333334;
    res[10] = h4_7_2 * 0.3333333333333334;
    res[11] = h4_7_3 * 0.3333333333333334;
    res[12] = h4_8_1 * 0.5773502691896258;
    res[13] = h4_8_2 * 0.5773502691896258;
    res[14] = h4_8_3 * 0.5773502691896258;
    res[15] = h4_9_1 * 0.3333333333333334;
    res[16] = h4_9_2 * 0.3333333333333334;
    res[17] = h4_9_3 * 0.3333333333333334;
    res[18] = h5_4_1 * 0.5773502691896258;
    res[19] = h5_4_2 * 0.5773502691896258;
    res[20] = h5_4_3 * 0.5773502691896258;
    res[21] = h5_5_1;
    res[22] = h5_5_2;
    res[23] = h5_5_3;
    res[24] = h5_6_1;
    res[25] = h5_6_2;
    res[26] = h5_6_3;
    res[27] = h5_7_1 * 0.5773502691896258;
    res[28] = h5_7_2 * 0.5773502691896258;
    res[29] = h5_7_3 * 0.5773502691896258;
    res[30] = h5_8_1;
    res[31] = h5_8_2;
    res[32] = h5_8_3;
    res[33] = h5_9_1 * 0.5773502691896258;
    res[34] = h5_9_2 * 0.5773502691896258;
    res[35] = h5_9_3 * 0.5773502691896258;
    res[36] = h6_4_1 * 0.5773502691896258;
    res[37] = h6_4_2 * 0.5773502691896258;
    res[38] = h6_4_3 * 0.5773502691896258;
    res[39] = h6_5_1;
    res[40] = h6_5_2;
    res[41] = h6_5_3;
    res[42] = h6_6_1;
    res[43] = h6_6_2;
    res[44] = h6_6_3;
    res[45] = h6_7_1 * 0.5773502691896258;
    res[46] = h6_7_2 * 0.5773502691896258;
    res[47] = h6_7_3 * 0.5773502691896258;
    res[48] = h6_8_1;
    res[49] = h6_8_2;
    res[50] = h6_8_3;
    res[51] = h6_9_1 * 0.5773502691896258;
    res[52] = h6_9_2 * 0.5773502691896258;
    res[53] = h6_9_3 * 0.5773502691896258;
    res[54] = h7_4_1 * 0.3333333333333334;
    res[55] = h7_4_2 * 0.3333333333333334;
    res[56] = h7_4_3 * 0.3333333333333334;
    res[57] = h7_5_1 * 0.5773502691896258;
    res[58] = h7_5_2 * 0.5773502691896258;
    res[59] = h7_5_3 * 0.5773502691896258;
    res[60] = h7_6_1 * 0.5773502691896258;
    res[61] = h7_6_2 * 0.5773502691896258;
    res[62] = h7_6_3 * 0.5773502691896258;
    res[63] = h7_7_1 * 0.3333333333333334;
    res[64] = h7_7_2 * 0.3333333333333334;
    res[65] = h7_7_3 * 0.3333333333333334;
    res[66] = h7_8_1 * 0.5773502691896258;
    res[67] = h7_8_2 * 0.5773502691896258;
    res[68] = h7_8_3 * 0.5773502691896258;
    res[69] = h7_9_1 * 0.3333333333333334;
    res[70] = h7_9_2 * 0.3333333333333334;
    res[71] = h7_9_3 * 0.3333333333333334;
    res[72] = h8_4_1 * 0.5773502691896258;
    res[73] = h8_4_2 * 0.5773502691896258;
    res[74] = h8_4_3 * 0.5773502691896258;
    res[75] = h8_5_1;
    res[76] = h8_5_2;
    res[77] = h8_5_3;
    res[78] = h8_6_1;
    res[79] = h8_6_2;
    res[80] = h8_6_3;
    res[81] = h8_7_1 * 0.5773502691896258;
    res[82] = h8_7_2 * 0.5773502691896258;
    res[83] = h8_7_3 * 0.5773502691896258;
    res[84] = h8_8_1;
    res[85] = h8_8_2;
    res[86] = h8_8_3;
    res[87] = h8_9_1 * 0.5773502691896258;
    res[88] = h8_9_2 * 0.5773502691896258;
    res[89] = h8_9_3 * 0.5773502691896258;
    res[90] = h9_4_1 * 0.3333333333333334;
    res[91] = h9_4_2 * 0.3333333333333334;
    res[92] = h9_4_3 * 0.3333333333333334;
    res[93] = h9_5_1 * 0.5773502691896258;
    res[94] = h9_5_2 * 0.5773502691896258;
    res[95] = h9_5_3 * 0.5773502691896258;
    res[96] = h9_6_1 * 0.5773502691896258;
    res[97] = h9_6_2 * 0.5773502691896258;
    res[98] = h9_6_3 * 0.5773502691896258;
    res[99] = h9_7_1 * 0.3333333333333334;
    res[100] = h9_7_2 * 0.3333333333333334;
    res[101] = h9_7_3 * 0.3333333333333334;
    res[102] = h9_8_1 * 0.5773502691896258;
    res[103] = h9_8_2 * 0.5773502691896258;
    res[104] = h9_8_3 * 0.5773502691896258;
    res[105] = h9_9_1 * 0.3333333333333334;
    res[106] = h9_9_2 * 0.3333333333333334;
    res[107] = h9_9_3 * 0.3333333333333334;
}

// (ab|cd) over the bra primitive pairs [i0, i1) and ket primitive pairs [j0, j1) into
// res[108]; the contracted block also into acc_out when given (the bound kernels).
template <typename VT>
__device__ __forceinline__ void quartet_ddps(const PairTab &P, const BoysTab &B, int p, int q,
                                              int i0, int i1, int j0, int j1,
                                              double *__restrict__ res,
                                              double *__restrict__ acc_out = nullptr) {
    double acc[93];
    vrr_ddps<VT>(P, B, p, q, i0, i1, 1, j0, j1, 1, acc);
    if (acc_out) {
#pragma unroll
        for (int x = 0; x < 93; ++x) acc_out[x] = acc[x];
    }
    hrr_ddps(P, p, q, acc, res);
}

__device__ __forceinline__ void store_ddps(double *__restrict__ out, const int4 ib_, const int4 ik_,
                                            bool same, const double *__restrict__ res) {
    const bool dab = ib_.z == ib_.w, dcd = ik_.z == ik_.w;
    (void)dab; (void)dcd;
    const long long ij_0_0 = pair_index(ib_.z + 0, ib_.w + 0);
    const long long ij_0_1 = pair_index(ib_.z + 0, ib_.w + 1);
    const long long ij_0_2 = pair_index(ib_.z + 0, ib_.w + 2);
    const long long ij_0_3 = pair_index(ib_.z + 0, ib_.w + 3);
    const long long ij_0_4 = pair_index(ib_.z + 0, ib_.w + 4);
    const long long ij_0_5 = pair_index(ib_.z + 0, ib_.w + 5);
    const long long ij_1_0 = pair_index(ib_.z + 1, ib_.w + 0);
    const long long ij_1_1 = pair_index(ib_.z + 1, ib_.w + 1);
    const long long ij_1_2 = pair_index(ib_.z + 1, ib_.w + 2);
    const long long ij_1_3 = pair_index(ib_.z + 1, ib_.w + 3);
    const long long ij_1_4 = pair_index(ib_.z + 1, ib_.w + 4);
    const long long ij_1_5 = pair_index(ib_.z + 1, ib_.w + 5);
    const long long ij_2_0 = pair_index(ib_.z + 2, ib_.w + 0);
    const long long ij_2_1 = pair_index(ib_.z + 2, ib_.w + 1);
    const long long ij_2_2 = pair_index(ib_.z + 2, ib_.w + 2);
    const long long ij_2_3 = pair_index(ib_.z + 2, ib_.w + 3);
    const long long ij_2_4 = pair_index(ib_.z + 2, ib_.w + 4);
    const long long ij_2_5 = pair_index(ib_.z + 2, ib_.w + 5);
    const long long ij_3_0 = pair_index(ib_.z + 3, ib_.w + 0);
    const long long ij_3_1 = pair_index(ib_.z + 3, ib_.w + 1);
    const long long ij_3_2 = pair_index(ib_.z + 3, ib_.w + 2);
    const long long ij_3_3 = pair_index(ib_.z + 3, ib_.w + 3);
    const long long ij_3_4 = pair_index(ib_.z + 3, ib_.w + 4);
    const long long ij_3_5 = pair_index(ib_.z + 3, ib_.w + 5);
    const long long ij_4_0 = pair_index(ib_.z + 4, ib_.w + 0);
    const long long ij_4_1 = pair_index(ib_.z + 4, ib_.w + 1);
    const long long ij_4_2 = pair_index(ib_.z + 4, ib_.w + 2);
    const long long ij_4_3 = pair_index(ib_.z + 4, ib_.w + 3);
    const long long ij_4_4 = pair_index(ib_.z + 4, ib_.w + 4);
    const long long ij_4_5 = pair_index(ib_.z + 4, ib_.w + 5);
    const long long ij_5_0 = pair_index(ib_.z + 5, ib_.w + 0);
    const long long ij_5_1 = pair_index(ib_.z + 5, ib_.w + 1);
    const long long ij_5_2 = pair_index(ib_.z + 5, ib_.w + 2);
    const long long ij_5_3 = pair_index(ib_.z + 5, ib_.w + 3);
    const long long ij_5_4 = pair_index(ib_.z + 5, ib_.w + 4);
    const long long ij_5_5 = pair_index(ib_.z + 5, ib_.w + 5);
    const long long kl_0_0 = pair_index(ik_.z + 0, ik_.w + 0);
    const long long kl_1_0 = pair_index(ik_.z + 1, ik_.w + 0);
    const long long kl_2_0 = pair_index(ik_.z + 2, ik_.w + 0);
    { const long long ij = ij_0_0, kl = kl_0_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[0]; }
    { const long long ij = ij_0_0, kl = kl_1_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[1]; }
    { const long long ij = ij_0_0, kl = kl_2_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[2]; }
    { const long long ij = ij_0_1, kl = kl_0_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[3]; }
    { const long long ij = ij_0_1, kl = kl_1_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[4]; }
    { const long long ij = ij_0_1, kl = kl_2_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[5]; }
    { const long long ij = ij_0_2, kl = kl_0_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[6]; }
    { const long long ij = ij_0_2, kl = kl_1_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[7]; }
    { const long long ij = ij_0_2, kl = kl_2_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[8]; }
    { const long long ij = ij_0_3, kl = kl_0_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[9]; }
    { const long long ij = ij_0_3, kl = kl_1_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[10]; }
    { const long long ij = ij_0_3, kl = kl_2_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[11]; }
    { const long long ij = ij_0_4, kl = kl_0_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[12]; }
    { const long long ij = ij_0_4, kl = kl_1_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[13]; }
    { const long long ij = ij_0_4, kl = kl_2_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[14]; }
    { const long long ij = ij_0_5, kl = kl_0_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[15]; }
    { const long long ij = ij_0_5, kl = kl_1_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[16]; }
    { const long long ij = ij_0_5, kl = kl_2_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[17]; }
    { const long long ij = ij_1_0, kl = kl_0_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[18]; }
    { const long long ij = ij_1_0, kl = kl_1_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[19]; }
    { const long long ij = ij_1_0, kl = kl_2_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[20]; }
    { const long long ij = ij_1_1, kl = kl_0_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[21]; }
    { const long long ij = ij_1_1, kl = kl_1_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[22]; }
    { const long long ij = ij_1_1, kl = kl_2_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[23]; }
    { const long long ij = ij_1_2, kl = kl_0_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[24]; }
    { const long long ij = ij_1_2, kl = kl_1_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[25]; }
    { const long long ij = ij_1_2, kl = kl_2_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[26]; }
    { const long long ij = ij_1_3, kl = kl_0_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[27]; }
    { const long long ij = ij_1_3, kl = kl_1_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[28]; }
    { const long long ij = ij_1_3, kl = kl_2_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[29]; }
    { const long long ij = ij_1_4, kl = kl_0_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[30]; }
    { const long long ij = ij_1_4, kl = kl_1_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[31]; }
    { const long long ij = ij_1_4, kl = kl_2_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[32]; }
    { const long long ij = ij_1_5, kl = kl_0_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[33]; }
    { const long long ij = ij_1_5, kl = kl_1_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[34]; }
    { const long long ij = ij_1_5, kl = kl_2_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[35]; }
    { const long long ij = ij_2_0, kl = kl_0_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[36]; }
    { const long long ij = ij_2_0, kl = kl_1_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[37]; }
    { const long long ij = ij_2_0, kl = kl_2_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[38]; }
    { const long long ij = ij_2_1, kl = kl_0_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[39]; }
    { const long long ij = ij_2_1, kl = kl_1_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[40]; }
    { const long long ij = ij_2_1, kl = kl_2_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[41]; }
    { const long long ij = ij_2_2, kl = kl_0_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[42]; }
    { const long long ij = ij_2_2, kl = kl_1_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[43]; }
    { const long long ij = ij_2_2, kl = kl_2_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[44]; }
    { const long long ij = ij_2_3, kl = kl_0_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[45]; }
    { const long long ij = ij_2_3, kl = kl_1_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[46]; }
    { const long long ij = ij_2_3, kl = kl_2_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[47]; }
    { const long long ij = ij_2_4, kl = kl_0_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[48]; }
    { const long long ij = ij_2_4, kl = kl_1_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[49]; }
    { const long long ij = ij_2_4, kl = kl_2_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[50]; }
    { const long long ij = ij_2_5, kl = kl_0_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[51]; }
    { const long long ij = ij_2_5, kl = kl_1_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[52]; }
    { const long long ij = ij_2_5, kl = kl_2_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[53]; }
    { const long long ij = ij_3_0, kl = kl_0_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[54]; }
    { const long long ij = ij_3_0, kl = kl_1_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[55]; }
    { const long long ij = ij_3_0, kl = kl_2_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[56]; }
    { const long long ij = ij_3_1, kl = kl_0_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[57]; }
    { const long long ij = ij_3_1, kl = kl_1_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[58]; }
    { const long long ij = ij_3_1, kl = kl_2_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[59]; }
    { const long long ij = ij_3_2, kl = kl_0_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[60]; }
    { const long long ij = ij_3_2, kl = kl_1_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[61]; }
    { const long long ij = ij_3_2, kl = kl_2_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[62]; }
    { const long long ij = ij_3_3, kl = kl_0_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[63]; }
    { const long long ij = ij_3_3, kl = kl_1_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[64]; }
    { const long long ij = ij_3_3, kl = kl_2_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[65]; }
    { const long long ij = ij_3_4, kl = kl_0_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[66]; }
    { const long long ij = ij_3_4, kl = kl_1_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[67]; }
    { const long long ij = ij_3_4, kl = kl_2_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[68]; }
    { const long long ij = ij_3_5, kl = kl_0_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[69]; }
    { const long long ij = ij_3_5, kl = kl_1_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[70]; }
    { const long long ij = ij_3_5, kl = kl_2_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[71]; }
    { const long long ij = ij_4_0, kl = kl_0_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[72]; }
    { const long long ij = ij_4_0, kl = kl_1_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[73]; }
    { const long long ij = ij_4_0, kl = kl_2_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[74]; }
    { const long long ij = ij_4_1, kl = kl_0_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[75]; }
    { const long long ij = ij_4_1, kl = kl_1_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[76]; }
    { const long long ij = ij_4_1, kl = kl_2_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[77]; }
    { const long long ij = ij_4_2, kl = kl_0_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[78]; }
    { const long long ij = ij_4_2, kl = kl_1_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[79]; }
    { const long long ij = ij_4_2, kl = kl_2_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[80]; }
    { const long long ij = ij_4_3, kl = kl_0_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[81]; }
    { const long long ij = ij_4_3, kl = kl_1_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[82]; }
    { const long long ij = ij_4_3, kl = kl_2_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[83]; }
    { const long long ij = ij_4_4, kl = kl_0_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[84]; }
    { const long long ij = ij_4_4, kl = kl_1_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[85]; }
    { const long long ij = ij_4_4, kl = kl_2_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[86]; }
    { const long long ij = ij_4_5, kl = kl_0_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[87]; }
    { const long long ij = ij_4_5, kl = kl_1_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[88]; }
    { const long long ij = ij_4_5, kl = kl_2_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[89]; }
    { const long long ij = ij_5_0, kl = kl_0_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[90]; }
    { const long long ij = ij_5_0, kl = kl_1_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[91]; }
    { const long long ij = ij_5_0, kl = kl_2_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[92]; }
    { const long long ij = ij_5_1, kl = kl_0_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[93]; }
    { const long long ij = ij_5_1, kl = kl_1_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[94]; }
    { const long long ij = ij_5_1, kl = kl_2_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[95]; }
    { const long long ij = ij_5_2, kl = kl_0_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[96]; }
    { const long long ij = ij_5_2, kl = kl_1_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[97]; }
    { const long long ij = ij_5_2, kl = kl_2_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[98]; }
    { const long long ij = ij_5_3, kl = kl_0_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[99]; }
    { const long long ij = ij_5_3, kl = kl_1_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[100]; }
    { const long long ij = ij_5_3, kl = kl_2_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[101]; }
    { const long long ij = ij_5_4, kl = kl_0_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[102]; }
    { const long long ij = ij_5_4, kl = kl_1_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[103]; }
    { const long long ij = ij_5_4, kl = kl_2_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[104]; }
    { const long long ij = ij_5_5, kl = kl_0_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[105]; }
    { const long long ij = ij_5_5, kl = kl_1_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[106]; }
    { const long long ij = ij_5_5, kl = kl_2_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[107]; }
}

// The quartet's share of J and K (molints_plan_jk, eri_common.cuh): every integral of the block,
// times f, into one orientation of each target; J_ab stays in the lane (one bra pair per chunk).
__device__ __forceinline__ void jk_ddps(const JKOut &jk, const int4 ib_, const int4 ik_, double f,
                                         const double *__restrict__ res, double *__restrict__ jab) {
    const long long n = jk.n;
    const double *__restrict__ D = jk.D;
    const double *__restrict__ Db = D + ib_.w * n, *__restrict__ Dc = D + ik_.z * n;
    double dcd[3], dbc[18], dbd[6], jcd[3], kbc[18], kbd[6];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 1; ++l) {
            dcd[k * 1 + l] = __ldg(&Dc[k * n + ik_.w + l]);
            jcd[k * 1 + l] = 0.0;
        }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            dbc[j * 3 + k] = __ldg(&Db[j * n + ik_.z + k]);
            kbc[j * 3 + k] = 0.0;
        }
#pragma unroll
        for (int l = 0; l < 1; ++l) {
            dbd[j * 1 + l] = __ldg(&Db[j * n + ik_.w + l]);
            kbd[j * 1 + l] = 0.0;
        }
    }
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
        const double *__restrict__ Da = D + (ib_.z + i) * n;
        double dab[6], dac[3], dad[1], kac[3], kad[1];
#pragma unroll
        for (int j = 0; j < 6; ++j) dab[j] = __ldg(&Da[ib_.w + j]);
#pragma unroll
        for (int k = 0; k < 3; ++k) { dac[k] = __ldg(&Da[ik_.z + k]); kac[k] = 0.0; }
#pragma unroll
        for (int l = 0; l < 1; ++l) { dad[l] = __ldg(&Da[ik_.w + l]); kad[l] = 0.0; }
        { const double v = f * res[(i * 6 + 0) * 3 + 0];
          jab[i * 6 + 0] = fma(dcd[0], v, jab[i * 6 + 0]);
          jcd[0] = fma(dab[0], v, jcd[0]);
          kac[0] = fma(dbd[0], v, kac[0]);
          kad[0] = fma(dbc[0], v, kad[0]);
          kbc[0] = fma(dad[0], v, kbc[0]);
          kbd[0] = fma(dac[0], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 3 + 1];
          jab[i * 6 + 0] = fma(dcd[1], v, jab[i * 6 + 0]);
          jcd[1] = fma(dab[0], v, jcd[1]);
          kac[1] = fma(dbd[0], v, kac[1]);
          kad[0] = fma(dbc[1], v, kad[0]);
          kbc[1] = fma(dad[0], v, kbc[1]);
          kbd[0] = fma(dac[1], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 3 + 2];
          jab[i * 6 + 0] = fma(dcd[2], v, jab[i * 6 + 0]);
          jcd[2] = fma(dab[0], v, jcd[2]);
          kac[2] = fma(dbd[0], v, kac[2]);
          kad[0] = fma(dbc[2], v, kad[0]);
          kbc[2] = fma(dad[0], v, kbc[2]);
          kbd[0] = fma(dac[2], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 1) * 3 + 0];
          jab[i * 6 + 1] = fma(dcd[0], v, jab[i * 6 + 1]);
          jcd[0] = fma(dab[1], v, jcd[0]);
          kac[0] = fma(dbd[1], v, kac[0]);
          kad[0] = fma(dbc[3], v, kad[0]);
          kbc[3] = fma(dad[0], v, kbc[3]);
          kbd[1] = fma(dac[0], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 3 + 1];
          jab[i * 6 + 1] = fma(dcd[1], v, jab[i * 6 + 1]);
          jcd[1] = fma(dab[1], v, jcd[1]);
          kac[1] = fma(dbd[1], v, kac[1]);
          kad[0] = fma(dbc[4], v, kad[0]);
          kbc[4] = fma(dad[0], v, kbc[4]);
          kbd[1] = fma(dac[1], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 3 + 2];
          jab[i * 6 + 1] = fma(dcd[2], v, jab[i * 6 + 1]);
          jcd[2] = fma(dab[1], v, jcd[2]);
          kac[2] = fma(dbd[1], v, kac[2]);
          kad[0] = fma(dbc[5], v, kad[0]);
          kbc[5] = fma(dad[0], v, kbc[5]);
          kbd[1] = fma(dac[2], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 2) * 3 + 0];
          jab[i * 6 + 2] = fma(dcd[0], v, jab[i * 6 + 2]);
          jcd[0] = fma(dab[2], v, jcd[0]);
          kac[0] = fma(dbd[2], v, kac[0]);
          kad[0] = fma(dbc[6], v, kad[0]);
          kbc[6] = fma(dad[0], v, kbc[6]);
          kbd[2] = fma(dac[0], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 3 + 1];
          jab[i * 6 + 2] = fma(dcd[1], v, jab[i * 6 + 2]);
          jcd[1] = fma(dab[2], v, jcd[1]);
          kac[1] = fma(dbd[2], v, kac[1]);
          kad[0] = fma(dbc[7], v, kad[0]);
          kbc[7] = fma(dad[0], v, kbc[7]);
          kbd[2] = fma(dac[1], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 3 + 2];
          jab[i * 6 + 2] = fma(dcd[2], v, jab[i * 6 + 2]);
          jcd[2] = fma(dab[2], v, jcd[2]);
          kac[2] = fma(dbd[2], v, kac[2]);
          kad[0] = fma(dbc[8], v, kad[0]);
          kbc[8] = fma(dad[0], v, kbc[8]);
          kbd[2] = fma(dac[2], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 3) * 3 + 0];
          jab[i * 6 + 3] = fma(dcd[0], v, jab[i * 6 + 3]);
          jcd[0] = fma(dab[3], v, jcd[0]);
          kac[0] = fma(dbd[3], v, kac[0]);
          kad[0] = fma(dbc[9], v, kad[0]);
          kbc[9] = fma(dad[0], v, kbc[9]);
          kbd[3] = fma(dac[0], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 3 + 1];
          jab[i * 6 + 3] = fma(dcd[1], v, jab[i * 6 + 3]);
          jcd[1] = fma(dab[3], v, jcd[1]);
          kac[1] = fma(dbd[3], v, kac[1]);
          kad[0] = fma(dbc[10], v, kad[0]);
          kbc[10] = fma(dad[0], v, kbc[10]);
          kbd[3] = fma(dac[1], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 3 + 2];
          jab[i * 6 + 3] = fma(dcd[2], v, jab[i * 6 + 3]);
          jcd[2] = fma(dab[3], v, jcd[2]);
          kac[2] = fma(dbd[3], v, kac[2]);
          kad[0] = fma(dbc[11], v, kad[0]);
          kbc[11] = fma(dad[0], v, kbc[11]);
          kbd[3] = fma(dac[2], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 4) * 3 + 0];
          jab[i * 6 + 4] = fma(dcd[0], v, jab[i * 6 + 4]);
          jcd[0] = fma(dab[4], v, jcd[0]);
          kac[0] = fma(dbd[4], v, kac[0]);
          kad[0] = fma(dbc[12], v, kad[0]);
          kbc[12] = fma(dad[0], v, kbc[12]);
          kbd[4] = fma(dac[0], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 3 + 1];
          jab[i * 6 + 4] = fma(dcd[1], v, jab[i * 6 + 4]);
          jcd[1] = fma(dab[4], v, jcd[1]);
          kac[1] = fma(dbd[4], v, kac[1]);
          kad[0] = fma(dbc[13], v, kad[0]);
          kbc[13] = fma(dad[0], v, kbc[13]);
          kbd[4] = fma(dac[1], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 3 + 2];
          jab[i * 6 + 4] = fma(dcd[2], v, jab[i * 6 + 4]);
          jcd[2] = fma(dab[4], v, jcd[2]);
          kac[2] = fma(dbd[4], v, kac[2]);
          kad[0] = fma(dbc[14], v, kad[0]);
          kbc[14] = fma(dad[0], v, kbc[14]);
          kbd[4] = fma(dac[2], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 5) * 3 + 0];
          jab[i * 6 + 5] = fma(dcd[0], v, jab[i * 6 + 5]);
          jcd[0] = fma(dab[5], v, jcd[0]);
          kac[0] = fma(dbd[5], v, kac[0]);
          kad[0] = fma(dbc[15], v, kad[0]);
          kbc[15] = fma(dad[0], v, kbc[15]);
          kbd[5] = fma(dac[0], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 3 + 1];
          jab[i * 6 + 5] = fma(dcd[1], v, jab[i * 6 + 5]);
          jcd[1] = fma(dab[5], v, jcd[1]);
          kac[1] = fma(dbd[5], v, kac[1]);
          kad[0] = fma(dbc[16], v, kad[0]);
          kbc[16] = fma(dad[0], v, kbc[16]);
          kbd[5] = fma(dac[1], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 3 + 2];
          jab[i * 6 + 5] = fma(dcd[2], v, jab[i * 6 + 5]);
          jcd[2] = fma(dab[5], v, jcd[2]);
          kac[2] = fma(dbd[5], v, kac[2]);
          kad[0] = fma(dbc[17], v, kad[0]);
          kbc[17] = fma(dad[0], v, kbc[17]);
          kbd[5] = fma(dac[2], v, kbd[5]); }
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.z + k], kac[k]);
#pragma unroll
        for (int l = 0; l < 1; ++l) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.w + l], kad[l]);
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.z + k], kbc[j * 3 + k]);
#pragma unroll
        for (int l = 0; l < 1; ++l) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.w + l], kbd[j * 1 + l]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 1; ++l) atomicAdd(&jk.J[(ik_.z + k) * n + ik_.w + l], 2.0 * jcd[k * 1 + l]);
}

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
__global__ void __launch_bounds__(128) eri_queue_ddps(const EriQueue Q) {
    const int lane = threadIdx.x & 31;
    for (;;) {
        int c = 0;
        if (lane == 0) c = atomicAdd(Q.counter, 1);
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= Q.nchunks) return;
        const int4 ch = __ldg(&Q.chunks[c]);
        const int p = ch.x, cnt = ch.z & 0xffff, lg = (ch.z >> 16) & 7, lgj = (ch.z >> 20) & 7;
        const int W = 32 >> lg, kq = lane & (W - 1), s = lane >> (5 - lg);
        const int js = s & ((1 << lgj) - 1), is = s >> lgj;
        double jab[JK ? 36 : 1];  // J/K digestion: the bra pair's J, over the chunk
        if constexpr (JK) {
#pragma unroll
            for (int x = 0; x < 36; ++x) jab[x] = 0.0;
        }
        for (int base = 0; base < cnt; base += W) {
        const int q = ch.y + base + kq;
        const bool live = base + kq < cnt;
        double acc[93];
        double2 bp = make_double2(0.0, 0.0), bq = bp;
        if (live) {
            bp = __ldg(&Q.pairs.bnd[p]);
            bq = __ldg(&Q.pairs.bnd[q]);
        }
        if (!live || bp.x * bq.x < Q.screen_cut) {
#pragma unroll
            for (int x = 0; x < 93; ++x) acc[x] = 0.0;
        } else {
            const int nb = __ldg(&Q.pairs.info[p]).y, nk = __ldg(&Q.pairs.info[q]).y;
            if (MIXED && bp.y * bq.y < Q.fp32_cut)
                vrr_ddps<float>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
            else vrr_ddps<double>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
        }
        if (lg) {
            for (int off = W; off < 32; off <<= 1) {
#pragma unroll
                for (int x = 0; x < 93; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
            }
        }
        const bool lead = live && s == 0;
        if (!JK && Q.scratch) {
            // two-phase: the leaders' HRR writes the blocks of the chunk's quartets straight
            // into shared memory, where they lie as in the scratch (consecutive slots); the warp
            // then copies them out as one contiguous run
            extern __shared__ double stg[];  // 4 * 32 * 108 doubles (launch_eri_ddps)
            double *sb = stg + (threadIdx.x >> 5) * (32 * 108);
            if (lead) hrr_ddps(Q.pairs, p, q, acc, sb + kq * 108);
            __syncwarp();
            const int nlive = min(W, cnt - base);
            double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                (__ldg(&Q.chunk_slot[c]) + base) * (long long)108;
            for (int t = lane; t < nlive * 108; t += 32) dst[t] = sb[t];
            __syncwarp();
        } else if (lead) {
            double res[108];
            hrr_ddps(Q.pairs, p, q, acc, res);
            if constexpr (JK) {
                const int4 ib_ = __ldg(&Q.pairs.info[p]), ik_ = __ldg(&Q.pairs.info[q]);
                jk_ddps(Q.jk, ib_, ik_, jk_weight(ib_.z == ib_.w, ik_.z == ik_.w, p == q), res, jab);
            } else {
                store_ddps(Q.out + __ldg(&Q.mol_out[ch.w]), __ldg(&Q.pairs.info[p]), __ldg(&Q.pairs.info[q]),
                            p == q, res);
            }
        }
        }
        if constexpr (JK) {
            // one addition per J_ab and chunk
            const int4 ib_ = __ldg(&Q.pairs.info[p]);
#pragma unroll
            for (int x = 0; x < 36; ++x) {
                double v = jab[x];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == 0) atomicAdd(&Q.jk.J[(long long)(ib_.z + x / 6) * Q.jk.n + ib_.w + x % 6], 2.0 * v);
            }
        }
    }
}


// The dynamic shared memory of the two-phase staging (110592 bytes), allowed once per device
// (before any graph capture: the occupancy query of plan creation calls it first).
static void eri_prepare_ddps() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(eri_queue_ddps<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 110592);
        cudaFuncSetAttribute(eri_queue_ddps<1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 110592);
        done[dev] = true;
    }
}

void launch_eri_ddps(const EriQueue &Q, int mixed, int grid, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid <= 0) return;
    // two-phase plans stage the chunk's blocks in 110592 bytes of dynamic shared memory
    const size_t smem = Q.scratch && !Q.jk.J ? 110592 : 0;
    if (smem) eri_prepare_ddps();
    const bool jk = Q.jk.J != nullptr;
    if (mixed) { if (jk) eri_queue_ddps<1, 1><<<grid, 128, 0, s>>>(Q); else eri_queue_ddps<1, 0><<<grid, 128, smem, s>>>(Q); }
    else if (jk) eri_queue_ddps<0, 1><<<grid, 128, 0, s>>>(Q);
    else eri_queue_ddps<0, 0><<<grid, 128, smem, s>>>(Q);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_eri_ddps(int mixed) {
    eri_prepare_ddps();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_ddps<1, 0>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_ddps<0, 0>, 128, 0);
    return n;
}

}  // namespace molints
