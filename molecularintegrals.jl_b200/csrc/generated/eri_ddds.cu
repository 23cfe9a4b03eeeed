// Generated by gen_eri.py -- class (dd|ds).  Do not edit.
// VRR entries: 521, contracted block: 186, HRR lines: 474, outputs: 216.
#include "../eri_common.cuh"

namespace molints {

// The contracted [e0|f0] block of bra pair p and ket pair q into acc[186], summed over
// the bra primitive pairs i0, i0 + istep, ... < i1 and the ket primitive pairs j0, j0 + jstep,
// ... < j1 of the two shell pairs.  VT is the VRR arithmetic type (double, or float for MIXED).
// The ket loop is outside: a warp shares its bra pair, so the inner bra loads are broadcasts
// and each lane's ket record is loaded once.  Steps above 1 split one quartet's primitive
// quartets over the lanes of a split group (their blocks are summed before the HRR).
template <typename VT>
__device__ __forceinline__ void vrr_ddds(const PairTab &P, const BoysTab &B, int p, int q,
                                          int i0, int i1, int istep, int j0, int j1, int jstep,
                                          double *__restrict__ acc) {
    const int4 ib_ = __ldg(&P.info[p]);
    const int4 ik_ = __ldg(&P.info[q]);
#pragma unroll
    for (int x = 0; x < 186; ++x) acc[x] = 0.0;
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
            double F[7];
            boys_scaled<6>(far, ze * r2, B, F);
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
            const VT v0_0_6 = (VT)(pref * F[6]);
            const VT v1_0_0 = PAx * v0_0_0 + WPx * v0_0_1;
            const VT v1_0_1 = PAx * v0_0_1 + WPx * v0_0_2;
            const VT v1_0_2 = PAx * v0_0_2 + WPx * v0_0_3;
            const VT v1_0_3 = PAx * v0_0_3 + WPx * v0_0_4;
            const VT v1_0_4 = PAx * v0_0_4 + WPx * v0_0_5;
            const VT v1_0_5 = PAx * v0_0_5 + WPx * v0_0_6;
            const VT v2_0_0 = PAy * v0_0_0 + WPy * v0_0_1;
            const VT v2_0_1 = PAy * v0_0_1 + WPy * v0_0_2;
            const VT v2_0_2 = PAy * v0_0_2 + WPy * v0_0_3;
            const VT v2_0_3 = PAy * v0_0_3 + WPy * v0_0_4;
            const VT v2_0_4 = PAy * v0_0_4 + WPy * v0_0_5;
            const VT v2_0_5 = PAy * v0_0_5 + WPy * v0_0_6;
            const VT v3_0_0 = PAz * v0_0_0 + WPz * v0_0_1;
            const VT v3_0_1 = PAz * v0_0_1 + WPz * v0_0_2;
            const VT v3_0_2 = PAz * v0_0_2 + WPz * v0_0_3;
            const VT v3_0_3 = PAz * v0_0_3 + WPz * v0_0_4;
            const VT v3_0_4 = PAz * v0_0_4 + WPz * v0_0_5;
            const VT v3_0_5 = PAz * v0_0_5 + WPz * v0_0_6;
            const VT v4_0_0 = PAx * v1_0_0 + WPx * v1_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v4_0_1 = PAx * v1_0_1 + WPx * v1_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v4_0_2 = PAx * v1_0_2 + WPx * v1_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v4_0_3 = PAx * v1_0_3 + WPx * v1_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v4_0_4 = PAx * v1_0_4 + WPx * v1_0_5 + (VT)1.0 * oo2z * (v0_0_4 - rho_z * v0_0_5);
            const VT v5_0_0 = PAx * v2_0_0 + WPx * v2_0_1;
            const VT v5_0_1 = PAx * v2_0_1 + WPx * v2_0_2;
            const VT v5_0_2 = PAx * v2_0_2 + WPx * v2_0_3;
            const VT v5_0_3 = PAx * v2_0_3 + WPx * v2_0_4;
            const VT v5_0_4 = PAx * v2_0_4 + WPx * v2_0_5;
            const VT v6_0_0 = PAx * v3_0_0 + WPx * v3_0_1;
            const VT v6_0_1 = PAx * v3_0_1 + WPx * v3_0_2;
            const VT v6_0_2 = PAx * v3_0_2 + WPx * v3_0_3;
            const VT v6_0_3 = PAx * v3_0_3 + WPx * v3_0_4;
            const VT v6_0_4 = PAx * v3_0_4 + WPx * v3_0_5;
            const VT v7_0_0 = PAy * v2_0_0 + WPy * v2_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v7_0_1 = PAy * v2_0_1 + WPy * v2_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v7_0_2 = PAy * v2_0_2 + WPy * v2_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v7_0_3 = PAy * v2_0_3 + WPy * v2_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v7_0_4 = PAy * v2_0_4 + WPy * v2_0_5 + (VT)1.0 * oo2z * (v0_0_4 - rho_z * v0_0_5);
            const VT v8_0_0 = PAy * v3_0_0 + WPy * v3_0_1;
            const VT v8_0_1 = PAy * v3_0_1 + WPy * v3_0_2;
            const VT v8_0_2 = PAy * v3_0_2 + WPy * v3_0_3;
            const VT v8_0_3 = PAy * v3_0_3 + WPy * v3_0_4;
            const VT v8_0_4 = PAy * v3_0_4 + WPy * v3_0_5;
            const VT v9_0_0 = PAz * v3_0_0 + WPz * v3_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v9_0_1 = PAz * v3_0_1 + WPz * v3_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v9_0_2 = PAz * v3_0_2 + WPz * v3_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v9_0_3 = PAz * v3_0_3 + WPz * v3_0_4 + (VT)1.0 * oo2z * (v0_0_3 - rho_z * v0_0_4);
            const VT v9_0_4 = PAz * v3_0_4 + WPz * v3_0_5 + (VT)1.0 * oo2z * (v0_0_4 - rho_z * v0_0_5);
            const VT v10_0_0 = PAx * v4_0_0 + WPx * v4_0_1 + (VT)2.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v10_0_1 = PAx * v4_0_1 + WPx * v4_0_2 + (VT)2.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v10_0_2 = PAx * v4_0_2 + WPx * v4_0_3 + (VT)2.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v10_0_3 = PAx * v4_0_3 + WPx * v4_0_4 + (VT)2.0 * oo2z * (v1_0_3 - rho_z * v1_0_4);
            const VT v11_0_0 = PAx * v5_0_0 + WPx * v5_0_1 + (VT)1.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v11_0_1 = PAx * v5_0_1 + WPx * v5_0_2 + (VT)1.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v11_0_2 = PAx * v5_0_2 + WPx * v5_0_3 + (VT)1.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v11_0_3 = PAx * v5_0_3 + WPx * v5_0_4 + (VT)1.0 * oo2z * (v2_0_3 - rho_z * v2_0_4);
            const VT v12_0_0 = PAx * v6_0_0 + WPx * v6_0_1 + (VT)1.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v12_0_1 = PAx * v6_0_1 + WPx * v6_0_2 + (VT)1.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v12_0_2 = PAx * v6_0_2 + WPx * v6_0_3 + (VT)1.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v12_0_3 = PAx * v6_0_3 + WPx * v6_0_4 + (VT)1.0 * oo2z * (v3_0_3 - rho_z * v3_0_4);
            const VT v13_0_0 = PAy * v5_0_0 + WPy * v5_0_1 + (VT)1.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v13_0_1 = PAy * v5_0_1 + WPy * v5_0_2 + (VT)1.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v13_0_2 = PAy * v5_0_2 + WPy * v5_0_3 + (VT)1.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v13_0_3 = PAy * v5_0_3 + WPy * v5_0_4 + (VT)1.0 * oo2z * (v1_0_3 - rho_z * v1_0_4);
            const VT v14_0_0 = PAz * v6_0_0 + WPz * v6_0_1 + (VT)1.0 * oo2z * (v1_0_0 - rho_z * v1_0_1);
            const VT v14_0_1 = PAz * v6_0_1 + WPz * v6_0_2 + (VT)1.0 * oo2z * (v1_0_1 - rho_z * v1_0_2);
            const VT v14_0_2 = PAz * v6_0_2 + WPz * v6_0_3 + (VT)1.0 * oo2z * (v1_0_2 - rho_z * v1_0_3);
            const VT v14_0_3 = PAz * v6_0_3 + WPz * v6_0_4 + (VT)1.0 * oo2z * (v1_0_3 - rho_z * v1_0_4);
            const VT v15_0_0 = PAx * v8_0_0 + WPx * v8_0_1;
            const VT v15_0_1 = PAx * v8_0_1 + WPx * v8_0_2;
            const VT v15_0_2 = PAx * v8_0_2 + WPx * v8_0_3;
            const VT v15_0_3 = PAx * v8_0_3 + WPx * v8_0_4;
            const VT v16_0_0 = PAy * v7_0_0 + WPy * v7_0_1 + (VT)2.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v16_0_1 = PAy * v7_0_1 + WPy * v7_0_2 + (VT)2.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v16_0_2 = PAy * v7_0_2 + WPy * v7_0_3 + (VT)2.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v16_0_3 = PAy * v7_0_3 + WPy * v7_0_4 + (VT)2.0 * oo2z * (v2_0_3 - rho_z * v2_0_4);
            const VT v17_0_0 = PAy * v8_0_0 + WPy * v8_0_1 + (VT)1.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v17_0_1 = PAy * v8_0_1 + WPy * v8_0_2 + (VT)1.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v17_0_2 = PAy * v8_0_2 + WPy * v8_0_3 + (VT)1.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v17_0_3 = PAy * v8_0_3 + WPy * v8_0_4 + (VT)1.0 * oo2z * (v3_0_3 - rho_z * v3_0_4);
            const VT v18_0_0 = PAz * v8_0_0 + WPz * v8_0_1 + (VT)1.0 * oo2z * (v2_0_0 - rho_z * v2_0_1);
            const VT v18_0_1 = PAz * v8_0_1 + WPz * v8_0_2 + (VT)1.0 * oo2z * (v2_0_1 - rho_z * v2_0_2);
            const VT v18_0_2 = PAz * v8_0_2 + WPz * v8_0_3 + (VT)1.0 * oo2z * (v2_0_2 - rho_z * v2_0_3);
            const VT v18_0_3 = PAz * v8_0_3 + WPz * v8_0_4 + (VT)1.0 * oo2z * (v2_0_3 - rho_z * v2_0_4);
            const VT v19_0_0 = PAz * v9_0_0 + WPz * v9_0_1 + (VT)2.0 * oo2z * (v3_0_0 - rho_z * v3_0_1);
            const VT v19_0_1 = PAz * v9_0_1 + WPz * v9_0_2 + (VT)2.0 * oo2z * (v3_0_1 - rho_z * v3_0_2);
            const VT v19_0_2 = PAz * v9_0_2 + WPz * v9_0_3 + (VT)2.0 * oo2z * (v3_0_2 - rho_z * v3_0_3);
            const VT v19_0_3 = PAz * v9_0_3 + WPz * v9_0_4 + (VT)2.0 * oo2z * (v3_0_3 - rho_z * v3_0_4);
            const VT v20_0_0 = PAx * v10_0_0 + WPx * v10_0_1 + (VT)3.0 * oo2z * (v4_0_0 - rho_z * v4_0_1);
            const VT v20_0_1 = PAx * v10_0_1 + WPx * v10_0_2 + (VT)3.0 * oo2z * (v4_0_1 - rho_z * v4_0_2);
            const VT v20_0_2 = PAx * v10_0_2 + WPx * v10_0_3 + (VT)3.0 * oo2z * (v4_0_2 - rho_z * v4_0_3);
            const VT v21_0_0 = PAx * v11_0_0 + WPx * v11_0_1 + (VT)2.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v21_0_1 = PAx * v11_0_1 + WPx * v11_0_2 + (VT)2.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v21_0_2 = PAx * v11_0_2 + WPx * v11_0_3 + (VT)2.0 * oo2z * (v5_0_2 - rho_z * v5_0_3);
            const VT v22_0_0 = PAx * v12_0_0 + WPx * v12_0_1 + (VT)2.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v22_0_1 = PAx * v12_0_1 + WPx * v12_0_2 + (VT)2.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v22_0_2 = PAx * v12_0_2 + WPx * v12_0_3 + (VT)2.0 * oo2z * (v6_0_2 - rho_z * v6_0_3);
            const VT v23_0_0 = PAx * v13_0_0 + WPx * v13_0_1 + (VT)1.0 * oo2z * (v7_0_0 - rho_z * v7_0_1);
            const VT v23_0_1 = PAx * v13_0_1 + WPx * v13_0_2 + (VT)1.0 * oo2z * (v7_0_1 - rho_z * v7_0_2);
            const VT v23_0_2 = PAx * v13_0_2 + WPx * v13_0_3 + (VT)1.0 * oo2z * (v7_0_2 - rho_z * v7_0_3);
            const VT v24_0_0 = PAx * v15_0_0 + WPx * v15_0_1 + (VT)1.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v24_0_1 = PAx * v15_0_1 + WPx * v15_0_2 + (VT)1.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v24_0_2 = PAx * v15_0_2 + WPx * v15_0_3 + (VT)1.0 * oo2z * (v8_0_2 - rho_z * v8_0_3);
            const VT v25_0_0 = PAx * v14_0_0 + WPx * v14_0_1 + (VT)1.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v25_0_1 = PAx * v14_0_1 + WPx * v14_0_2 + (VT)1.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            const VT v25_0_2 = PAx * v14_0_2 + WPx * v14_0_3 + (VT)1.0 * oo2z * (v9_0_2 - rho_z * v9_0_3);
            const VT v26_0_0 = PAy * v13_0_0 + WPy * v13_0_1 + (VT)2.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v26_0_1 = PAy * v13_0_1 + WPy * v13_0_2 + (VT)2.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v26_0_2 = PAy * v13_0_2 + WPy * v13_0_3 + (VT)2.0 * oo2z * (v5_0_2 - rho_z * v5_0_3);
            const VT v27_0_0 = PAy * v15_0_0 + WPy * v15_0_1 + (VT)1.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v27_0_1 = PAy * v15_0_1 + WPy * v15_0_2 + (VT)1.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v27_0_2 = PAy * v15_0_2 + WPy * v15_0_3 + (VT)1.0 * oo2z * (v6_0_2 - rho_z * v6_0_3);
            const VT v28_0_0 = PAz * v15_0_0 + WPz * v15_0_1 + (VT)1.0 * oo2z * (v5_0_0 - rho_z * v5_0_1);
            const VT v28_0_1 = PAz * v15_0_1 + WPz * v15_0_2 + (VT)1.0 * oo2z * (v5_0_1 - rho_z * v5_0_2);
            const VT v28_0_2 = PAz * v15_0_2 + WPz * v15_0_3 + (VT)1.0 * oo2z * (v5_0_2 - rho_z * v5_0_3);
            const VT v29_0_0 = PAz * v14_0_0 + WPz * v14_0_1 + (VT)2.0 * oo2z * (v6_0_0 - rho_z * v6_0_1);
            const VT v29_0_1 = PAz * v14_0_1 + WPz * v14_0_2 + (VT)2.0 * oo2z * (v6_0_1 - rho_z * v6_0_2);
            const VT v29_0_2 = PAz * v14_0_2 + WPz * v14_0_3 + (VT)2.0 * oo2z * (v6_0_2 - rho_z * v6_0_3);
            const VT v30_0_0 = PAy * v16_0_0 + WPy * v16_0_1 + (VT)3.0 * oo2z * (v7_0_0 - rho_z * v7_0_1);
            const VT v30_0_1 = PAy * v16_0_1 + WPy * v16_0_2 + (VT)3.0 * oo2z * (v7_0_1 - rho_z * v7_0_2);
            const VT v30_0_2 = PAy * v16_0_2 + WPy * v16_0_3 + (VT)3.0 * oo2z * (v7_0_2 - rho_z * v7_0_3);
            const VT v31_0_0 = PAy * v17_0_0 + WPy * v17_0_1 + (VT)2.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v31_0_1 = PAy * v17_0_1 + WPy * v17_0_2 + (VT)2.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v31_0_2 = PAy * v17_0_2 + WPy * v17_0_3 + (VT)2.0 * oo2z * (v8_0_2 - rho_z * v8_0_3);
            const VT v32_0_0 = PAy * v18_0_0 + WPy * v18_0_1 + (VT)1.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v32_0_1 = PAy * v18_0_1 + WPy * v18_0_2 + (VT)1.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            const VT v32_0_2 = PAy * v18_0_2 + WPy * v18_0_3 + (VT)1.0 * oo2z * (v9_0_2 - rho_z * v9_0_3);
            const VT v33_0_0 = PAz * v18_0_0 + WPz * v18_0_1 + (VT)2.0 * oo2z * (v8_0_0 - rho_z * v8_0_1);
            const VT v33_0_1 = PAz * v18_0_1 + WPz * v18_0_2 + (VT)2.0 * oo2z * (v8_0_1 - rho_z * v8_0_2);
            const VT v33_0_2 = PAz * v18_0_2 + WPz * v18_0_3 + (VT)2.0 * oo2z * (v8_0_2 - rho_z * v8_0_3);
            const VT v34_0_0 = PAz * v19_0_0 + WPz * v19_0_1 + (VT)3.0 * oo2z * (v9_0_0 - rho_z * v9_0_1);
            const VT v34_0_1 = PAz * v19_0_1 + WPz * v19_0_2 + (VT)3.0 * oo2z * (v9_0_1 - rho_z * v9_0_2);
            const VT v34_0_2 = PAz * v19_0_2 + WPz * v19_0_3 + (VT)3.0 * oo2z * (v9_0_2 - rho_z * v9_0_3);
            const VT v1_1_1 = QCx * v1_0_1 + WQx * v1_0_2 + (VT)1.0 * oo2ze * v0_0_2;
            const VT v2_1_1 = QCx * v2_0_1 + WQx * v2_0_2;
            const VT v3_1_1 = QCx * v3_0_1 + WQx * v3_0_2;
            const VT v4_1_0 = QCx * v4_0_0 + WQx * v4_0_1 + (VT)2.0 * oo2ze * v1_0_1;
            const VT v4_1_1 = QCx * v4_0_1 + WQx * v4_0_2 + (VT)2.0 * oo2ze * v1_0_2;
            const VT v5_1_0 = QCx * v5_0_0 + WQx * v5_0_1 + (VT)1.0 * oo2ze * v2_0_1;
            const VT v5_1_1 = QCx * v5_0_1 + WQx * v5_0_2 + (VT)1.0 * oo2ze * v2_0_2;
            const VT v6_1_0 = QCx * v6_0_0 + WQx * v6_0_1 + (VT)1.0 * oo2ze * v3_0_1;
            const VT v6_1_1 = QCx * v6_0_1 + WQx * v6_0_2 + (VT)1.0 * oo2ze * v3_0_2;
            const VT v7_1_0 = QCx * v7_0_0 + WQx * v7_0_1;
            const VT v7_1_1 = QCx * v7_0_1 + WQx * v7_0_2;
            const VT v8_1_0 = QCx * v8_0_0 + WQx * v8_0_1;
            const VT v8_1_1 = QCx * v8_0_1 + WQx * v8_0_2;
            const VT v9_1_0 = QCx * v9_0_0 + WQx * v9_0_1;
            const VT v9_1_1 = QCx * v9_0_1 + WQx * v9_0_2;
            const VT v10_1_0 = QCx * v10_0_0 + WQx * v10_0_1 + (VT)3.0 * oo2ze * v4_0_1;
            const VT v10_1_1 = QCx * v10_0_1 + WQx * v10_0_2 + (VT)3.0 * oo2ze * v4_0_2;
            const VT v11_1_0 = QCx * v11_0_0 + WQx * v11_0_1 + (VT)2.0 * oo2ze * v5_0_1;
            const VT v11_1_1 = QCx * v11_0_1 + WQx * v11_0_2 + (VT)2.0 * oo2ze * v5_0_2;
            const VT v12_1_0 = QCx * v12_0_0 + WQx * v12_0_1 + (VT)2.0 * oo2ze * v6_0_1;
            const VT v12_1_1 = QCx * v12_0_1 + WQx * v12_0_2 + (VT)2.0 * oo2ze * v6_0_2;
            const VT v13_1_0 = QCx * v13_0_0 + WQx * v13_0_1 + (VT)1.0 * oo2ze * v7_0_1;
            const VT v13_1_1 = QCx * v13_0_1 + WQx * v13_0_2 + (VT)1.0 * oo2ze * v7_0_2;
            const VT v14_1_0 = QCx * v14_0_0 + WQx * v14_0_1 + (VT)1.0 * oo2ze * v9_0_1;
            const VT v14_1_1 = QCx * v14_0_1 + WQx * v14_0_2 + (VT)1.0 * oo2ze * v9_0_2;
            const VT v15_1_0 = QCx * v15_0_0 + WQx * v15_0_1 + (VT)1.0 * oo2ze * v8_0_1;
            const VT v15_1_1 = QCx * v15_0_1 + WQx * v15_0_2 + (VT)1.0 * oo2ze * v8_0_2;
            const VT v16_1_0 = QCx * v16_0_0 + WQx * v16_0_1;
            const VT v16_1_1 = QCx * v16_0_1 + WQx * v16_0_2;
            const VT v17_1_0 = QCx * v17_0_0 + WQx * v17_0_1;
            const VT v17_1_1 = QCx * v17_0_1 + WQx * v17_0_2;
            const VT v18_1_0 = QCx * v18_0_0 + WQx * v18_0_1;
            const VT v18_1_1 = QCx * v18_0_1 + WQx * v18_0_2;
            const VT v19_1_0 = QCx * v19_0_0 + WQx * v19_0_1;
            const VT v19_1_1 = QCx * v19_0_1 + WQx * v19_0_2;
            const VT v20_1_0 = QCx * v20_0_0 + WQx * v20_0_1 + (VT)4.0 * oo2ze * v10_0_1;
            const VT v20_1_1 = QCx * v20_0_1 + WQx * v20_0_2 + (VT)4.0 * oo2ze * v10_0_2;
            const VT v21_1_0 = QCx * v21_0_0 + WQx * v21_0_1 + (VT)3.0 * oo2ze * v11_0_1;
            const VT v21_1_1 = QCx * v21_0_1 + WQx * v21_0_2 + (VT)3.0 * oo2ze * v11_0_2;
            const VT v22_1_0 = QCx * v22_0_0 + WQx * v22_0_1 + (VT)3.0 * oo2ze * v12_0_1;
            const VT v22_1_1 = QCx * v22_0_1 + WQx * v22_0_2 + (VT)3.0 * oo2ze * v12_0_2;
            const VT v23_1_0 = QCx * v23_0_0 + WQx * v23_0_1 + (VT)2.0 * oo2ze * v13_0_1;
            const VT v23_1_1 = QCx * v23_0_1 + WQx * v23_0_2 + (VT)2.0 * oo2ze * v13_0_2;
            const VT v24_1_0 = QCx * v24_0_0 + WQx * v24_0_1 + (VT)2.0 * oo2ze * v15_0_1;
            const VT v24_1_1 = QCx * v24_0_1 + WQx * v24_0_2 + (VT)2.0 * oo2ze * v15_0_2;
            const VT v25_1_0 = QCx * v25_0_0 + WQx * v25_0_1 + (VT)2.0 * oo2ze * v14_0_1;
            const VT v25_1_1 = QCx * v25_0_1 + WQx * v25_0_2 + (VT)2.0 * oo2ze * v14_0_2;
            const VT v26_1_0 = QCx * v26_0_0 + WQx * v26_0_1 + (VT)1.0 * oo2ze * v16_0_1;
            const VT v26_1_1 = QCx * v26_0_1 + WQx * v26_0_2 + (VT)1.0 * oo2ze * v16_0_2;
            const VT v27_1_0 = QCx * v27_0_0 + WQx * v27_0_1 + (VT)1.0 * oo2ze * v17_0_1;
            const VT v27_1_1 = QCx * v27_0_1 + WQx * v27_0_2 + (VT)1.0 * oo2ze * v17_0_2;
            const VT v28_1_0 = QCx * v28_0_0 + WQx * v28_0_1 + (VT)1.0 * oo2ze * v18_0_1;
            const VT v28_1_1 = QCx * v28_0_1 + WQx * v28_0_2 + (VT)1.0 * oo2ze * v18_0_2;
            const VT v29_1_0 = QCx * v29_0_0 + WQx * v29_0_1 + (VT)1.0 * oo2ze * v19_0_1;
            const VT v29_1_1 = QCx * v29_0_1 + WQx * v29_0_2 + (VT)1.0 * oo2ze * v19_0_2;
            const VT v30_1_0 = QCx * v30_0_0 + WQx * v30_0_1;
            const VT v30_1_1 = QCx * v30_0_1 + WQx * v30_0_2;
            const VT v31_1_0 = QCx * v31_0_0 + WQx * v31_0_1;
            const VT v31_1_1 = QCx * v31_0_1 + WQx * v31_0_2;
            const VT v32_1_0 = QCx * v32_0_0 + WQx * v32_0_1;
            const VT v32_1_1 = QCx * v32_0_1 + WQx * v32_0_2;
            const VT v33_1_0 = QCx * v33_0_0 + WQx * v33_0_1;
            const VT v33_1_1 = QCx * v33_0_1 + WQx * v33_0_2;
            const VT v34_1_0 = QCx * v34_0_0 + WQx * v34_0_1;
            const VT v34_1_1 = QCx * v34_0_1 + WQx * v34_0_2;
            const VT v1_2_1 = QCy * v1_0_1 + WQy * v1_0_2;
            const VT v2_2_1 = QCy * v2_0_1 + WQy * v2_0_2 + (VT)1.0 * oo2ze * v0_0_2;
            const VT v3_2_1 = QCy * v3_0_1 + WQy * v3_0_2;
            const VT v4_2_0 = QCy * v4_0_0 + WQy * v4_0_1;
            const VT v4_2_1 = QCy * v4_0_1 + WQy * v4_0_2;
            const VT v5_2_0 = QCy * v5_0_0 + WQy * v5_0_1 + (VT)1.0 * oo2ze * v1_0_1;
            const VT v5_2_1 = QCy * v5_0_1 + WQy * v5_0_2 + (VT)1.0 * oo2ze * v1_0_2;
            const VT v6_2_0 = QCy * v6_0_0 + WQy * v6_0_1;
            const VT v6_2_1 = QCy * v6_0_1 + WQy * v6_0_2;
            const VT v7_2_0 = QCy * v7_0_0 + WQy * v7_0_1 + (VT)2.0 * oo2ze * v2_0_1;
            const VT v7_2_1 = QCy * v7_0_1 + WQy * v7_0_2 + (VT)2.0 * oo2ze * v2_0_2;
            const VT v8_2_0 = QCy * v8_0_0 + WQy * v8_0_1 + (VT)1.0 * oo2ze * v3_0_1;
            const VT v8_2_1 = QCy * v8_0_1 + WQy * v8_0_2 + (VT)1.0 * oo2ze * v3_0_2;
            const VT v9_2_0 = QCy * v9_0_0 + WQy * v9_0_1;
            const VT v9_2_1 = QCy * v9_0_1 + WQy * v9_0_2;
            const VT v10_2_0 = QCy * v10_0_0 + WQy * v10_0_1;
            const VT v10_2_1 = QCy * v10_0_1 + WQy * v10_0_2;
            const VT v11_2_0 = QCy * v11_0_0 + WQy * v11_0_1 + (VT)1.0 * oo2ze * v4_0_1;
            const VT v11_2_1 = QCy * v11_0_1 + WQy * v11_0_2 + (VT)1.0 * oo2ze * v4_0_2;
            const VT v12_2_0 = QCy * v12_0_0 + WQy * v12_0_1;
            const VT v12_2_1 = QCy * v12_0_1 + WQy * v12_0_2;
            const VT v13_2_0 = QCy * v13_0_0 + WQy * v13_0_1 + (VT)2.0 * oo2ze * v5_0_1;
            const VT v13_2_1 = QCy * v13_0_1 + WQy * v13_0_2 + (VT)2.0 * oo2ze * v5_0_2;
            const VT v14_2_0 = QCy * v14_0_0 + WQy * v14_0_1;
            const VT v14_2_1 = QCy * v14_0_1 + WQy * v14_0_2;
            const VT v15_2_0 = QCy * v15_0_0 + WQy * v15_0_1 + (VT)1.0 * oo2ze * v6_0_1;
            const VT v15_2_1 = QCy * v15_0_1 + WQy * v15_0_2 + (VT)1.0 * oo2ze * v6_0_2;
            const VT v16_2_0 = QCy * v16_0_0 + WQy * v16_0_1 + (VT)3.0 * oo2ze * v7_0_1;
            const VT v16_2_1 = QCy * v16_0_1 + WQy * v16_0_2 + (VT)3.0 * oo2ze * v7_0_2;
            const VT v17_2_0 = QCy * v17_0_0 + WQy * v17_0_1 + (VT)2.0 * oo2ze * v8_0_1;
            const VT v17_2_1 = QCy * v17_0_1 + WQy * v17_0_2 + (VT)2.0 * oo2ze * v8_0_2;
            const VT v18_2_0 = QCy * v18_0_0 + WQy * v18_0_1 + (VT)1.0 * oo2ze * v9_0_1;
            const VT v18_2_1 = QCy * v18_0_1 + WQy * v18_0_2 + (VT)1.0 * oo2ze * v9_0_2;
            const VT v19_2_0 = QCy * v19_0_0 + WQy * v19_0_1;
            const VT v19_2_1 = QCy * v19_0_1 + WQy * v19_0_2;
            const VT v20_2_0 = QCy * v20_0_0 + WQy * v20_0_1;
            const VT v20_2_1 = QCy * v20_0_1 + WQy * v20_0_2;
            const VT v21_2_0 = QCy * v21_0_0 + WQy * v21_0_1 + (VT)1.0 * oo2ze * v10_0_1;
            const VT v21_2_1 = QCy * v21_0_1 + WQy * v21_0_2 + (VT)1.0 * oo2ze * v10_0_2;
            const VT v22_2_0 = QCy * v22_0_0 + WQy * v22_0_1;
            const VT v22_2_1 = QCy * v22_0_1 + WQy * v22_0_2;
            const VT v23_2_0 = QCy * v23_0_0 + WQy * v23_0_1 + (VT)2.0 * oo2ze * v11_0_1;
            const VT v23_2_1 = QCy * v23_0_1 + WQy * v23_0_2 + (VT)2.0 * oo2ze * v11_0_2;
            const VT v24_2_0 = QCy * v24_0_0 + WQy * v24_0_1 + (VT)1.0 * oo2ze * v12_0_1;
            const VT v24_2_1 = QCy * v24_0_1 + WQy * v24_0_2 + (VT)1.0 * oo2ze * v12_0_2;
            const VT v25_2_0 = QCy * v25_0_0 + WQy * v25_0_1;
            const VT v25_2_1 = QCy * v25_0_1 + WQy * v25_0_2;
            const VT v26_2_0 = QCy * v26_0_0 + WQy * v26_0_1 + (VT)3.0 * oo2ze * v13_0_1;
            const VT v26_2_1 = QCy * v26_0_1 + WQy * v26_0_2 + (VT)3.0 * oo2ze * v13_0_2;
            const VT v27_2_0 = QCy * v27_0_0 + WQy * v27_0_1 + (VT)2.0 * oo2ze * v15_0_1;
            const VT v27_2_1 = QCy * v27_0_1 + WQy * v27_0_2 + (VT)2.0 * oo2ze * v15_0_2;
            const VT v28_2_0 = QCy * v28_0_0 + WQy * v28_0_1 + (VT)1.0 * oo2ze * v14_0_1;
            const VT v28_2_1 = QCy * v28_0_1 + WQy * v28_0_2 + (VT)1.0 * oo2ze * v14_0_2;
            const VT v29_2_0 = QCy * v29_0_0 + WQy * v29_0_1;
            const VT v29_2_1 = QCy * v29_0_1 + WQy * v29_0_2;
            const VT v30_2_0 = QCy * v30_0_0 + WQy * v30_0_1 + (VT)4.0 * oo2ze * v16_0_1;
            const VT v30_2_1 = QCy * v30_0_1 + WQy * v30_0_2 + (VT)4.0 * oo2ze * v16_0_2;
            const VT v31_2_0 = QCy * v31_0_0 + WQy * v31_0_1 + (VT)3.0 * oo2ze * v17_0_1;
            const VT v31_2_1 = QCy * v31_0_1 + WQy * v31_0_2 + (VT)3.0 * oo2ze * v17_0_2;
            const VT v32_2_0 = QCy * v32_0_0 + WQy * v32_0_1 + (VT)2.0 * oo2ze * v18_0_1;
            const VT v32_2_1 = QCy * v32_0_1 + WQy * v32_0_2 + (VT)2.0 * oo2ze * v18_0_2;
            const VT v33_2_0 = QCy * v33_0_0 + WQy * v33_0_1 + (VT)1.0 * oo2ze * v19_0_1;
            const VT v33_2_1 = QCy * v33_0_1 + WQy * v33_0_2 + (VT)1.0 * oo2ze * v19_0_2;
            const VT v34_2_0 = QCy * v34_0_0 + WQy * v34_0_1;
            const VT v34_2_1 = QCy * v34_0_1 + WQy * v34_0_2;
            const VT v1_3_1 = QCz * v1_0_1 + WQz * v1_0_2;
            const VT v2_3_1 = QCz * v2_0_1 + WQz * v2_0_2;
            const VT v3_3_1 = QCz * v3_0_1 + WQz * v3_0_2 + (VT)1.0 * oo2ze * v0_0_2;
            const VT v4_3_0 = QCz * v4_0_0 + WQz * v4_0_1;
            const VT v4_3_1 = QCz * v4_0_1 + WQz * v4_0_2;
            const VT v5_3_0 = QCz * v5_0_0 + WQz * v5_0_1;
            const VT v5_3_1 = QCz * v5_0_1 + WQz * v5_0_2;
            const VT v6_3_0 = QCz * v6_0_0 + WQz * v6_0_1 + (VT)1.0 * oo2ze * v1_0_1;
            const VT v6_3_1 = QCz * v6_0_1 + WQz * v6_0_2 + (VT)1.0 * oo2ze * v1_0_2;
            const VT v7_3_0 = QCz * v7_0_0 + WQz * v7_0_1;
            const VT v7_3_1 = QCz * v7_0_1 + WQz * v7_0_2;
            const VT v8_3_0 = QCz * v8_0_0 + WQz * v8_0_1 + (VT)1.0 * oo2ze * v2_0_1;
            const VT v8_3_1 = QCz * v8_0_1 + WQz * v8_0_2 + (VT)1.0 * oo2ze * v2_0_2;
            const VT v9_3_0 = QCz * v9_0_0 + WQz * v9_0_1 + (VT)2.0 * oo2ze * v3_0_1;
            const VT v9_3_1 = QCz * v9_0_1 + WQz * v9_0_2 + (VT)2.0 * oo2ze * v3_0_2;
            const VT v10_3_0 = QCz * v10_0_0 + WQz * v10_0_1;
            const VT v10_3_1 = QCz * v10_0_1 + WQz * v10_0_2;
            const VT v11_3_0 = QCz * v11_0_0 + WQz * v11_0_1;
            const VT v11_3_1 = QCz * v11_0_1 + WQz * v11_0_2;
            const VT v12_3_0 = QCz * v12_0_0 + WQz * v12_0_1 + (VT)1.0 * oo2ze * v4_0_1;
            const VT v12_3_1 = QCz * v12_0_1 + WQz * v12_0_2 + (VT)1.0 * oo2ze * v4_0_2;
            const VT v13_3_0 = QCz * v13_0_0 + WQz * v13_0_1;
            const VT v13_3_1 = QCz * v13_0_1 + WQz * v13_0_2;
            const VT v14_3_0 = QCz * v14_0_0 + WQz * v14_0_1 + (VT)2.0 * oo2ze * v6_0_1;
            const VT v14_3_1 = QCz * v14_0_1 + WQz * v14_0_2 + (VT)2.0 * oo2ze * v6_0_2;
            const VT v15_3_0 = QCz * v15_0_0 + WQz * v15_0_1 + (VT)1.0 * oo2ze * v5_0_1;
            const VT v15_3_1 = QCz * v15_0_1 + WQz * v15_0_2 + (VT)1.0 * oo2ze * v5_0_2;
            const VT v16_3_0 = QCz * v16_0_0 + WQz * v16_0_1;
            const VT v16_3_1 = QCz * v16_0_1 + WQz * v16_0_2;
            const VT v17_3_0 = QCz * v17_0_0 + WQz * v17_0_1 + (VT)1.0 * oo2ze * v7_0_1;
            const VT v17_3_1 = QCz * v17_0_1 + WQz * v17_0_2 + (VT)1.0 * oo2ze * v7_0_2;
            const VT v18_3_0 = QCz * v18_0_0 + WQz * v18_0_1 + (VT)2.0 * oo2ze * v8_0_1;
            const VT v18_3_1 = QCz * v18_0_1 + WQz * v18_0_2 + (VT)2.0 * oo2ze * v8_0_2;
            const VT v19_3_0 = QCz * v19_0_0 + WQz * v19_0_1 + (VT)3.0 * oo2ze * v9_0_1;
            const VT v19_3_1 = QCz * v19_0_1 + WQz * v19_0_2 + (VT)3.0 * oo2ze * v9_0_2;
            const VT v20_3_0 = QCz * v20_0_0 + WQz * v20_0_1;
            const VT v20_3_1 = QCz * v20_0_1 + WQz * v20_0_2;
            const VT v21_3_0 = QCz * v21_0_0 + WQz * v21_0_1;
            const VT v21_3_1 = QCz * v21_0_1 + WQz * v21_0_2;
            const VT v22_3_0 = QCz * v22_0_0 + WQz * v22_0_1 + (VT)1.0 * oo2ze * v10_0_1;
            const VT v22_3_1 = QCz * v22_0_1 + WQz * v22_0_2 + (VT)1.0 * oo2ze * v10_0_2;
            const VT v23_3_0 = QCz * v23_0_0 + WQz * v23_0_1;
            const VT v23_3_1 = QCz * v23_0_1 + WQz * v23_0_2;
            const VT v24_3_0 = QCz * v24_0_0 + WQz * v24_0_1 + (VT)1.0 * oo2ze * v11_0_1;
            const VT v24_3_1 = QCz * v24_0_1 + WQz * v24_0_2 + (VT)1.0 * oo2ze * v11_0_2;
            const VT v25_3_0 = QCz * v25_0_0 + WQz * v25_0_1 + (VT)2.0 * oo2ze * v12_0_1;
            const VT v25_3_1 = QCz * v25_0_1 + WQz * v25_0_2 + (VT)2.0 * oo2ze * v12_0_2;
            const VT v26_3_0 = QCz * v26_0_0 + WQz * v26_0_1;
            const VT v26_3_1 = QCz * v26_0_1 + WQz * v26_0_2;
            const VT v27_3_0 = QCz * v27_0_0 + WQz * v27_0_1 + (VT)1.0 * oo2ze * v13_0_1;
            const VT v27_3_1 = QCz * v27_0_1 + WQz * v27_0_2 + (VT)1.0 * oo2ze * v13_0_2;
            const VT v28_3_0 = QCz * v28_0_0 + WQz * v28_0_1 + (VT)2.0 * oo2ze * v15_0_1;
            const VT v28_3_1 = QCz * v28_0_1 + WQz * v28_0_2 + (VT)2.0 * oo2ze * v15_0_2;
            const VT v29_3_0 = QCz * v29_0_0 + WQz * v29_0_1 + (VT)3.0 * oo2ze * v14_0_1;
            const VT v29_3_1 = QCz * v29_0_1 + WQz * v29_0_2 + (VT)3.0 * oo2ze * v14_0_2;
            const VT v30_3_0 = QCz * v30_0_0 + WQz * v30_0_1;
            const VT v30_3_1 = QCz * v30_0_1 + WQz * v30_0_2;
            const VT v31_3_0 = QCz * v31_0_0 + WQz * v31_0_1 + (VT)1.0 * oo2ze * v16_0_1;
            const VT v31_3_1 = QCz * v31_0_1 + WQz * v31_0_2 + (VT)1.0 * oo2ze * v16_0_2;
            const VT v32_3_0 = QCz * v32_0_0 + WQz * v32_0_1 + (VT)2.0 * oo2ze * v17_0_1;
            const VT v32_3_1 = QCz * v32_0_1 + WQz * v32_0_2 + (VT)2.0 * oo2ze * v17_0_2;
            const VT v33_3_0 = QCz * v33_0_0 + WQz * v33_0_1 + (VT)3.0 * oo2ze * v18_0_1;
            const VT v33_3_1 = QCz * v33_0_1 + WQz * v33_0_2 + (VT)3.0 * oo2ze * v18_0_2;
            const VT v34_3_0 = QCz * v34_0_0 + WQz * v34_0_1 + (VT)4.0 * oo2ze * v19_0_1;
            const VT v34_3_1 = QCz * v34_0_1 + WQz * v34_0_2 + (VT)4.0 * oo2ze * v19_0_2;
            if constexpr (sizeof(VT) == 8) {
                acc[0] = fma(QCx, v4_1_0, fma(WQx, v4_1_1, fma(2.0 * oo2ze, v1_1_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[0]))));
                acc[1] = fma(QCx, v4_2_0, fma(WQx, v4_2_1, fma(2.0 * oo2ze, v1_2_1, acc[1])));
                acc[2] = fma(QCx, v4_3_0, fma(WQx, v4_3_1, fma(2.0 * oo2ze, v1_3_1, acc[2])));
                acc[3] = fma(QCy, v4_2_0, fma(WQy, v4_2_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[3])));
                acc[4] = fma(QCy, v4_3_0, fma(WQy, v4_3_1, acc[4]));
                acc[5] = fma(QCz, v4_3_0, fma(WQz, v4_3_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[5])));
                acc[6] = fma(QCx, v5_1_0, fma(WQx, v5_1_1, fma(1.0 * oo2ze, v2_1_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[6]))));
                acc[7] = fma(QCx, v5_2_0, fma(WQx, v5_2_1, fma(1.0 * oo2ze, v2_2_1, acc[7])));
                acc[8] = fma(QCx, v5_3_0, fma(WQx, v5_3_1, fma(1.0 * oo2ze, v2_3_1, acc[8])));
                acc[9] = fma(QCy, v5_2_0, fma(WQy, v5_2_1, fma(1.0 * oo2ze, v1_2_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[9]))));
                acc[10] = fma(QCy, v5_3_0, fma(WQy, v5_3_1, fma(1.0 * oo2ze, v1_3_1, acc[10])));
                acc[11] = fma(QCz, v5_3_0, fma(WQz, v5_3_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[11])));
                acc[12] = fma(QCx, v6_1_0, fma(WQx, v6_1_1, fma(1.0 * oo2ze, v3_1_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[12]))));
                acc[13] = fma(QCx, v6_2_0, fma(WQx, v6_2_1, fma(1.0 * oo2ze, v3_2_1, acc[13])));
                acc[14] = fma(QCx, v6_3_0, fma(WQx, v6_3_1, fma(1.0 * oo2ze, v3_3_1, acc[14])));
                acc[15] = fma(QCy, v6_2_0, fma(WQy, v6_2_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[15])));
                acc[16] = fma(QCy, v6_3_0, fma(WQy, v6_3_1, acc[16]));
                acc[17] = fma(QCz, v6_3_0, fma(WQz, v6_3_1, fma(1.0 * oo2ze, v1_3_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[17]))));
                acc[18] = fma(QCx, v7_1_0, fma(WQx, v7_1_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[18])));
                acc[19] = fma(QCx, v7_2_0, fma(WQx, v7_2_1, acc[19]));
                acc[20] = fma(QCx, v7_3_0, fma(WQx, v7_3_1, acc[20]));
                acc[21] = fma(QCy, v7_2_0, fma(WQy, v7_2_1, fma(2.0 * oo2ze, v2_2_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[21]))));
                acc[22] = fma(QCy, v7_3_0, fma(WQy, v7_3_1, fma(2.0 * oo2ze, v2_3_1, acc[22])));
                acc[23] = fma(QCz, v7_3_0, fma(WQz, v7_3_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[23])));
                acc[24] = fma(QCx, v8_1_0, fma(WQx, v8_1_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[24])));
                acc[25] = fma(QCx, v8_2_0, fma(WQx, v8_2_1, acc[25]));
                acc[26] = fma(QCx, v8_3_0, fma(WQx, v8_3_1, acc[26]));
                acc[27] = fma(QCy, v8_2_0, fma(WQy, v8_2_1, fma(1.0 * oo2ze, v3_2_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[27]))));
                acc[28] = fma(QCy, v8_3_0, fma(WQy, v8_3_1, fma(1.0 * oo2ze, v3_3_1, acc[28])));
                acc[29] = fma(QCz, v8_3_0, fma(WQz, v8_3_1, fma(1.0 * oo2ze, v2_3_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[29]))));
                acc[30] = fma(QCx, v9_1_0, fma(WQx, v9_1_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[30])));
                acc[31] = fma(QCx, v9_2_0, fma(WQx, v9_2_1, acc[31]));
                acc[32] = fma(QCx, v9_3_0, fma(WQx, v9_3_1, acc[32]));
                acc[33] = fma(QCy, v9_2_0, fma(WQy, v9_2_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[33])));
                acc[34] = fma(QCy, v9_3_0, fma(WQy, v9_3_1, acc[34]));
                acc[35] = fma(QCz, v9_3_0, fma(WQz, v9_3_1, fma(2.0 * oo2ze, v3_3_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[35]))));
                acc[36] = fma(QCx, v10_1_0, fma(WQx, v10_1_1, fma(3.0 * oo2ze, v4_1_1, fma(1.0 * oo2e, (v10_0_0 - rho_e * v10_0_1), acc[36]))));
                acc[37] = fma(QCx, v10_2_0, fma(WQx, v10_2_1, fma(3.0 * oo2ze, v4_2_1, acc[37])));
                acc[38] = fma(QCx, v10_3_0, fma(WQx, v10_3_1, fma(3.0 * oo2ze, v4_3_1, acc[38])));
                acc[39] = fma(QCy, v10_2_0, fma(WQy, v10_2_1, fma(1.0 * oo2e, (v10_0_0 - rho_e * v10_0_1), acc[39])));
                acc[40] = fma(QCy, v10_3_0, fma(WQy, v10_3_1, acc[40]));
                acc[41] = fma(QCz, v10_3_0, fma(WQz, v10_3_1, fma(1.0 * oo2e, (v10_0_0 - rho_e * v10_0_1), acc[41])));
                acc[42] = fma(QCx, v11_1_0, fma(WQx, v11_1_1, fma(2.0 * oo2ze, v5_1_1, fma(1.0 * oo2e, (v11_0_0 - rho_e * v11_0_1), acc[42]))));
                acc[43] = fma(QCx, v11_2_0, fma(WQx, v11_2_1, fma(2.0 * oo2ze, v5_2_1, acc[43])));
                acc[44] = fma(QCx, v11_3_0, fma(WQx, v11_3_1, fma(2.0 * oo2ze, v5_3_1, acc[44])));
                acc[45] = fma(QCy, v11_2_0, fma(WQy, v11_2_1, fma(1.0 * oo2ze, v4_2_1, fma(1.0 * oo2e, (v11_0_0 - rho_e * v11_0_1), acc[45]))));
                acc[46] = fma(QCy, v11_3_0, fma(WQy, v11_3_1, fma(1.0 * oo2ze, v4_3_1, acc[46])));
                acc[47] = fma(QCz, v11_3_0, fma(WQz, v11_3_1, fma(1.0 * oo2e, (v11_0_0 - rho_e * v11_0_1), acc[47])));
                acc[48] = fma(QCx, v12_1_0, fma(WQx, v12_1_1, fma(2.0 * oo2ze, v6_1_1, fma(1.0 * oo2e, (v12_0_0 - rho_e * v12_0_1), acc[48]))));
                acc[49] = fma(QCx, v12_2_0, fma(WQx, v12_2_1, fma(2.0 * oo2ze, v6_2_1, acc[49])));
                acc[50] = fma(QCx, v12_3_0, fma(WQx, v12_3_1, fma(2.0 * oo2ze, v6_3_1, acc[50])));
                acc[51] = fma(QCy, v12_2_0, fma(WQy, v12_2_1, fma(1.0 * oo2e, (v12_0_0 - rho_e * v12_0_1), acc[51])));
                acc[52] = fma(QCy, v12_3_0, fma(WQy, v12_3_1, acc[52]));
                acc[53] = fma(QCz, v12_3_0, fma(WQz, v12_3_1, fma(1.0 * oo2ze, v4_3_1, fma(1.0 * oo2e, (v12_0_0 - rho_e * v12_0_1), acc[53]))));
                acc[54] = fma(QCx, v13_1_0, fma(WQx, v13_1_1, fma(1.0 * oo2ze, v7_1_1, fma(1.0 * oo2e, (v13_0_0 - rho_e * v13_0_1), acc[54]))));
                acc[55] = fma(QCx, v13_2_0, fma(WQx, v13_2_1, fma(1.0 * oo2ze, v7_2_1, acc[55])));
                acc[56] = fma(QCx, v13_3_0, fma(WQx, v13_3_1, fma(1.0 * oo2ze, v7_3_1, acc[56])));
                acc[57] = fma(QCy, v13_2_0, fma(WQy, v13_2_1, fma(2.0 * oo2ze, v5_2_1, fma(1.0 * oo2e, (v13_0_0 - rho_e * v13_0_1), acc[57]))));
                acc[58] = fma(QCy, v13_3_0, fma(WQy, v13_3_1, fma(2.0 * oo2ze, v5_3_1, acc[58])));
                acc[59] = fma(QCz, v13_3_0, fma(WQz, v13_3_1, fma(1.0 * oo2e, (v13_0_0 - rho_e * v13_0_1), acc[59])));
                acc[60] = fma(QCx, v14_1_0, fma(WQx, v14_1_1, fma(1.0 * oo2ze, v9_1_1, fma(1.0 * oo2e, (v14_0_0 - rho_e * v14_0_1), acc[60]))));
                acc[61] = fma(QCx, v14_2_0, fma(WQx, v14_2_1, fma(1.0 * oo2ze, v9_2_1, acc[61])));
                acc[62] = fma(QCx, v14_3_0, fma(WQx, v14_3_1, fma(1.0 * oo2ze, v9_3_1, acc[62])));
                acc[63] = fma(QCy, v14_2_0, fma(WQy, v14_2_1, fma(1.0 * oo2e, (v14_0_0 - rho_e * v14_0_1), acc[63])));
                acc[64] = fma(QCy, v14_3_0, fma(WQy, v14_3_1, acc[64]));
                acc[65] = fma(QCz, v14_3_0, fma(WQz, v14_3_1, fma(2.0 * oo2ze, v6_3_1, fma(1.0 * oo2e, (v14_0_0 - rho_e * v14_0_1), acc[65]))));
                acc[66] = fma(QCx, v15_1_0, fma(WQx, v15_1_1, fma(1.0 * oo2ze, v8_1_1, fma(1.0 * oo2e, (v15_0_0 - rho_e * v15_0_1), acc[66]))));
                acc[67] = fma(QCx, v15_2_0, fma(WQx, v15_2_1, fma(1.0 * oo2ze, v8_2_1, acc[67])));
                acc[68] = fma(QCx, v15_3_0, fma(WQx, v15_3_1, fma(1.0 * oo2ze, v8_3_1, acc[68])));
                acc[69] = fma(QCy, v15_2_0, fma(WQy, v15_2_1, fma(1.0 * oo2ze, v6_2_1, fma(1.0 * oo2e, (v15_0_0 - rho_e * v15_0_1), acc[69]))));
                acc[70] = fma(QCy, v15_3_0, fma(WQy, v15_3_1, fma(1.0 * oo2ze, v6_3_1, acc[70])));
                acc[71] = fma(QCz, v15_3_0, fma(WQz, v15_3_1, fma(1.0 * oo2ze, v5_3_1, fma(1.0 * oo2e, (v15_0_0 - rho_e * v15_0_1), acc[71]))));
                acc[72] = fma(QCx, v16_1_0, fma(WQx, v16_1_1, fma(1.0 * oo2e, (v16_0_0 - rho_e * v16_0_1), acc[72])));
                acc[73] = fma(QCx, v16_2_0, fma(WQx, v16_2_1, acc[73]));
                acc[74] = fma(QCx, v16_3_0, fma(WQx, v16_3_1, acc[74]));
                acc[75] = fma(QCy, v16_2_0, fma(WQy, v16_2_1, fma(3.0 * oo2ze, v7_2_1, fma(1.0 * oo2e, (v16_0_0 - rho_e * v16_0_1), acc[75]))));
                acc[76] = fma(QCy, v16_3_0, fma(WQy, v16_3_1, fma(3.0 * oo2ze, v7_3_1, acc[76])));
                acc[77] = fma(QCz, v16_3_0, fma(WQz, v16_3_1, fma(1.0 * oo2e, (v16_0_0 - rho_e * v16_0_1), acc[77])));
                acc[78] = fma(QCx, v17_1_0, fma(WQx, v17_1_1, fma(1.0 * oo2e, (v17_0_0 - rho_e * v17_0_1), acc[78])));
                acc[79] = fma(QCx, v17_2_0, fma(WQx, v17_2_1, acc[79]));
                acc[80] = fma(QCx, v17_3_0, fma(WQx, v17_3_1, acc[80]));
                acc[81] = fma(QCy, v17_2_0, fma(WQy, v17_2_1, fma(2.0 * oo2ze, v8_2_1, fma(1.0 * oo2e, (v17_0_0 - rho_e * v17_0_1), acc[81]))));
                acc[82] = fma(QCy, v17_3_0, fma(WQy, v17_3_1, fma(2.0 * oo2ze, v8_3_1, acc[82])));
                acc[83] = fma(QCz, v17_3_0, fma(WQz, v17_3_1, fma(1.0 * oo2ze, v7_3_1, fma(1.0 * oo2e, (v17_0_0 - rho_e * v17_0_1), acc[83]))));
                acc[84] = fma(QCx, v18_1_0, fma(WQx, v18_1_1, fma(1.0 * oo2e, (v18_0_0 - rho_e * v18_0_1), acc[84])));
                acc[85] = fma(QCx, v18_2_0, fma(WQx, v18_2_1, acc[85]));
                acc[86] = fma(QCx, v18_3_0, fma(WQx, v18_3_1, acc[86]));
                acc[87] = fma(QCy, v18_2_0, fma(WQy, v18_2_1, fma(1.0 * oo2ze, v9_2_1, fma(1.0 * oo2e, (v18_0_0 - rho_e * v18_0_1), acc[87]))));
                acc[88] = fma(QCy, v18_3_0, fma(WQy, v18_3_1, fma(1.0 * oo2ze, v9_3_1, acc[88])));
                acc[89] = fma(QCz, v18_3_0, fma(WQz, v18_3_1, fma(2.0 * oo2ze, v8_3_1, fma(1.0 * oo2e, (v18_0_0 - rho_e * v18_0_1), acc[89]))));
                acc[90] = fma(QCx, v19_1_0, fma(WQx, v19_1_1, fma(1.0 * oo2e, (v19_0_0 - rho_e * v19_0_1), acc[90])));
                acc[91] = fma(QCx, v19_2_0, fma(WQx, v19_2_1, acc[91]));
                acc[92] = fma(QCx, v19_3_0, fma(WQx, v19_3_1, acc[92]));
                acc[93] = fma(QCy, v19_2_0, fma(WQy, v19_2_1, fma(1.0 * oo2e, (v19_0_0 - rho_e * v19_0_1), acc[93])));
                acc[94] = fma(QCy, v19_3_0, fma(WQy, v19_3_1, acc[94]));
                acc[95] = fma(QCz, v19_3_0, fma(WQz, v19_3_1, fma(3.0 * oo2ze, v9_3_1, fma(1.0 * oo2e, (v19_0_0 - rho_e * v19_0_1), acc[95]))));
                acc[96] = fma(QCx, v20_1_0, fma(WQx, v20_1_1, fma(4.0 * oo2ze, v10_1_1, fma(1.0 * oo2e, (v20_0_0 - rho_e * v20_0_1), acc[96]))));
                acc[97] = fma(QCx, v20_2_0, fma(WQx, v20_2_1, fma(4.0 * oo2ze, v10_2_1, acc[97])));
                acc[98] = fma(QCx, v20_3_0, fma(WQx, v20_3_1, fma(4.0 * oo2ze, v10_3_1, acc[98])));
                acc[99] = fma(QCy, v20_2_0, fma(WQy, v20_2_1, fma(1.0 * oo2e, (v20_0_0 - rho_e * v20_0_1), acc[99])));
                acc[100] = fma(QCy, v20_3_0, fma(WQy, v20_3_1, acc[100]));
                acc[101] = fma(QCz, v20_3_0, fma(WQz, v20_3_1, fma(1.0 * oo2e, (v20_0_0 - rho_e * v20_0_1), acc[101])));
                acc[102] = fma(QCx, v21_1_0, fma(WQx, v21_1_1, fma(3.0 * oo2ze, v11_1_1, fma(1.0 * oo2e, (v21_0_0 - rho_e * v21_0_1), acc[102]))));
                acc[103] = fma(QCx, v21_2_0, fma(WQx, v21_2_1, fma(3.0 * oo2ze, v11_2_1, acc[103])));
                acc[104] = fma(QCx, v21_3_0, fma(WQx, v21_3_1, fma(3.0 * oo2ze, v11_3_1, acc[104])));
                acc[105] = fma(QCy, v21_2_0, fma(WQy, v21_2_1, fma(1.0 * oo2ze, v10_2_1, fma(1.0 * oo2e, (v21_0_0 - rho_e * v21_0_1), acc[105]))));
                acc[106] = fma(QCy, v21_3_0, fma(WQy, v21_3_1, fma(1.0 * oo2ze, v10_3_1, acc[106])));
                acc[107] = fma(QCz, v21_3_0, fma(WQz, v21_3_1, fma(1.0 * oo2e, (v21_0_0 - rho_e * v21_0_1), acc[107])));
                acc[108] = fma(QCx, v22_1_0, fma(WQx, v22_1_1, fma(3.0 * oo2ze, v12_1_1, fma(1.0 * oo2e, (v22_0_0 - rho_e * v22_0_1), acc[108]))));
                acc[109] = fma(QCx, v22_2_0, fma(WQx, v22_2_1, fma(3.0 * oo2ze, v12_2_1, acc[109])));
                acc[110] = fma(QCx, v22_3_0, fma(WQx, v22_3_1, fma(3.0 * oo2ze, v12_3_1, acc[110])));
                acc[111] = fma(QCy, v22_2_0, fma(WQy, v22_2_1, fma(1.0 * oo2e, (v22_0_0 - rho_e * v22_0_1), acc[111])));
                acc[112] = fma(QCy, v22_3_0, fma(WQy, v22_3_1, acc[112]));
                acc[113] = fma(QCz, v22_3_0, fma(WQz, v22_3_1, fma(1.0 * oo2ze, v10_3_1, fma(1.0 * oo2e, (v22_0_0 - rho_e * v22_0_1), acc[113]))));
                acc[114] = fma(QCx, v23_1_0, fma(WQx, v23_1_1, fma(2.0 * oo2ze, v13_1_1, fma(1.0 * oo2e, (v23_0_0 - rho_e * v23_0_1), acc[114]))));
                acc[115] = fma(QCx, v23_2_0, fma(WQx, v23_2_1, fma(2.0 * oo2ze, v13_2_1, acc[115])));
                acc[116] = fma(QCx, v23_3_0, fma(WQx, v23_3_1, fma(2.0 * oo2ze, v13_3_1, acc[116])));
                acc[117] = fma(QCy, v23_2_0, fma(WQy, v23_2_1, fma(2.0 * oo2ze, v11_2_1, fma(1.0 * oo2e, (v23_0_0 - rho_e * v23_0_1), acc[117]))));
                acc[118] = fma(QCy, v23_3_0, fma(WQy, v23_3_1, fma(2.0 * oo2ze, v11_3_1, acc[118])));
                acc[119] = fma(QCz, v23_3_0, fma(WQz, v23_3_1, fma(1.0 * oo2e, (v23_0_0 - rho_e * v23_0_1), acc[119])));
                acc[120] = fma(QCx, v24_1_0, fma(WQx, v24_1_1, fma(2.0 * oo2ze, v15_1_1, fma(1.0 * oo2e, (v24_0_0 - rho_e * v24_0_1), acc[120]))));
                acc[121] = fma(QCx, v24_2_0, fma(WQx, v24_2_1, fma(2.0 * oo2ze, v15_2_1, acc[121])));
                acc[122] = fma(QCx, v24_3_0, fma(WQx, v24_3_1, fma(2.0 * oo2ze, v15_3_1, acc[122])));
                acc[123] = fma(QCy, v24_2_0, fma(WQy, v24_2_1, fma(1.0 * oo2ze, v12_2_1, fma(1.0 * oo2e, (v24_0_0 - rho_e * v24_0_1), acc[123]))));
                acc[124] = fma(QCy, v24_3_0, fma(WQy, v24_3_1, fma(1.0 * oo2ze, v12_3_1, acc[124])));
                acc[125] = fma(QCz, v24_3_0, fma(WQz, v24_3_1, fma(1.0 * oo2ze, v11_3_1, fma(1.0 * oo2e, (v24_0_0 - rho_e * v24_0_1), acc[125]))));
                acc[126] = fma(QCx, v25_1_0, fma(WQx, v25_1_1, fma(2.0 * oo2ze, v14_1_1, fma(1.0 * oo2e, (v25_0_0 - rho_e * v25_0_1), acc[126]))));
                acc[127] = fma(QCx, v25_2_0, fma(WQx, v25_2_1, fma(2.0 * oo2ze, v14_2_1, acc[127])));
                acc[128] = fma(QCx, v25_3_0, fma(WQx, v25_3_1, fma(2.0 * oo2ze, v14_3_1, acc[128])));
                acc[129] = fma(QCy, v25_2_0, fma(WQy, v25_2_1, fma(1.0 * oo2e, (v25_0_0 - rho_e * v25_0_1), acc[129])));
                acc[130] = fma(QCy, v25_3_0, fma(WQy, v25_3_1, acc[130]));
                acc[131] = fma(QCz, v25_3_0, fma(WQz, v25_3_1, fma(2.0 * oo2ze, v12_3_1, fma(1.0 * oo2e, (v25_0_0 - rho_e * v25_0_1), acc[131]))));
                acc[132] = fma(QCx, v26_1_0, fma(WQx, v26_1_1, fma(1.0 * oo2ze, v16_1_1, fma(1.0 * oo2e, (v26_0_0 - rho_e * v26_0_1), acc[132]))));
                acc[133] = fma(QCx, v26_2_0, fma(WQx, v26_2_1, fma(1.0 * oo2ze, v16_2_1, acc[133])));
                acc[134] = fma(QCx, v26_3_0, fma(WQx, v26_3_1, fma(1.0 * oo2ze, v16_3_1, acc[134])));
                acc[135] = fma(QCy, v26_2_0, fma(WQy, v26_2_1, fma(3.0 * oo2ze, v13_2_1, fma(1.0 * oo2e, (v26_0_0 - rho_e * v26_0_1), acc[135]))));
                acc[136] = fma(QCy, v26_3_0, fma(WQy, v26_3_1, fma(3.0 * oo2ze, v13_3_1, acc[136])));
                acc[137] = fma(QCz, v26_3_0, fma(WQz, v26_3_1, fma(1.0 * oo2e, (v26_0_0 - rho_e * v26_0_1), acc[137])));
                acc[138] = fma(QCx, v27_1_0, fma(WQx, v27_1_1, fma(1.0 * oo2ze, v17_1_1, fma(1.0 * oo2e, (v27_0_0 - rho_e * v27_0_1), acc[138]))));
                acc[139] = fma(QCx, v27_2_0, fma(WQx, v27_2_1, fma(1.0 * oo2ze, v17_2_1, acc[139])));
                acc[140] = fma(QCx, v27_3_0, fma(WQx, v27_3_1, fma(1.0 * oo2ze, v17_3_1, acc[140])));
                acc[141] = fma(QCy, v27_2_0, fma(WQy, v27_2_1, fma(2.0 * oo2ze, v15_2_1, fma(1.0 * oo2e, (v27_0_0 - rho_e * v27_0_1), acc[141]))));
                acc[142] = fma(QCy, v27_3_0, fma(WQy, v27_3_1, fma(2.0 * oo2ze, v15_3_1, acc[142])));
                acc[143] = fma(QCz, v27_3_0, fma(WQz, v27_3_1, fma(1.0 * oo2ze, v13_3_1, fma(1.0 * oo2e, (v27_0_0 - rho_e * v27_0_1), acc[143]))));
                acc[144] = fma(QCx, v28_1_0, fma(WQx, v28_1_1, fma(1.0 * oo2ze, v18_1_1, fma(1.0 * oo2e, (v28_0_0 - rho_e * v28_0_1), acc[144]))));
                acc[145] = fma(QCx, v28_2_0, fma(WQx, v28_2_1, fma(1.0 * oo2ze, v18_2_1, acc[145])));
                acc[146] = fma(QCx, v28_3_0, fma(WQx, v28_3_1, fma(1.0 * oo2ze, v18_3_1, acc[146])));
                acc[147] = fma(QCy, v28_2_0, fma(WQy, v28_2_1, fma(1.0 * oo2ze, v14_2_1, fma(1.0 * oo2e, (v28_0_0 - rho_e * v28_0_1), acc[147]))));
                acc[148] = fma(QCy, v28_3_0, fma(WQy, v28_3_1, fma(1.0 * oo2ze, v14_3_1, acc[148])));
                acc[149] = fma(QCz, v28_3_0, fma(WQz, v28_3_1, fma(2.0 * oo2ze, v15_3_1, fma(1.0 * oo2e, (v28_0_0 - rho_e * v28_0_1), acc[149]))));
                acc[150] = fma(QCx, v29_1_0, fma(WQx, v29_1_1, fma(1.0 * oo2ze, v19_1_1, fma(1.0 * oo2e, (v29_0_0 - rho_e * v29_0_1), acc[150]))));
                acc[151] = fma(QCx, v29_2_0, fma(WQx, v29_2_1, fma(1.0 * oo2ze, v19_2_1, acc[151])));
                acc[152] = fma(QCx, v29_3_0, fma(WQx, v29_3_1, fma(1.0 * oo2ze, v19_3_1, acc[152])));
                acc[153] = fma(QCy, v29_2_0, fma(WQy, v29_2_1, fma(1.0 * oo2e, (v29_0_0 - rho_e * v29_0_1), acc[153])));
                acc[154] = fma(QCy, v29_3_0, fma(WQy, v29_3_1, acc[154]));
                acc[155] = fma(QCz, v29_3_0, fma(WQz, v29_3_1, fma(3.0 * oo2ze, v14_3_1, fma(1.0 * oo2e, (v29_0_0 - rho_e * v29_0_1), acc[155]))));
                acc[156] = fma(QCx, v30_1_0, fma(WQx, v30_1_1, fma(1.0 * oo2e, (v30_0_0 - rho_e * v30_0_1), acc[156])));
                acc[157] = fma(QCx, v30_2_0, fma(WQx, v30_2_1, acc[157]));
                acc[158] = fma(QCx, v30_3_0, fma(WQx, v30_3_1, acc[158]));
                acc[159] = fma(QCy, v30_2_0, fma(WQy, v30_2_1, fma(4.0 * oo2ze, v16_2_1, fma(1.0 * oo2e, (v30_0_0 - rho_e * v30_0_1), acc[159]))));
                acc[160] = fma(QCy, v30_3_0, fma(WQy, v30_3_1, fma(4.0 * oo2ze, v16_3_1, acc[160])));
                acc[161] = fma(QCz, v30_3_0, fma(WQz, v30_3_1, fma(1.0 * oo2e, (v30_0_0 - rho_e * v30_0_1), acc[161])));
                acc[162] = fma(QCx, v31_1_0, fma(WQx, v31_1_1, fma(1.0 * oo2e, (v31_0_0 - rho_e * v31_0_1), acc[162])));
                acc[163] = fma(QCx, v31_2_0, fma(WQx, v31_2_1, acc[163]));
                acc[164] = fma(QCx, v31_3_0, fma(WQx, v31_3_1, acc[164]));
                acc[165] = fma(QCy, v31_2_0, fma(WQy, v31_2_1, fma(3.0 * oo2ze, v17_2_1, fma(1.0 * oo2e, (v31_0_0 - rho_e * v31_0_1), acc[165]))));
                acc[166] = fma(QCy, v31_3_0, fma(WQy, v31_3_1, fma(3.0 * oo2ze, v17_3_1, acc[166])));
                acc[167] = fma(QCz, v31_3_0, fma(WQz, v31_3_1, fma(1.0 * oo2ze, v16_3_1, fma(1.0 * oo2e, (v31_0_0 - rho_e * v31_0_1), acc[167]))));
                acc[168] = fma(QCx, v32_1_0, fma(WQx, v32_1_1, fma(1.0 * oo2e, (v32_0_0 - rho_e * v32_0_1), acc[168])));
                acc[169] = fma(QCx, v32_2_0, fma(WQx, v32_2_1, acc[169]));
                acc[170] = fma(QCx, v32_3_0, fma(WQx, v32_3_1, acc[170]));
                acc[171] = fma(QCy, v32_2_0, fma(WQy, v32_2_1, fma(2.0 * oo2ze, v18_2_1, fma(1.0 * oo2e, (v32_0_0 - rho_e * v32_0_1), acc[171]))));
                acc[172] = fma(QCy, v32_3_0, fma(WQy, v32_3_1, fma(2.0 * oo2ze, v18_3_1, acc[172])));
                acc[173] = fma(QCz, v32_3_0, fma(WQz, v32_3_1, fma(2.0 * oo2ze, v17_3_1, fma(1.0 * oo2e, (v32_0_0 - rho_e * v32_0_1), acc[173]))));
                acc[174] = fma(QCx, v33_1_0, fma(WQx, v33_1_1, fma(1.0 * oo2e, (v33_0_0 - rho_e * v33_0_1), acc[174])));
                acc[175] = fma(QCx, v33_2_0, fma(WQx, v33_2_1, acc[175]));
                acc[176] = fma(QCx, v33_3_0, fma(WQx, v33_3_1, acc[176]));
                acc[177] = fma(QCy, v33_2_0, fma(WQy, v33_2_1, fma(1.0 * oo2ze, v19_2_1, fma(1.0 * oo2e, (v33_0_0 - rho_e * v33_0_1), acc[177]))));
                acc[178] = fma(QCy, v33_3_0, fma(WQy, v33_3_1, fma(1.0 * oo2ze, v19_3_1, acc[178])));
                acc[179] = fma(QCz, v33_3_0, fma(WQz, v33_3_1, fma(3.0 * oo2ze, v18_3_1, fma(1.0 * oo2e, (v33_0_0 - rho_e * v33_0_1), acc[179]))));
                acc[180] = fma(QCx, v34_1_0, fma(WQx, v34_1_1, fma(1.0 * oo2e, (v34_0_0 - rho_e * v34_0_1), acc[180])));
                acc[181] = fma(QCx, v34_2_0, fma(WQx, v34_2_1, acc[181]));
                acc[182] = fma(QCx, v34_3_0, fma(WQx, v34_3_1, acc[182]));
                acc[183] = fma(QCy, v34_2_0, fma(WQy, v34_2_1, fma(1.0 * oo2e, (v34_0_0 - rho_e * v34_0_1), acc[183])));
                acc[184] = fma(QCy, v34_3_0, fma(WQy, v34_3_1, acc[184]));
                acc[185] = fma(QCz, v34_3_0, fma(WQz, v34_3_1, fma(4.0 * oo2ze, v19_3_1, fma(1.0 * oo2e, (v34_0_0 - rho_e * v34_0_1), acc[185]))));
            } else {
                const VT v4_4_0 = QCx * v4_1_0 + WQx * v4_1_1 + (VT)2.0 * oo2ze * v1_1_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[0] += (double)v4_4_0;
                const VT v4_5_0 = QCx * v4_2_0 + WQx * v4_2_1 + (VT)2.0 * oo2ze * v1_2_1;
                acc[1] += (double)v4_5_0;
                const VT v4_6_0 = QCx * v4_3_0 + WQx * v4_3_1 + (VT)2.0 * oo2ze * v1_3_1;
                acc[2] += (double)v4_6_0;
                const VT v4_7_0 = QCy * v4_2_0 + WQy * v4_2_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[3] += (double)v4_7_0;
                const VT v4_8_0 = QCy * v4_3_0 + WQy * v4_3_1;
                acc[4] += (double)v4_8_0;
                const VT v4_9_0 = QCz * v4_3_0 + WQz * v4_3_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[5] += (double)v4_9_0;
                const VT v5_4_0 = QCx * v5_1_0 + WQx * v5_1_1 + (VT)1.0 * oo2ze * v2_1_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[6] += (double)v5_4_0;
                const VT v5_5_0 = QCx * v5_2_0 + WQx * v5_2_1 + (VT)1.0 * oo2ze * v2_2_1;
                acc[7] += (double)v5_5_0;
                const VT v5_6_0 = QCx * v5_3_0 + WQx * v5_3_1 + (VT)1.0 * oo2ze * v2_3_1;
                acc[8] += (double)v5_6_0;
                const VT v5_7_0 = QCy * v5_2_0 + WQy * v5_2_1 + (VT)1.0 * oo2ze * v1_2_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[9] += (double)v5_7_0;
                const VT v5_8_0 = QCy * v5_3_0 + WQy * v5_3_1 + (VT)1.0 * oo2ze * v1_3_1;
                acc[10] += (double)v5_8_0;
                const VT v5_9_0 = QCz * v5_3_0 + WQz * v5_3_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[11] += (double)v5_9_0;
                const VT v6_4_0 = QCx * v6_1_0 + WQx * v6_1_1 + (VT)1.0 * oo2ze * v3_1_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[12] += (double)v6_4_0;
                const VT v6_5_0 = QCx * v6_2_0 + WQx * v6_2_1 + (VT)1.0 * oo2ze * v3_2_1;
                acc[13] += (double)v6_5_0;
                const VT v6_6_0 = QCx * v6_3_0 + WQx * v6_3_1 + (VT)1.0 * oo2ze * v3_3_1;
                acc[14] += (double)v6_6_0;
                const VT v6_7_0 = QCy * v6_2_0 + WQy * v6_2_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[15] += (double)v6_7_0;
                const VT v6_8_0 = QCy * v6_3_0 + WQy * v6_3_1;
                acc[16] += (double)v6_8_0;
                const VT v6_9_0 = QCz * v6_3_0 + WQz * v6_3_1 + (VT)1.0 * oo2ze * v1_3_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[17] += (double)v6_9_0;
                const VT v7_4_0 = QCx * v7_1_0 + WQx * v7_1_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[18] += (double)v7_4_0;
                const VT v7_5_0 = QCx * v7_2_0 + WQx * v7_2_1;
                acc[19] += (double)v7_5_0;
                const VT v7_6_0 = QCx * v7_3_0 + WQx * v7_3_1;
                acc[20] += (double)v7_6_0;
                const VT v7_7_0 = QCy * v7_2_0 + WQy * v7_2_1 + (VT)2.0 * oo2ze * v2_2_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[21] += (double)v7_7_0;
                const VT v7_8_0 = QCy * v7_3_0 + WQy * v7_3_1 + (VT)2.0 * oo2ze * v2_3_1;
                acc[22] += (double)v7_8_0;
                const VT v7_9_0 = QCz * v7_3_0 + WQz * v7_3_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[23] += (double)v7_9_0;
                const VT v8_4_0 = QCx * v8_1_0 + WQx * v8_1_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[24] += (double)v8_4_0;
                const VT v8_5_0 = QCx * v8_2_0 + WQx * v8_2_1;
                acc[25] += (double)v8_5_0;
                const VT v8_6_0 = QCx * v8_3_0 + WQx * v8_3_1;
                acc[26] += (double)v8_6_0;
                const VT v8_7_0 = QCy * v8_2_0 + WQy * v8_2_1 + (VT)1.0 * oo2ze * v3_2_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[27] += (double)v8_7_0;
                const VT v8_8_0 = QCy * v8_3_0 + WQy * v8_3_1 + (VT)1.0 * oo2ze * v3_3_1;
                acc[28] += (double)v8_8_0;
                const VT v8_9_0 = QCz * v8_3_0 + WQz * v8_3_1 + (VT)1.0 * oo2ze * v2_3_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[29] += (double)v8_9_0;
                const VT v9_4_0 = QCx * v9_1_0 + WQx * v9_1_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[30] += (double)v9_4_0;
                const VT v9_5_0 = QCx * v9_2_0 + WQx * v9_2_1;
                acc[31] += (double)v9_5_0;
                const VT v9_6_0 = QCx * v9_3_0 + WQx * v9_3_1;
                acc[32] += (double)v9_6_0;
                const VT v9_7_0 = QCy * v9_2_0 + WQy * v9_2_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[33] += (double)v9_7_0;
                const VT v9_8_0 = QCy * v9_3_0 + WQy * v9_3_1;
                acc[34] += (double)v9_8_0;
                const VT v9_9_0 = QCz * v9_3_0 + WQz * v9_3_1 + (VT)2.0 * oo2ze * v3_3_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[35] += (double)v9_9_0;
                const VT v10_4_0 = QCx * v10_1_0 + WQx * v10_1_1 + (VT)3.0 * oo2ze * v4_1_1 + (VT)1.0 * oo2e * (v10_0_0 - rho_e * v10_0_1);
                acc[36] += (double)v10_4_0;
                const VT v10_5_0 = QCx * v10_2_0 + WQx * v10_2_1 + (VT)3.0 * oo2ze * v4_2_1;
                acc[37] += (double)v10_5_0;
                const VT v10_6_0 = QCx * v10_3_0 + WQx * v10_3_1 + (VT)3.0 * oo2ze * v4_3_1;
                acc[38] += (double)v10_6_0;
                const VT v10_7_0 = QCy * v10_2_0 + WQy * v10_2_1 + (VT)1.0 * oo2e * (v10_0_0 - rho_e * v10_0_1);
                acc[39] += (double)v10_7_0;
                const VT v10_8_0 = QCy * v10_3_0 + WQy * v10_3_1;
                acc[40] += (double)v10_8_0;
                const VT v10_9_0 = QCz * v10_3_0 + WQz * v10_3_1 + (VT)1.0 * oo2e * (v10_0_0 - rho_e * v10_0_1);
                acc[41] += (double)v10_9_0;
                const VT v11_4_0 = QCx * v11_1_0 + WQx * v11_1_1 + (VT)2.0 * oo2ze * v5_1_1 + (VT)1.0 * oo2e * (v11_0_0 - rho_e * v11_0_1);
                acc[42] += (double)v11_4_0;
                const VT v11_5_0 = QCx * v11_2_0 + WQx * v11_2_1 + (VT)2.0 * oo2ze * v5_2_1;
                acc[43] += (double)v11_5_0;
                const VT v11_6_0 = QCx * v11_3_0 + WQx * v11_3_1 + (VT)2.0 * oo2ze * v5_3_1;
                acc[44] += (double)v11_6_0;
                const VT v11_7_0 = QCy * v11_2_0 + WQy * v11_2_1 + (VT)1.0 * oo2ze * v4_2_1 + (VT)1.0 * oo2e * (v11_0_0 - rho_e * v11_0_1);
                acc[45] += (double)v11_7_0;
                const VT v11_8_0 = QCy * v11_3_0 + WQy * v11_3_1 + (VT)1.0 * oo2ze * v4_3_1;
                acc[46] += (double)v11_8_0;
                const VT v11_9_0 = QCz * v11_3_0 + WQz * v11_3_1 + (VT)1.0 * oo2e * (v11_0_0 - rho_e * v11_0_1);
                acc[47] += (double)v11_9_0;
                const VT v12_4_0 = QCx * v12_1_0 + WQx * v12_1_1 + (VT)2.0 * oo2ze * v6_1_1 + (VT)1.0 * oo2e * (v12_0_0 - rho_e * v12_0_1);
                acc[48] += (double)v12_4_0;
                const VT v12_5_0 = QCx * v12_2_0 + WQx * v12_2_1 + (VT)2.0 * oo2ze * v6_2_1;
                acc[49] += (double)v12_5_0;
                const VT v12_6_0 = QCx * v12_3_0 + WQx * v12_3_1 + (VT)2.0 * oo2ze * v6_3_1;
                acc[50] += (double)v12_6_0;
                const VT v12_7_0 = QCy * v12_2_0 + WQy * v12_2_1 + (VT)1.0 * oo2e * (v12_0_0 - rho_e * v12_0_1);
                acc[51] += (double)v12_7_0;
                const VT v12_8_0 = QCy * v12_3_0 + WQy * v12_3_1;
                acc[52] += (double)v12_8_0;
                const VT v12_9_0 = QCz * v12_3_0 + WQz * v12_3_1 + (VT)1.0 * oo2ze * v4_3_1 + (VT)1.0 * oo2e * (v12_0_0 - rho_e * v12_0_1);
                acc[53] += (double)v12_9_0;
                const VT v13_4_0 = QCx * v13_1_0 + WQx * v13_1_1 + (VT)1.0 * oo2ze * v7_1_1 + (VT)1.0 * oo2e * (v13_0_0 - rho_e * v13_0_1);
                acc[54] += (double)v13_4_0;
                const VT v13_5_0 = QCx * v13_2_0 + WQx * v13_2_1 + (VT)1.0 * oo2ze * v7_2_1;
                acc[55] += (double)v13_5_0;
                const VT v13_6_0 = QCx * v13_3_0 + WQx * v13_3_1 + (VT)1.0 * oo2ze * v7_3_1;
                acc[56] += (double)v13_6_0;
                const VT v13_7_0 = QCy * v13_2_0 + WQy * v13_2_1 + (VT)2.0 * oo2ze * v5_2_1 + (VT)1.0 * oo2e * (v13_0_0 - rho_e * v13_0_1);
                acc[57] += (double)v13_7_0;
                const VT v13_8_0 = QCy * v13_3_0 + WQy * v13_3_1 + (VT)2.0 * oo2ze * v5_3_1;
                acc[58] += (double)v13_8_0;
                const VT v13_9_0 = QCz * v13_3_0 + WQz * v13_3_1 + (VT)1.0 * oo2e * (v13_0_0 - rho_e * v13_0_1);
                acc[59] += (double)v13_9_0;
                const VT v14_4_0 = QCx * v14_1_0 + WQx * v14_1_1 + (VT)1.0 * oo2ze * v9_1_1 + (VT)1.0 * oo2e * (v14_0_0 - rho_e * v14_0_1);
                acc[60] += (double)v14_4_0;
                const VT v14_5_0 = QCx * v14_2_0 + WQx * v14_2_1 + (VT)1.0 * oo2ze * v9_2_1;
                acc[61] += (double)v14_5_0;
                const VT v14_6_0 = QCx * v14_3_0 + WQx * v14_3_1 + (VT)1.0 * oo2ze * v9_3_1;
                acc[62] += (double)v14_6_0;
                const VT v14_7_0 = QCy * v14_2_0 + WQy * v14_2_1 + (VT)1.0 * oo2e * (v14_0_0 - rho_e * v14_0_1);
                acc[63] += (double)v14_7_0;
                const VT v14_8_0 = QCy * v14_3_0 + WQy * v14_3_1;
                acc[64] += (double)v14_8_0;
                const VT v14_9_0 = QCz * v14_3_0 + WQz * v14_3_1 + (VT)2.0 * oo2ze * v6_3_1 + (VT)1.0 * oo2e * (v14_0_0 - rho_e * v14_0_1);
                acc[65] += (double)v14_9_0;
                const VT v15_4_0 = QCx * v15_1_0 + WQx * v15_1_1 + (VT)1.0 * oo2ze * v8_1_1 + (VT)1.0 * oo2e * (v15_0_0 - rho_e * v15_0_1);
                acc[66] += (double)v15_4_0;
                const VT v15_5_0 = QCx * v15_2_0 + WQx * v15_2_1 + (VT)1.0 * oo2ze * v8_2_1;
                acc[67] += (double)v15_5_0;
                const VT v15_6_0 = QCx * v15_3_0 + WQx * v15_3_1 + (VT)1.0 * oo2ze * v8_3_1;
                acc[68] += (double)v15_6_0;
                const VT v15_7_0 = QCy * v15_2_0 + WQy * v15_2_1 + (VT)1.0 * oo2ze * v6_2_1 + (VT)1.0 * oo2e * (v15_0_0 - rho_e * v15_0_1);
                acc[69] += (double)v15_7_0;
                const VT v15_8_0 = QCy * v15_3_0 + WQy * v15_3_1 + (VT)1.0 * oo2ze * v6_3_1;
                acc[70] += (double)v15_8_0;
                const VT v15_9_0 = QCz * v15_3_0 + WQz * v15_3_1 + (VT)1.0 * oo2ze * v5_3_1 + (VT)1.0 * oo2e * (v15_0_0 - rho_e * v15_0_1);
                acc[71] += (double)v15_9_0;
                const VT v16_4_0 = QCx * v16_1_0 + WQx * v16_1_1 + (VT)1.0 * oo2e * (v16_0_0 - rho_e * v16_0_1);
                acc[72] += (double)v16_4_0;
                const VT v16_5_0 = QCx * v16_2_0 + WQx * v16_2_1;
                acc[73] += (double)v16_5_0;
                const VT v16_6_0 = QCx * v16_3_0 + WQx * v16_3_1;
                acc[74] += (double)v16_6_0;
                const VT v16_7_0 = QCy * v16_2_0 + WQy * v16_2_1 + (VT)3.0 * oo2ze * v7_2_1 + (VT)1.0 * oo2e * (v16_0_0 - rho_e * v16_0_1);
                acc[75] += (double)v16_7_0;
                const VT v16_8_0 = QCy * v16_3_0 + WQy * v16_3_1 + (VT)3.0 * oo2ze * v7_3_1;
                acc[76] += (double)v16_8_0;
                const VT v16_9_0 = QCz * v16_3_0 + WQz * v16_3_1 + (VT)1.0 * oo2e * (v16_0_0 - rho_e * v16_0_1);
                acc[77] += (double)v16_9_0;
                const VT v17_4_0 = QCx * v17_1_0 + WQx * v17_1_1 + (VT)1.0 * oo2e * (v17_0_0 - rho_e * v17_0_1);
                acc[78] += (double)v17_4_0;
                const VT v17_5_0 = QCx * v17_2_0 + WQx * v17_2_1;
                acc[79] += (double)v17_5_0;
                const VT v17_6_0 = QCx * v17_3_0 + WQx * v17_3_1;
                acc[80] += (double)v17_6_0;
                const VT v17_7_0 = QCy * v17_2_0 + WQy * v17_2_1 + (VT)2.0 * oo2ze * v8_2_1 + (VT)1.0 * oo2e * (v17_0_0 - rho_e * v17_0_1);
                acc[81] += (double)v17_7_0;
                const VT v17_8_0 = QCy * v17_3_0 + WQy * v17_3_1 + (VT)2.0 * oo2ze * v8_3_1;
                acc[82] += (double)v17_8_0;
                const VT v17_9_0 = QCz * v17_3_0 + WQz * v17_3_1 + (VT)1.0 * oo2ze * v7_3_1 + (VT)1.0 * oo2e * (v17_0_0 - rho_e * v17_0_1);
                acc[83] += (double)v17_9_0;
                const VT v18_4_0 = QCx * v18_1_0 + WQx * v18_1_1 + (VT)1.0 * oo2e * (v18_0_0 - rho_e * v18_0_1);
                acc[84] += (double)v18_4_0;
                const VT v18_5_0 = QCx * v18_2_0 + WQx * v18_2_1;
                acc[85] += (double)v18_5_0;
                const VT v18_6_0 = QCx * v18_3_0 + WQx * v18_3_1;
                acc[86] += (double)v18_6_0;
                const VT v18_7_0 = QCy * v18_2_0 + WQy * v18_2_1 + (VT)1.0 * oo2ze * v9_2_1 + (VT)1.0 * oo2e * (v18_0_0 - rho_e * v18_0_1);
                acc[87] += (double)v18_7_0;
                const VT v18_8_0 = QCy * v18_3_0 + WQy * v18_3_1 + (VT)1.0 * oo2ze * v9_3_1;
                acc[88] += (double)v18_8_0;
                const VT v18_9_0 = QCz * v18_3_0 + WQz * v18_3_1 + (VT)2.0 * oo2ze * v8_3_1 + (VT)1.0 * oo2e * (v18_0_0 - rho_e * v18_0_1);
                acc[89] += (double)v18_9_0;
                const VT v19_4_0 = QCx * v19_1_0 + WQx * v19_1_1 + (VT)1.0 * oo2e * (v19_0_0 - rho_e * v19_0_1);
                acc[90] += (double)v19_4_0;
                const VT v19_5_0 = QCx * v19_2_0 + WQx * v19_2_1;
                acc[91] += (double)v19_5_0;
                const VT v19_6_0 = QCx * v19_3_0 + WQx * v19_3_1;
                acc[92] += (double)v19_6_0;
                const VT v19_7_0 = QCy * v19_2_0 + WQy * v19_2_1 + (VT)1.0 * oo2e * (v19_0_0 - rho_e * v19_0_1);
                acc[93] += (double)v19_7_0;
                const VT v19_8_0 = QCy * v19_3_0 + WQy * v19_3_1;
                acc[94] += (double)v19_8_0;
                const VT v19_9_0 = QCz * v19_3_0 + WQz * v19_3_1 + (VT)3.0 * oo2ze * v9_3_1 + (VT)1.0 * oo2e * (v19_0_0 - rho_e * v19_0_1);
                acc[95] += (double)v19_9_0;
                const VT v20_4_0 = QCx * v20_1_0 + WQx * v20_1_1 + (VT)4.0 * oo2ze * v10_1_1 + (VT)1.0 * oo2e * (v20_0_0 - rho_e * v20_0_1);
                acc[96] += (double)v20_4_0;
                const VT v20_5_0 = QCx * v20_2_0 + WQx * v20_2_1 + (VT)4.0 * oo2ze * v10_2_1;
                acc[97] += (double)v20_5_0;
                const VT v20_6_0 = QCx * v20_3_0 + WQx * v20_3_1 + (VT)4.0 * oo2ze * v10_3_1;
                acc[98] += (double)v20_6_0;
                const VT v20_7_0 = QCy * v20_2_0 + WQy * v20_2_1 + (VT)1.0 * oo2e * (v20_0_0 - rho_e * v20_0_1);
                acc[99] += (double)v20_7_0;
                const VT v20_8_0 = QCy * v20_3_0 + WQy * v20_3_1;
                acc[100] += (double)v20_8_0;
                const VT v20_9_0 = QCz * v20_3_0 + WQz * v20_3_1 + (VT)1.0 * oo2e * (v20_0_0 - rho_e * v20_0_1);
                acc[101] += (double)v20_9_0;
                const VT v21_4_0 = QCx * v21_1_0 + WQx * v21_1_1 + (VT)3.0 * oo2ze * v11_1_1 + (VT)1.0 * oo2e * (v21_0_0 - rho_e * v21_0_1);
                acc[102] += (double)v21_4_0;
                const VT v21_5_0 = QCx * v21_2_0 + WQx * v21_2_1 + (VT)3.0 * oo2ze * v11_2_1;
                acc[103] += (double)v21_5_0;
                const VT v21_6_0 = QCx * v21_3_0 + WQx * v21_3_1 + (VT)3.0 * oo2ze * v11_3_1;
                acc[104] += (double)v21_6_0;
                const VT v21_7_0 = QCy * v21_2_0 + WQy * v21_2_1 + (VT)1.0 * oo2ze * v10_2_1 + (VT)1.0 * oo2e * (v21_0_0 - rho_e * v21_0_1);
                acc[105] += (double)v21_7_0;
                const VT v21_8_0 = QCy * v21_3_0 + WQy * v21_3_1 + (VT)1.0 * oo2ze * v10_3_1;
                acc[106] += (double)v21_8_0;
                const VT v21_9_0 = QCz * v21_3_0 + WQz * v21_3_1 + (VT)1.0 * oo2e * (v21_0_0 - rho_e * v21_0_1);
                acc[107] += (double)v21_9_0;
                const VT v22_4_0 = QCx * v22_1_0 + WQx * v22_1_1 + (VT)3.0 * oo2ze * v12_1_1 + (VT)1.0 * oo2e * (v22_0_0 - rho_e * v22_0_1);
                acc[108] += (double)v22_4_0;
                const VT v22_5_0 = QCx * v22_2_0 + WQx * v22_2_1 + (VT)3.0 * oo2ze * v12_2_1;
                acc[109] += (double)v22_5_0;
                const VT v22_6_0 = QCx * v22_3_0 + WQx * v22_3_1 + (VT)3.0 * oo2ze * v12_3_1;
                acc[110] += (double)v22_6_0;
                const VT v22_7_0 = QCy * v22_2_0 + WQy * v22_2_1 + (VT)1.0 * oo2e * (v22_0_0 - rho_e * v22_0_1);
                acc[111] += (double)v22_7_0;
                const VT v22_8_0 = QCy * v22_3_0 + WQy * v22_3_1;
                acc[112] += (double)v22_8_0;
                const VT v22_9_0 = QCz * v22_3_0 + WQz * v22_3_1 + (VT)1.0 * oo2ze * v10_3_1 + (VT)1.0 * oo2e * (v22_0_0 - rho_e * v22_0_1);
                acc[113] += (double)v22_9_0;
                const VT v23_4_0 = QCx * v23_1_0 + WQx * v23_1_1 + (VT)2.0 * oo2ze * v13_1_1 + (VT)1.0 * oo2e * (v23_0_0 - rho_e * v23_0_1);
                acc[114] += (double)v23_4_0;
                const VT v23_5_0 = QCx * v23_2_0 + WQx * v23_2_1 + (VT)2.0 * oo2ze * v13_2_1;
                acc[115] += (double)v23_5_0;
                const VT v23_6_0 = QCx * v23_3_0 + WQx * v23_3_1 + (VT)2.0 * oo2ze * v13_3_1;
                acc[116] += (double)v23_6_0;
                const VT v23_7_0 = QCy * v23_2_0 + WQy * v23_2_1 + (VT)2.0 * oo2ze * v11_2_1 + (VT)1.0 * oo2e * (v23_0_0 - rho_e * v23_0_1);
                acc[117] += (double)v23_7_0;
                const VT v23_8_0 = QCy * v23_3_0 + WQy * v23_3_1 + (VT)2.0 * oo2ze * v11_3_1;
                acc[118] += (double)v23_8_0;
                const VT v23_9_0 = QCz * v23_3_0 + WQz * v23_3_1 + (VT)1.0 * oo2e * (v23_0_0 - rho_e * v23_0_1);
                acc[119] += (double)v23_9_0;
                const VT v24_4_0 = QCx * v24_1_0 + WQx * v24_1_1 + (VT)2.0 * oo2ze * v15_1_1 + (VT)1.0 * oo2e * (v24_0_0 - rho_e * v24_0_1);
                acc[120] += (double)v24_4_0;
                const VT v24_5_0 = QCx * v24_2_0 + WQx * v24_2_1 + (VT)2.0 * oo2ze * v15_2_1;
                acc[121] += (double)v24_5_0;
                const VT v24_6_0 = QCx * v24_3_0 + WQx * v24_3_1 + (VT)2.0 * oo2ze * v15_3_1;
                acc[122] += (double)v24_6_0;
                const VT v24_7_0 = QCy * v24_2_0 + WQy * v24_2_1 + (VT)1.0 * oo2ze * v12_2_1 + (VT)1.0 * oo2e * (v24_0_0 - rho_e * v24_0_1);
                acc[123] += (double)v24_7_0;
                const VT v24_8_0 = QCy * v24_3_0 + WQy * v24_3_1 + (VT)1.0 * oo2ze * v12_3_1;
                acc[124] += (double)v24_8_0;
                const VT v24_9_0 = QCz * v24_3_0 + WQz * v24_3_1 + (VT)1.0 * oo2ze * v11_3_1 + (VT)1.0 * oo2e * (v24_0_0 - rho_e * v24_0_1);
                acc[125] += (double)v24_9_0;
                const VT v25_4_0 = QCx * v25_1_0 + WQx * v25_1_1 + (VT)2.0 * oo2ze * v14_1_1 + (VT)1.0 * oo2e * (v25_0_0 - rho_e * v25_0_1);
                acc[126] += (double)v25_4_0;
                const VT v25_5_0 = QCx * v25_2_0 + WQx * v25_2_1 + (VT)2.0 * oo2ze * v14_2_1;
                acc[127] += (double)v25_5_0;
                const VT v25_6_0 = QCx * v25_3_0 + WQx * v25_3_1 + (VT)2.0 * oo2ze * v14_3_1;
                acc[128] += (double)v25_6_0;
                const VT v25_7_0 = QCy * v25_2_0 + WQy * v25_2_1 + (VT)1.0 * oo2e * (v25_0_0 - rho_e * v25_0_1);
                acc[129] += (double)v25_7_0;
                const VT v25_8_0 = QCy * v25_3_0 + WQy * v25_3_1;
                acc[130] += (double)v25_8_0;
                const VT v25_9_0 = QCz * v25_3_0 + WQz * v25_3_1 + (VT)2.0 * oo2ze * v12_3_1 + (VT)1.0 * oo2e * (v25_0_0 - rho_e * v25_0_1);
                acc[131] += (double)v25_9_0;
                const VT v26_4_0 = QCx * v26_1_0 + WQx * v26_1_1 + (VT)1.0 * oo2ze * v16_1_1 + (VT)1.0 * oo2e * (v26_0_0 - rho_e * v26_0_1);
                acc[132] += (double)v26_4_0;
                const VT v26_5_0 = QCx * v26_2_0 + WQx * v26_2_1 + (VT)1.0 * oo2ze * v16_2_1;
                acc[133] += (double)v26_5_0;
                const VT v26_6_0 = QCx * v26_3_0 + WQx * v26_3_1 + (VT)1.0 * oo2ze * v16_3_1;
                acc[134] += (double)v26_6_0;
                const VT v26_7_0 = QCy * v26_2_0 + WQy * v26_2_1 + (VT)3.0 * oo2ze * v13_2_1 + (VT)1.0 * oo2e * (v26_0_0 - rho_e * v26_0_1);
                acc[135] += (double)v26_7_0;
                const VT v26_8_0 = QCy * v26_3_0 + WQy * v26_3_1 + (VT)3.0 * oo2ze * v13_3_1;
                acc[136] += (double)v26_8_0;
                const VT v26_9_0 = QCz * v26_3_0 + WQz * v26_3_1 + (VT)1.0 * oo2e * (v26_0_0 - rho_e * v26_0_1);
                acc[137] += (double)v26_9_0;
                const VT v27_4_0 = QCx * v27_1_0 + WQx * v27_1_1 + (VT)1.0 * oo2ze * v17_1_1 + (VT)1.0 * oo2e * (v27_0_0 - rho_e * v27_0_1);
                acc[138] += (double)v27_4_0;
                const VT v27_5_0 = QCx * v27_2_0 + WQx * v27_2_1 + (VT)1.0 * oo2ze * v17_2_1;
                acc[139] += (double)v27_5_0;
                const VT v27_6_0 = QCx * v27_3_0 + WQx * v27_3_1 + (VT)1.0 * oo2ze * v17_3_1;
                acc[140] += (double)v27_6_0;
                const VT v27_7_0 = QCy * v27_2_0 + WQy * v27_2_1 + (VT)2.0 * oo2ze * v15_2_1 + (VT)1.0 * oo2e * (v27_0_0 - rho_e * v27_0_1);
                acc[141] += (double)v27_7_0;
                const VT v27_8_0 = QCy * v27_3_0 + WQy * v27_3_1 + (VT)2.0 * oo2ze * v15_3_1;
                acc[142] += (double)v27_8_0;
                const VT v27_9_0 = QCz * v27_3_0 + WQz * v27_3_1 + (VT)1.0 * oo2ze * v13_3_1 + (VT)1.0 * oo2e * (v27_0_0 - rho_e * v27_0_1);
                acc[143] += (double)v27_9_0;
                const VT v28_4_0 = QCx * v28_1_0 + WQx * v28_1_1 + (VT)1.0 * oo2ze * v18_1_1 + (VT)1.0 * oo2e * (v28_0_0 - rho_e * v28_0_1);
                acc[144] += (double)v28_4_0;
                const VT v28_5_0 = QCx * v28_2_0 + WQx * v28_2_1 + (VT)1.0 * oo2ze * v18_2_1;
                acc[145] += (double)v28_5_0;
                const VT v28_6_0 = QCx * v28_3_0 + WQx * v28_3_1 + (VT)1.0 * oo2ze * v18_3_1;
                acc[146] += (double)v28_6_0;
                const VT v28_7_0 = QCy * v28_2_0 + WQy * v28_2_1 + (VT)1.0 * oo2ze * v14_2_1 + (VT)1.0 * oo2e * (v28_0_0 - rho_e * v28_0_1);
                acc[147] += (double)v28_7_0;
                const VT v28_8_0 = QCy * v28_3_0 + WQy * v28_3_1 + (VT)1.0 * oo2ze * v14_3_1;
                acc[148] += (double)v28_8_0;
                const VT v28_9_0 = QCz * v28_3_0 + WQz * v28_3_1 + (VT)2.0 * oo2ze * v15_3_1 + (VT)1.0 * oo2e * (v28_0_0 - rho_e * v28_0_1);
                acc[149] += (double)v28_9_0;
                const VT v29_4_0 = QCx * v29_1_0 + WQx * v29_1_1 + (VT)1.0 * oo2ze * v19_1_1 + (VT)1.0 * oo2e * (v29_0_0 - rho_e * v29_0_1);
                acc[150] += (double)v29_4_0;
                const VT v29_5_0 = QCx * v29_2_0 + WQx * v29_2_1 + (VT)1.0 * oo2ze * v19_2_1;
                acc[151] += (double)v29_5_0;
                const VT v29_6_0 = QCx * v29_3_0 + WQx * v29_3_1 + (VT)1.0 * oo2ze * v19_3_1;
                acc[152] += (double)v29_6_0;
                const VT v29_7_0 = QCy * v29_2_0 + WQy * v29_2_1 + (VT)1.0 * oo2e * (v29_0_0 - rho_e * v29_0_1);
                acc[153] += (double)v29_7_0;
                const VT v29_8_0 = QCy * v29_3_0 + WQy * v29_3_1;
                acc[154] += (double)v29_8_0;
                const VT v29_9_0 = QCz * v29_3_0 + WQz * v29_3_1 + (VT)3.0 * oo2ze * v14_3_1 + (VT)1.0 * oo2e * (v29_0_0 - rho_e * v29_0_1);
                acc[155] += (double)v29_9_0;
                const VT v30_4_0 = QCx * v30_1_0 + WQx * v30_1_1 + (VT)1.0 * oo2e * (v30_0_0 - rho_e * v30_0_1);
                acc[156] += (double)v30_4_0;
                const VT v30_5_0 = QCx * v30_2_0 + WQx * v30_2_1;
                acc[157] += (double)v30_5_0;
                const VT v30_6_0 = QCx * v30_3_0 + WQx * v30_3_1;
                acc[158] += (double)v30_6_0;
                const VT v30_7_0 = QCy * v30_2_0 + WQy * v30_2_1 + (VT)4.0 * oo2ze * v16_2_1 + (VT)1.0 * oo2e * (v30_0_0 - rho_e * v30_0_1);
                acc[159] += (double)v30_7_0;
                const VT v30_8_0 = QCy * v30_3_0 + WQy * v30_3_1 + (VT)4.0 * oo2ze * v16_3_1;
                acc[160] += (double)v30_8_0;
                const VT v30_9_0 = QCz * v30_3_0 + WQz * v30_3_1 + (VT)1.0 * oo2e * (v30_0_0 - rho_e * v30_0_1);
                acc[161] += (double)v30_9_0;
                const VT v31_4_0 = QCx * v31_1_0 + WQx * v31_1_1 + (VT)1.0 * oo2e * (v31_0_0 - rho_e * v31_0_1);
                acc[162] += (double)v31_4_0;
                const VT v31_5_0 = QCx * v31_2_0 + WQx * v31_2_1;
                acc[163] += (double)v31_5_0;
                const VT v31_6_0 = QCx * v31_3_0 + WQx * v31_3_1;
                acc[164] += (double)v31_6_0;
                const VT v31_7_0 = QCy * v31_2_0 + WQy * v31_2_1 + (VT)3.0 * oo2ze * v17_2_1 + (VT)1.0 * oo2e * (v31_0_0 - rho_e * v31_0_1);
                acc[165] += (double)v31_7_0;
                const VT v31_8_0 = QCy * v31_3_0 + WQy * v31_3_1 + (VT)3.0 * oo2ze * v17_3_1;
                acc[166] += (double)v31_8_0;
                const VT v31_9_0 = QCz * v31_3_0 + WQz * v31_3_1 + (VT)1.0 * oo2ze * v16_3_1 + (VT)1.0 * oo2e * (v31_0_0 - rho_e * v31_0_1);
                acc[167] += (double)v31_9_0;
                const VT v32_4_0 = QCx * v32_1_0 + WQx * v32_1_1 + (VT)1.0 * oo2e * (v32_0_0 - rho_e * v32_0_1);
                acc[168] += (double)v32_4_0;
                const VT v32_5_0 = QCx * v32_2_0 + WQx * v32_2_1;
                acc[169] += (double)v32_5_0;
                const VT v32_6_0 = QCx * v32_3_0 + WQx * v32_3_1;
                acc[170] += (double)v32_6_0;
                const VT v32_7_0 = QCy * v32_2_0 + WQy * v32_2_1 + (VT)2.0 * oo2ze * v18_2_1 + (VT)1.0 * oo2e * (v32_0_0 - rho_e * v32_0_1);
                acc[171] += (double)v32_7_0;
                const VT v32_8_0 = QCy * v32_3_0 + WQy * v32_3_1 + (VT)2.0 * oo2ze * v18_3_1;
                acc[172] += (double)v32_8_0;
                const VT v32_9_0 = QCz * v32_3_0 + WQz * v32_3_1 + (VT)2.0 * oo2ze * v17_3_1 + (VT)1.0 * oo2e * (v32_0_0 - rho_e * v32_0_1);
                acc[173] += (double)v32_9_0;
                const VT v33_4_0 = QCx * v33_1_0 + WQx * v33_1_1 + (VT)1.0 * oo2e * (v33_0_0 - rho_e * v33_0_1);
                acc[174] += (double)v33_4_0;
                const VT v33_5_0 = QCx * v33_2_0 + WQx * v33_2_1;
                acc[175] += (double)v33_5_0;
                const VT v33_6_0 = QCx * v33_3_0 + WQx * v33_3_1;
                acc[176] += (double)v33_6_0;
                const VT v33_7_0 = QCy * v33_2_0 + WQy * v33_2_1 + (VT)1.0 * oo2ze * v19_2_1 + (VT)1.0 * oo2e * (v33_0_0 - rho_e * v33_0_1);
                acc[177] += (double)v33_7_0;
                const VT v33_8_0 = QCy * v33_3_0 + WQy * v33_3_1 + (VT)1.0 * oo2ze * v19_3_1;
                acc[178] += (double)v33_8_0;
                const VT v33_9_0 = QCz * v33_3_0 + WQz * v33_3_1 + (VT)3.0 * oo2ze * v18_3_1 + (VT)1.0 * oo2e * (v33_0_0 - rho_e * v33_0_1);
                acc[179] += (double)v33_9_0;
                const VT v34_4_0 = QCx * v34_1_0 + WQx * v34_1_1 + (VT)1.0 * oo2e * (v34_0_0 - rho_e * v34_0_1);
                acc[180] += (double)v34_4_0;
                const VT v34_5_0 = QCx * v34_2_0 + WQx * v34_2_1;
                acc[181] += (double)v34_5_0;
                const VT v34_6_0 = QCx * v34_3_0 + WQx * v34_3_1;
                acc[182] += (double)v34_6_0;
                const VT v34_7_0 = QCy * v34_2_0 + WQy * v34_2_1 + (VT)1.0 * oo2e * (v34_0_0 - rho_e * v34_0_1);
                acc[183] += (double)v34_7_0;
                const VT v34_8_0 = QCy * v34_3_0 + WQy * v34_3_1;
                acc[184] += (double)v34_8_0;
                const VT v34_9_0 = QCz * v34_3_0 + WQz * v34_3_1 + (VT)4.0 * oo2ze * v19_3_1 + (VT)1.0 * oo2e * (v34_0_0 - rho_e * v34_0_1);
                acc[185] += (double)v34_9_0;
            }
        }
    }
}

// Bra and ket HRR of the contracted block (src/HGP.jl:92-114), then the component norms:
// the normalised (ab|cd) of bra pair p and ket pair q into res[216] (ma, mb, mc, md
// row-major).
__device__ __forceinline__ void hrr_ddds(const PairTab &P, int p, int q, const double *__restrict__ acc,
                                          double *__restrict__ res) {
    const double4 gb = ldg4(&P.geo[p]);
    const double4 gk = ldg4(&P.geo[q]);
    const double ABx = gb.x, ABy = gb.y, ABz = gb.z;
    const double CDx = gk.x, CDy = gk.y, CDz = gk.z;
    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;
    const double h10_1_4 = acc[96] + ABx * acc[36];
    const double h4_1_4 = acc[36] + ABx * acc[0];
    const double h4_4_4 = h10_1_4 + ABx * h4_1_4;
    const double h10_1_5 = acc[97] + ABx * acc[37];
    const double h4_1_5 = acc[37] + ABx * acc[1];
    const double h4_4_5 = h10_1_5 + ABx * h4_1_5;
    const double h10_1_6 = acc[98] + ABx * acc[38];
    const double h4_1_6 = acc[38] + ABx * acc[2];
    const double h4_4_6 = h10_1_6 + ABx * h4_1_6;
    const double h10_1_7 = acc[99] + ABx * acc[39];
    const double h4_1_7 = acc[39] + ABx * acc[3];
    const double h4_4_7 = h10_1_7 + ABx * h4_1_7;
    const double h10_1_8 = acc[100] + ABx * acc[40];
    const double h4_1_8 = acc[40] + ABx * acc[4];
    const double h4_4_8 = h10_1_8 + ABx * h4_1_8;
    const double h10_1_9 = acc[101] + ABx * acc[41];
    const double h4_1_9 = acc[41] + ABx * acc[5];
    const double h4_4_9 = h10_1_9 + ABx * h4_1_9;
    const double h10_2_4 = acc[102] + ABy * acc[36];
    const double h4_2_4 = acc[42] + ABy * acc[0];
    const double h4_5_4 = h10_2_4 + ABx * h4_2_4;
    const double h10_2_5 = acc[103] + ABy * acc[37];
    const double h4_2_5 = acc[43] + ABy * acc[1];
    const double h4_5_5 = h10_2_5 + ABx * h4_2_5;
    const double h10_2_6 = acc[104] + ABy * acc[38];
    const double h4_2_6 = acc[44] + ABy * acc[2];
    const double h4_5_6 = h10_2_6 + ABx * h4_2_6;
    const double h10_2_7 = acc[105] + ABy * acc[39];
    const double h4_2_7 = acc[45] + ABy * acc[3];
    const double h4_5_7 = h10_2_7 + ABx * h4_2_7;
    const double h10_2_8 = acc[106] + ABy * acc[40];
    const double h4_2_8 = acc[46] + ABy * acc[4];
    const double h4_5_8 = h10_2_8 + ABx * h4_2_8;
    const double h10_2_9 = acc[107] + ABy * acc[41];
    const double h4_2_9 = acc[47] + ABy * acc[5];
    const double h4_5_9 = h10_2_9 + ABx * h4_2_9;
    const double h10_3_4 = acc[108] + ABz * acc[36];
    const double h4_3_4 = acc[48] + ABz * acc[0];
    const double h4_6_4 = h10_3_4 + ABx * h4_3_4;
    const double h10_3_5 = acc[109] + ABz * acc[37];
    const double h4_3_5 = acc[49] + ABz * acc[1];
    const double h4_6_5 = h10_3_5 + ABx * h4_3_5;
    const double h10_3_6 = acc[110] + ABz * acc[38];
    const double h4_3_6 = acc[50] + ABz * acc[2];
    const double h4_6_6 = h10_3_6 + ABx * h4_3_6;
    const double h10_3_7 = acc[111] + ABz * acc[39];
    const double h4_3_7 = acc[51] + ABz * acc[3];
    const double h4_6_7 = h10_3_7 + ABx * h4_3_7;
    const double h10_3_8 = acc[112] + ABz * acc[40];
    const double h4_3_8 = acc[52] + ABz * acc[4];
    const double h4_6_8 = h10_3_8 + ABx * h4_3_8;
    const double h10_3_9 = acc[113] + ABz * acc[41];
    const double h4_3_9 = acc[53] + ABz * acc[5];
    const double h4_6_9 = h10_3_9 + ABx * h4_3_9;
    const double h11_2_4 = acc[114] + ABy * acc[42];
    const double h4_7_4 = h11_2_4 + ABy * h4_2_4;
    const double h11_2_5 = acc[115] + ABy * acc[43];
    const double h4_7_5 = h11_2_5 + ABy * h4_2_5;
    const double h11_2_6 = acc[116] + ABy * acc[44];
    const double h4_7_6 = h11_2_6 + ABy * h4_2_6;
    const double h11_2_7 = acc[117] + ABy * acc[45];
    const double h4_7_7 = h11_2_7 + ABy * h4_2_7;
    const double h11_2_8 = acc[118] + ABy * acc[46];
    const double h4_7_8 = h11_2_8 + ABy * h4_2_8;
    const double h11_2_9 = acc[119] + ABy * acc[47];
    const double h4_7_9 = h11_2_9 + ABy * h4_2_9;
    const double h11_3_4 = acc[120] + ABz * acc[42];
    const double h4_8_4 = h11_3_4 + ABy * h4_3_4;
    const double h11_3_5 = acc[121] + ABz * acc[43];
    const double h4_8_5 = h11_3_5 + ABy * h4_3_5;
    const double h11_3_6 = acc[122] + ABz * acc[44];
    const double h4_8_6 = h11_3_6 + ABy * h4_3_6;
    const double h11_3_7 = acc[123] + ABz * acc[45];
    const double h4_8_7 = h11_3_7 + ABy * h4_3_7;
    const double h11_3_8 = acc[124] + ABz * acc[46];
    const double h4_8_8 = h11_3_8 + ABy * h4_3_8;
    const double h11_3_9 = acc[125] + ABz * acc[47];
    const double h4_8_9 = h11_3_9 + ABy * h4_3_9;
    const double h12_3_4 = acc[126] + ABz * acc[48];
    const double h4_9_4 = h12_3_4 + ABz * h4_3_4;
    const double h12_3_5 = acc[127] + ABz * acc[49];
    const double h4_9_5 = h12_3_5 + ABz * h4_3_5;
    const double h12_3_6 = acc[128] + ABz * acc[50];
    const double h4_9_6 = h12_3_6 + ABz * h4_3_6;
    const double h12_3_7 = acc[129] + ABz * acc[51];
    const double h4_9_7 = h12_3_7 + ABz * h4_3_7;
    const double h12_3_8 = acc[130] + ABz * acc[52];
    const double h4_9_8 = h12_3_8 + ABz * h4_3_8;
    const double h12_3_9 = acc[131] + ABz * acc[53];
    const double h4_9_9 = h12_3_9 + ABz * h4_3_9;
    const double h11_1_4 = acc[102] + ABx * acc[42];
    const double h5_1_4 = acc[42] + ABx * acc[6];
    const double h5_4_4 = h11_1_4 + ABx * h5_1_4;
    const double h11_1_5 = acc[103] + ABx * acc[43];
    const double h5_1_5 = acc[43] + ABx * acc[7];
    const double h5_4_5 = h11_1_5 + ABx * h5_1_5;
    const double h11_1_6 = acc[104] + ABx * acc[44];
    const double h5_1_6 = acc[44] + ABx * acc[8];
    const double h5_4_6 = h11_1_6 + ABx * h5_1_6;
    const double h11_1_7 = acc[105] + ABx * acc[45];
    const double h5_1_7 = acc[45] + ABx * acc[9];
    const double h5_4_7 = h11_1_7 + ABx * h5_1_7;
    const double h11_1_8 = acc[106] + ABx * acc[46];
    const double h5_1_8 = acc[46] + ABx * acc[10];
    const double h5_4_8 = h11_1_8 + ABx * h5_1_8;
    const double h11_1_9 = acc[107] + ABx * acc[47];
    const double h5_1_9 = acc[47] + ABx * acc[11];
    const double h5_4_9 = h11_1_9 + ABx * h5_1_9;
    const double h5_2_4 = acc[54] + ABy * acc[6];
    const double h5_5_4 = h11_2_4 + ABx * h5_2_4;
    const double h5_2_5 = acc[55] + ABy * acc[7];
    const double h5_5_5 = h11_2_5 + ABx * h5_2_5;
    const double h5_2_6 = acc[56] + ABy * acc[8];
    const double h5_5_6 = h11_2_6 + ABx * h5_2_6;
    const double h5_2_7 = acc[57] + ABy * acc[9];
    const double h5_5_7 = h11_2_7 + ABx * h5_2_7;
    const double h5_2_8 = acc[58] + ABy * acc[10];
    const double h5_5_8 = h11_2_8 + ABx * h5_2_8;
    const double h5_2_9 = acc[59] + ABy * acc[11];
    const double h5_5_9 = h11_2_9 + ABx * h5_2_9;
    const double h5_3_4 = acc[66] + ABz * acc[6];
    const double h5_6_4 = h11_3_4 + ABx * h5_3_4;
    const double h5_3_5 = acc[67] + ABz * acc[7];
    const double h5_6_5 = h11_3_5 + ABx * h5_3_5;
    const double h5_3_6 = acc[68] + ABz * acc[8];
    const double h5_6_6 = h11_3_6 + ABx * h5_3_6;
    const double h5_3_7 = acc[69] + ABz * acc[9];
    const double h5_6_7 = h11_3_7 + ABx * h5_3_7;
    const double h5_3_8 = acc[70] + ABz * acc[10];
    const double h5_6_8 = h11_3_8 + ABx * h5_3_8;
    const double h5_3_9 = acc[71] + ABz * acc[11];
    const double h5_6_9 = h11_3_9 + ABx * h5_3_9;
    const double h13_2_4 = acc[132] + ABy * acc[54];
    const double h5_7_4 = h13_2_4 + ABy * h5_2_4;
    const double h13_2_5 = acc[133] + ABy * acc[55];
    const double h5_7_5 = h13_2_5 + ABy * h5_2_5;
    const double h13_2_6 = acc[134] + ABy * acc[56];
    const double h5_7_6 = h13_2_6 + ABy * h5_2_6;
    const double h13_2_7 = acc[135] + ABy * acc[57];
    const double h5_7_7 = h13_2_7 + ABy * h5_2_7;
    const double h13_2_8 = acc[136] + ABy * acc[58];
    const double h5_7_8 = h13_2_8 + ABy * h5_2_8;
    const double h13_2_9 = acc[137] + ABy * acc[59];
    const double h5_7_9 = h13_2_9 + ABy * h5_2_9;
    const double h13_3_4 = acc[138] + ABz * acc[54];
    const double h5_8_4 = h13_3_4 + ABy * h5_3_4;
    const double h13_3_5 = acc[139] + ABz * acc[55];
    const double h5_8_5 = h13_3_5 + ABy * h5_3_5;
    const double h13_3_6 = acc[140] + ABz * acc[56];
    const double h5_8_6 = h13_3_6 + ABy * h5_3_6;
    const double h13_3_7 = acc[141] + ABz * acc[57];
    const double h5_8_7 = h13_3_7 + ABy * h5_3_7;
    const double h13_3_8 = acc[142] + ABz * acc[58];
    const double h5_8_8 = h13_3_8 + ABy * h5_3_8;
    const double h13_3_9 = acc[143] + ABz * acc[59];
    const double h5_8_9 = h13_3_9 + ABy * h5_3_9;
    const double h15_3_4 = acc[144] + ABz * acc[66];
    const double h5_9_4 = h15_3_4 + ABz * h5_3_4;
    const double h15_3_5 = acc[145] + ABz * acc[67];
    const double h5_9_5 = h15_3_5 + ABz * h5_3_5;
    const double h15_3_6 = acc[146] + ABz * acc[68];
    const double h5_9_6 = h15_3_6 + ABz * h5_3_6;
    const double h15_3_7 = acc[147] + ABz * acc[69];
    const double h5_9_7 = h15_3_7 + ABz * h5_3_7;
    const double h15_3_8 = acc[148] + ABz * acc[70];
    const double h5_9_8 = h15_3_8 + ABz * h5_3_8;
    const double h15_3_9 = acc[149] + ABz * acc[71];
    const double h5_9_9 = h15_3_9 + ABz * h5_3_9;
    const double h12_1_4 = acc[108] + ABx * acc[48];
    const double h6_1_4 = acc[48] + ABx * acc[12];
    const double h6_4_4 = h12_1_4 + ABx * h6_1_4;
    const double h12_1_5 = acc[109] + ABx * acc[49];
    const double h6_1_5 = acc[49] + ABx * acc[13];
    const double h6_4_5 = h12_1_5 + ABx * h6_1_5;
    const double h12_1_6 = acc[110] + ABx * acc[50];
    const double h6_1_6 = acc[50] + ABx * acc[14];
    const double h6_4_6 = h12_1_6 + ABx * h6_1_6;
    const double h12_1_7 = acc[111] + ABx * acc[51];
    const double h6_1_7 = acc[51] + ABx * acc[15];
    const double h6_4_7 = h12_1_7 + ABx * h6_1_7;
    const double h12_1_8 = acc[112] + ABx * acc[52];
    const double h6_1_8 = acc[52] + ABx * acc[16];
    const double h6_4_8 = h12_1_8 + ABx * h6_1_8;
    const double h12_1_9 = acc[113] + ABx * acc[53];
    const double h6_1_9 = acc[53] + ABx * acc[17];
    const double h6_4_9 = h12_1_9 + ABx * h6_1_9;
    const double h12_2_4 = acc[120] + ABy * acc[48];
    const double h6_2_4 = acc[66] + ABy * acc[12];
    const double h6_5_4 = h12_2_4 + ABx * h6_2_4;
    const double h12_2_5 = acc[121] + ABy * acc[49];
    const double h6_2_5 = acc[67] + ABy * acc[13];
    const double h6_5_5 = h12_2_5 + ABx * h6_2_5;
    const double h12_2_6 = acc[122] + ABy * acc[50];
    const double h6_2_6 = acc[68] + ABy * acc[14];
    const double h6_5_6 = h12_2_6 + ABx * h6_2_6;
    const double h12_2_7 = acc[123] + ABy * acc[51];
    const double h6_2_7 = acc[69] + ABy * acc[15];
    const double h6_5_7 = h12_2_7 + ABx * h6_2_7;
    const double h12_2_8 = acc[124] + ABy * acc[52];
    const double h6_2_8 = acc[70] + ABy * acc[16];
    const double h6_5_8 = h12_2_8 + ABx * h6_2_8;
    const double h12_2_9 = acc[125] + ABy * acc[53];
    const double h6_2_9 = acc[71] + ABy * acc[17];
    const double h6_5_9 = h12_2_9 + ABx * h6_2_9;
    const double h6_3_4 = acc[60] + ABz * acc[12];
    const double h6_6_4 = h12_3_4 + ABx * h6_3_4;
    const double h6_3_5 = acc[61] + ABz * acc[13];
    const double h6_6_5 = h12_3_5 + ABx * h6_3_5;
    const double h6_3_6 = acc[62] + ABz * acc[14];
    const double h6_6_6 = h12_3_6 + ABx * h6_3_6;
    const double h6_3_7 = acc[63] + ABz * acc[15];
    const double h6_6_7 = h12_3_7 + ABx * h6_3_7;
    const double h6_3_8 = acc[64] + ABz * acc[16];
    const double h6_6_8 = h12_3_8 + ABx * h6_3_8;
    const double h6_3_9 = acc[65] + ABz * acc[17];
    const double h6_6_9 = h12_3_9 + ABx * h6_3_9;
    const double h15_2_4 = acc[138] + ABy * acc[66];
    const double h6_7_4 = h15_2_4 + ABy * h6_2_4;
    const double h15_2_5 = acc[139] + ABy * acc[67];
    const double h6_7_5 = h15_2_5 + ABy * h6_2_5;
    const double h15_2_6 = acc[140] + ABy * acc[68];
    const double h6_7_6 = h15_2_6 + ABy * h6_2_6;
    const double h15_2_7 = acc[141] + ABy * acc[69];
    const double h6_7_7 = h15_2_7 + ABy * h6_2_7;
    const double h15_2_8 = acc[142] + ABy * acc[70];
    const double h6_7_8 = h15_2_8 + ABy * h6_2_8;
    const double h15_2_9 = acc[143] + ABy * acc[71];
    const double h6_7_9 = h15_2_9 + ABy * h6_2_9;
    const double h6_8_4 = h15_3_4 + ABy * h6_3_4;
    const double h6_8_5 = h15_3_5 + ABy * h6_3_5;
    const double h6_8_6 = h15_3_6 + ABy * h6_3_6;
    const double h6_8_7 = h15_3_7 + ABy * h6_3_7;
    const double h6_8_8 = h15_3_8 + ABy * h6_3_8;
    const double h6_8_9 = h15_3_9 + ABy * h6_3_9;
    const double h14_3_4 = acc[150] + ABz * acc[60];
    const double h6_9_4 = h14_3_4 + ABz * h6_3_4;
    const double h14_3_5 = acc[151] + ABz * acc[61];
    const double h6_9_5 = h14_3_5 + ABz * h6_3_5;
    const double h14_3_6 = acc[152] + ABz * acc[62];
    const double h6_9_6 = h14_3_6 + ABz * h6_3_6;
    const double h14_3_7 = acc[153] + ABz * acc[63];
    const double h6_9_7 = h14_3_7 + ABz * h6_3_7;
    const double h14_3_8 = acc[154] + ABz * acc[64];
    const double h6_9_8 = h14_3_8 + ABz * h6_3_8;
    const double h14_3_9 = acc[155] + ABz * acc[65];
    const double h6_9_9 = h14_3_9 + ABz * h6_3_9;
    const double h13_1_4 = acc[114] + ABx * acc[54];
    const double h7_1_4 = acc[54] + ABx * acc[18];
    const double h7_4_4 = h13_1_4 + ABx * h7_1_4;
    const double h13_1_5 = acc[115] + ABx * acc[55];
    const double h7_1_5 = acc[55] + ABx * acc[19];
    const double h7_4_5 = h13_1_5 + ABx * h7_1_5;
    const double h13_1_6 = acc[116] + ABx * acc[56];
    const double h7_1_6 = acc[56] + ABx * acc[20];
    const double h7_4_6 = h13_1_6 + ABx * h7_1_6;
    const double h13_1_7 = acc[117] + ABx * acc[57];
    const double h7_1_7 = acc[57] + ABx * acc[21];
    const double h7_4_7 = h13_1_7 + ABx * h7_1_7;
    const double h13_1_8 = acc[118] + ABx * acc[58];
    const double h7_1_8 = acc[58] + ABx * acc[22];
    const double h7_4_8 = h13_1_8 + ABx * h7_1_8;
    const double h13_1_9 = acc[119] + ABx * acc[59];
    const double h7_1_9 = acc[59] + ABx * acc[23];
    const double h7_4_9 = h13_1_9 + ABx * h7_1_9;
    const double h7_2_4 = acc[72] + ABy * acc[18];
    const double h7_5_4 = h13_2_4 + ABx * h7_2_4;
    const double h7_2_5 = acc[73] + ABy * acc[19];
    const double h7_5_5 = h13_2_5 + ABx * h7_2_5;
    const double h7_2_6 = acc[74] + ABy * acc[20];
    const double h7_5_6 = h13_2_6 + ABx * h7_2_6;
    const double h7_2_7 = acc[75] + ABy * acc[21];
    const double h7_5_7 = h13_2_7 + ABx * h7_2_7;
    const double h7_2_8 = acc[76] + ABy * acc[22];
    const double h7_5_8 = h13_2_8 + ABx * h7_2_8;
    const double h7_2_9 = acc[77] + ABy * acc[23];
    const double h7_5_9 = h13_2_9 + ABx * h7_2_9;
    const double h7_3_4 = acc[78] + ABz * acc[18];
    const double h7_6_4 = h13_3_4 + ABx * h7_3_4;
    const double h7_3_5 = acc[79] + ABz * acc[19];
    const double h7_6_5 = h13_3_5 + ABx * h7_3_5;
    const double h7_3_6 = acc[80] + ABz * acc[20];
    const double h7_6_6 = h13_3_6 + ABx * h7_3_6;
    const double h7_3_7 = acc[81] + ABz * acc[21];
    const double h7_6_7 = h13_3_7 + ABx * h7_3_7;
    const double h7_3_8 = acc[82] + ABz * acc[22];
    const double h7_6_8 = h13_3_8 + ABx * h7_3_8;
    const double h7_3_9 = acc[83] + ABz * acc[23];
    const double h7_6_9 = h13_3_9 + ABx * h7_3_9;
    const double h16_2_4 = acc[156] + ABy * acc[72];
    const double h7_7_4 = h16_2_4 + ABy * h7_2_4;
    const double h16_2_5 = acc[157] + ABy * acc[73];
    const double h7_7_5 = h16_2_5 + ABy * h7_2_5;
    const double h16_2_6 = acc[158] + ABy * acc[74];
    const double h7_7_6 = h16_2_6 + ABy * h7_2_6;
    const double h16_2_7 = acc[159] + ABy * acc[75];
    const double h7_7_7 = h16_2_7 + ABy * h7_2_7;
    const double h16_2_8 = acc[160] + ABy * acc[76];
    const double h7_7_8 = h16_2_8 + ABy * h7_2_8;
    const double h16_2_9 = acc[161] + ABy * acc[77];
    const double h7_7_9 = h16_2_9 + ABy * h7_2_9;
    const double h16_3_4 = acc[162] + ABz * acc[72];
    const double h7_8_4 = h16_3_4 + ABy * h7_3_4;
    const double h16_3_5 = acc[163] + ABz * acc[73];
    const double h7_8_5 = h16_3_5 + ABy * h7_3_5;
    const double h16_3_6 = acc[164] + ABz * acc[74];
    const double h7_8_6 = h16_3_6 + ABy * h7_3_6;
    const double h16_3_7 = acc[165] + ABz * acc[75];
    const double h7_8_7 = h16_3_7 + ABy * h7_3_7;
    const double h16_3_8 = acc[166] + ABz * acc[76];
    const double h7_8_8 = h16_3_8 + ABy * h7_3_8;
    const double h16_3_9 = acc[167] + ABz * acc[77];
    const double h7_8_9 = h16_3_9 + ABy * h7_3_9;
    const double h17_3_4 = acc[168] + ABz * acc[78];
    const double h7_9_4 = h17_3_4 + ABz * h7_3_4;
    const double h17_3_5 = acc[169] + ABz * acc[79];
    const double h7_9_5 = h17_3_5 + ABz * h7_3_5;
    const double h17_3_6 = acc[170] + ABz * acc[80];
    const double h7_9_6 = h17_3_6 + ABz * h7_3_6;
    const double h17_3_7 = acc[171] + ABz * acc[81];
    const double h7_9_7 = h17_3_7 + ABz * h7_3_7;
    const double h17_3_8 = acc[172] + ABz * acc[82];
    const double h7_9_8 = h17_3_8 + ABz * h7_3_8;
    const double h17_3_9 = acc[173] + ABz * acc[83];
    const double h7_9_9 = h17_3_9 + ABz * h7_3_9;
    const double h15_1_4 = acc[120] + ABx * acc[66];
    const double h8_1_4 = acc[66] + ABx * acc[24];
    const double h8_4_4 = h15_1_4 + ABx * h8_1_4;
    const double h15_1_5 = acc[121] + ABx * acc[67];
    const double h8_1_5 = acc[67] + ABx * acc[25];
    const double h8_4_5 = h15_1_5 + ABx * h8_1_5;
    const double h15_1_6 = acc[122] + ABx * acc[68];
    const double h8_1_6 = acc[68] + ABx * acc[26];
    const double h8_4_6 = h15_1_6 + ABx * h8_1_6;
    const double h15_1_7 = acc[123] + ABx * acc[69];
    const double h8_1_7 = acc[69] + ABx * acc[27];
    const double h8_4_7 = h15_1_7 + ABx * h8_1_7;
    const double h15_1_8 = acc[124] + ABx * acc[70];
    const double h8_1_8 = acc[70] + ABx * acc[28];
    const double h8_4_8 = h15_1_8 + ABx * h8_1_8;
    const double h15_1_9 = acc[125] + ABx * acc[71];
    const double h8_1_9 = acc[71] + ABx * acc[29];
    const double h8_4_9 = h15_1_9 + ABx * h8_1_9;
    const double h8_2_4 = acc[78] + ABy * acc[24];
    const double h8_5_4 = h15_2_4 + ABx * h8_2_4;
    const double h8_2_5 = acc[79] + ABy * acc[25];
    const double h8_5_5 = h15_2_5 + ABx * h8_2_5;
    const double h8_2_6 = acc[80] + ABy * acc[26];
    const double h8_5_6 = h15_2_6 + ABx * h8_2_6;
    const double h8_2_7 = acc[81] + ABy * acc[27];
    const double h8_5_7 = h15_2_7 + ABx * h8_2_7;
    const double h8_2_8 = acc[82] + ABy * acc[28];
    const double h8_5_8 = h15_2_8 + ABx * h8_2_8;
    const double h8_2_9 = acc[83] + ABy * acc[29];
    const double h8_5_9 = h15_2_9 + ABx * h8_2_9;
    const double h8_3_4 = acc[84] + ABz * acc[24];
    const double h8_6_4 = h15_3_4 + ABx * h8_3_4;
    const double h8_3_5 = acc[85] + ABz * acc[25];
    const double h8_6_5 = h15_3_5 + ABx * h8_3_5;
    const double h8_3_6 = acc[86] + ABz * acc[26];
    const double h8_6_6 = h15_3_6 + ABx * h8_3_6;
    const double h8_3_7 = acc[87] + ABz * acc[27];
    const double h8_6_7 = h15_3_7 + ABx * h8_3_7;
    const double h8_3_8 = acc[88] + ABz * acc[28];
    const double h8_6_8 = h15_3_8 + ABx * h8_3_8;
    const double h8_3_9 = acc[89] + ABz * acc[29];
    const double h8_6_9 = h15_3_9 + ABx * h8_3_9;
    const double h17_2_4 = acc[162] + ABy * acc[78];
    const double h8_7_4 = h17_2_4 + ABy * h8_2_4;
    const double h17_2_5 = acc[163] + ABy * acc[79];
    const double h8_7_5 = h17_2_5 + ABy * h8_2_5;
    const double h17_2_6 = acc[164] + ABy * acc[80];
    const double h8_7_6 = h17_2_6 + ABy * h8_2_6;
    const double h17_2_7 = acc[165] + ABy * acc[81];
    const double h8_7_7 = h17_2_7 + ABy * h8_2_7;
    const double h17_2_8 = acc[166] + ABy * acc[82];
    const double h8_7_8 = h17_2_8 + ABy * h8_2_8;
    const double h17_2_9 = acc[167] + ABy * acc[83];
    const double h8_7_9 = h17_2_9 + ABy * h8_2_9;
    const double h8_8_4 = h17_3_4 + ABy * h8_3_4;
    const double h8_8_5 = h17_3_5 + ABy * h8_3_5;
    const double h8_8_6 = h17_3_6 + ABy * h8_3_6;
    const double h8_8_7 = h17_3_7 + ABy * h8_3_7;
    const double h8_8_8 = h17_3_8 + ABy * h8_3_8;
    const double h8_8_9 = h17_3_9 + ABy * h8_3_9;
    const double h18_3_4 = acc[174] + ABz * acc[84];
    const double h8_9_4 = h18_3_4 + ABz * h8_3_4;
    const double h18_3_5 = acc[175] + ABz * acc[85];
    const double h8_9_5 = h18_3_5 + ABz * h8_3_5;
    const double h18_3_6 = acc[176] + ABz * acc[86];
    const double h8_9_6 = h18_3_6 + ABz * h8_3_6;
    const double h18_3_7 = acc[177] + ABz * acc[87];
    const double h8_9_7 = h18_3_7 + ABz * h8_3_7;
    const double h18_3_8 = acc[178] + ABz * acc[88];
    const double h8_9_8 = h18_3_8 + ABz * h8_3_8;
    const double h18_3_9 = acc[179] + ABz * acc[89];
    const double h8_9_9 = h18_3_9 + ABz * h8_3_9;
    const double h14_1_4 = acc[126] + ABx * acc[60];
    const double h9_1_4 = acc[60] + ABx * acc[30];
    const double h9_4_4 = h14_1_4 + ABx * h9_1_4;
    const double h14_1_5 = acc[127] + ABx * acc[61];
    const double h9_1_5 = acc[61] + ABx * acc[31];
    const double h9_4_5 = h14_1_5 + ABx * h9_1_5;
    const double h14_1_6 = acc[128] + ABx * acc[62];
    const double h9_1_6 = acc[62] + ABx * acc[32];
    const double h9_4_6 = h14_1_6 + ABx * h9_1_6;
    const double h14_1_7 = acc[129] + ABx * acc[63];
    const double h9_1_7 = acc[63] + ABx * acc[33];
    const double h9_4_7 = h14_1_7 + ABx * h9_1_7;
    const double h14_1_8 = acc[130] + ABx * acc[64];
    const double h9_1_8 = acc[64] + ABx * acc[34];
    const double h9_4_8 = h14_1_8 + ABx * h9_1_8;
    const double h14_1_9 = acc[131] + ABx * acc[65];
    const double h9_1_9 = acc[65] + ABx * acc[35];
    const double h9_4_9 = h14_1_9 + ABx * h9_1_9;
    const double h14_2_4 = acc[144] + ABy * acc[60];
    const double h9_2_4 = acc[84] + ABy * acc[30];
    const double h9_5_4 = h14_2_4 + ABx * h9_2_4;
    const double h14_2_5 = acc[145] + ABy * acc[61];
    const double h9_2_5 = acc[85] + ABy * acc[31];
    const double h9_5_5 = h14_2_5 + ABx * h9_2_5;
    const double h14_2_6 = acc[146] + ABy * acc[62];
    const double h9_2_6 = acc[86] + ABy * acc[32];
    const double h9_5_6 = h14_2_6 + ABx * h9_2_6;
    const double h14_2_7 = acc[147] + ABy * acc[63];
    const double h9_2_7 = acc[87] + ABy * acc[33];
    const double h9_5_7 = h14_2_7 + ABx * h9_2_7;
    const double h14_2_8 = acc[148] + ABy * acc[64];
    const double h9_2_8 = acc[88] + ABy * acc[34];
    const double h9_5_8 = h14_2_8 + ABx * h9_2_8;
    const double h14_2_9 = acc[149] + ABy * acc[65];
    const double h9_2_9 = acc[89] + ABy * acc[35];
    const double h9_5_9 = h14_2_9 + ABx * h9_2_9;
    const double h9_3_4 = acc[90] + ABz * acc[30];
    const double h9_6_4 = h14_3_4 + ABx * h9_3_4;
    const double h9_3_5 = acc[91] + ABz * acc[31];
    const double h9_6_5 = h14_3_5 + ABx * h9_3_5;
    const double h9_3_6 = acc[92] + ABz * acc[32];
    const double h9_6_6 = h14_3_6 + ABx * h9_3_6;
    const double h9_3_7 = acc[93] + ABz * acc[33];
    const double h9_6_7 = h14_3_7 + ABx * h9_3_7;
    const double h9_3_8 = acc[94] + ABz * acc[34];
    const double h9_6_8 = h14_3_8 + ABx * h9_3_8;
    const double h9_3_9 = acc[95] + ABz * acc[35];
    const double h9_6_9 = h14_3_9 + ABx * h9_3_9;
    const double h18_2_4 = acc[168] + ABy * acc[84];
    const double h9_7_4 = h18_2_4 + ABy * h9_2_4;
    const double h18_2_5 = acc[169] + ABy * acc[85];
    const double h9_7_5 = h18_2_5 + ABy * h9_2_5;
    const double h18_2_6 = acc[170] + ABy * acc[86];
    const double h9_7_6 = h18_2_6 + ABy * h9_2_6;
    const double h18_2_7 = acc[171] + ABy * acc[87];
    const double h9_7_7 = h18_2_7 + ABy * h9_2_7;
    const double h18_2_8 = acc[172] + ABy * acc[88];
    const double h9_7_8 = h18_2_8 + ABy * h9_2_8;
    const double h18_2_9 = acc[173] + ABy * acc[89];
    const double h9_7_9 = h18_2_9 + ABy * h9_2_9;
    const double h9_8_4 = h18_3_4 + ABy * h9_3_4;
    const double h9_8_5 = h18_3_5 + ABy * h9_3_5;
    const double h9_8_6 = h18_3_6 + ABy * h9_3_6;
    const double h9_8_7 = h18_3_7 + ABy * h9_3_7;
    const double h9_8_8 = h18_3_8 + ABy * h9_3_8;
    const double h9_8_9 = h18_3_9 + ABy * h9_3_9;
    const double h19_3_4 = acc[180] + ABz * acc[90];
    const double h9_9_4 = h19_3_4 + ABz * h9_3_4;
    const double h19_3_5 = acc[181] + ABz * acc[91];
    const double h9_9_5 = h19_3_5 + ABz * h9_3_5;
    const double h19_3_6 = acc[182] + ABz * acc[92];
    const double h9_9_6 = h19_3_6 + ABz * h9_3_6;
    const double h19_3_7 = acc[183] + ABz * acc[93];
    const double h9_9_7 = h19_3_7 + ABz * h9_3_7;
    const double h19_3_8 = acc[184] + ABz * acc[94];
    const double h9_9_8 = h19_3_8 + ABz * h9_3_8;
    const double h19_3_9 = acc[185] + ABz * acc[95];
    const double h9_9_9 = h19_3_9 + ABz * h9_3_9;
    res[0] = h4_4_4 * 0.19245008972987535;
    res[1] = h4_4_5 * 0.3333333333333334;
    res[2] = h4_4_6 * 0.3333333333333334;
    res[3] = h4_4_7 * 0.19245008972987535;
    res[4] = h4_4_8 * 0.3333333333333334;
    res[5] = h4_4_9 * 0.19245008972987535;
    res[6] = h4_5_4 * 0.3333333333333334;
    res[7] = h4_5_5 * 0.5773502691896258;
    res[8] = h4_5_6 * 0.5773502691896258;
    res[9] = h4_5_7 * 0.3333333333333334;
    res[10] = h4_5_8 * 0.5773502691896258;
    res[11] = h4_5_9 * 0.3333333333333334;
    res[12] = h4_6_4 * 0.3333333333333334;
    res[13] = h4_6_5 * 0.5773502691896258;
    res[14] = h4_6_6 * 0.5773502691896258;
    res[15] = h4_6_7 * 0.3333333333333334;
    res[16] = h4_6_8 * 0.5773502691896258;
    res[17] = h4_6_9 * 0.3333333333333334;
    res[18] = h4_7_4 * 0.19245008972987535;
    res[19] = h4_7_5 * 0.3333333333333334;
    res[20] = h4_7_6 * 0.3333333333333334;
    res[21] = h4_7_7 * 0.19245008972987535;
    res[22] = h4_7_8 * 0.3333333333333334;
    res[23] = h4_7_9 * 0.19245008972987535;
    res[24] = h4_8_4 * 0.3333333333333334;
    res[25] = h4_8_5 * 0.5773502691896258;
    res[26] = h4_8_6 * 0.5773502691896258;
    res[27] = h4_8_7 * 0.3333333333333334;
    res[28] = h4_8_8 * 0.5773502691896258;
    res[29] = h4_8_9 * 0.3333333333333334;
    res[30] = h4_9_4 * 0.19245008972987535;
    res[31] = h4_9_5 * 0.3333333333333334;
    res[32] = h4_9_6 * 0.3333333333333334;
    res[33] = h4_9_7 * 0.19245008972987535;
    res[34] = h4_9_8 * 0.3333333333333334;
    res[35] = h4_9_9 * 0.19245008972987535;
    res[36] = h5_4_4 * 0.3333333333333334;
    res[37] = h5_4_5 * 0.5773502691896258;
    res[38] = h5_4_6 * 0.5773502691896258;
    res[39] = h5_4_7 * 0.3333333333333334;
    res[40] = h5_4_8 * 0.5773502691896258;
    res[41] = h5_4_9 * 0.3333333333333334;
    res[42] = h5_5_4 * 0.5773502691896258;
    res[43] = h5_5_5;
    res[44] = h5_5_6;
    res[45] = h5_5_7 * 0.5773502691896258;
    res[46] = h5_5_8;
    res[47] = h5_5_9 * 0.5773502691896258;
    res[48] = h5_6_4 * 0.5773502691896258;
    res[49] = h5_6_5;
    res[50] = h5_6_6;
    res[51] = h5_6_7 * 0.5773502691896258;
    res[52] = h5_6_8;
    res[53] = h5_6_9 * 0.5773502691896258;
    res[54] = h5_7_4 * 0.3333333333333334;
    res[55] = h5_7_5 * 0.5773502691896258;
    res[56] = h5_7_6 * 0.5773502691896258;
    res[57] = h5_7_7 * 0.3333333333333334;
    res[58] = h5_7_8 * 0.5773502691896258;
    res[59] = h5_7_9 * 0.3333333333333334;
    res[60] = h5_8_4 * 0.5773502691896258;
    res[61] = h5_8_5;
    res[62] = h5_8_6;
    res[63] = h5_8_7 * 0.5773502691896258;
    res[64] = h5_8_8;
    res[65] = h5_8_9 * 0.5773502691896258;
    res[66] = h5_9_4 * 0.3333333333333334;
    res[67] = h5_9_5 * 0.5773502691896258;
    res[68] = h5_9_6 * 0.5773502691896258;
    res[69] = h5_9_7 * 0.3333333333333334;
    res[70] = h5_9_8 * 0.5773502691896258;
    res[71] = h5_9_9 * 0.3333333333333334;
    res[72] = h6_4_4 * 0.3333333333333334;
    res[73] = h6_4_5 * 0.5773502691896258;
    res[74] = h6_4_6 * 0.5773502691896258;
    res[75] = h6_4_7 * 0.3333333333333334;
    res[76] = h6_4_8 * 0.5773502691896258;
    res[77] = h6_4_9 * 0.3333333333333334;
    res[78] = h6_5_4 * 0.5773502691896258;
    res[79] = h6_5_5;
    res[80] = h6_5_6;
    res[81] = h6_5_7 * 0.5773502691896258;
    res[82] = h6_5_8;
    res[83] = h6_5_9 * 0.5773502691896258;
    res[84] = h6_6_4 * 0.5773502691896258;
    res[85] = h6_6_5;
    res[86] = h6_6_6;
    res[87] = h6_6_7 * 0.5773502691896258;
    res[88] = h6_6_8;
    res[89] = h6_6_9 * 0.5773502691896258;
    res[90] = h6_7_4 * 0.3333333333333334;
    res[91] = h6_7_5 * 0.5773502691896258;
    res[92] = h6_7_6 * 0.5773502691896258;
    res[93] = h6_7_7 * 0.3333333333333334;
    res[94] = h6_7_8 * 0.5773502691896258;
    res[95] = h6_7_9 * 0.3333333333333334;
    res[96] = h6_8_4 * 0.5773502691896258;
    res[97] = h6_8_5;
    res[98] = h6_8_6;
    res[99] = h6_8_7 * 0.5773502691896258;
    res[100] = h6_8_8;
    res[101] = h6_8_9 * 0.5773502691896258;
    res[102] = h6_9_4 * 0.3333333333333334;
    res[103] = h6_9_5 * 0.5773502691896258;
    res[104] = h6_9_6 * 0.5773502691896258;
    res[105] = h6_9_7 * 0.3333333333333334;
    res[106] = h6_9_8 * 0.5773502691896258;
    res[107] = h6_9_9 * 0.3333333333333334;
    res[108] = h7_4_4 * 0.19245008972987535;
    res[109] = h7_4_5 * 0.3333333333333334;
    res[110] = h7_4_6 * 0.3333333333333334;
    res[111] = h7_4_7 * 0.19245008972987535;
    res[112] = h7_4_8 * 0.3333333333333334;
    res[113] = h7_4_9 * 0.19245008972987535;
    res[114] = h7_5_4 * 0.3333333333333334;
    res[115] = h7_5_5 * 0.5773502691896258;
    res[116] = h7_5_6 * 0.5773502691896258;
    res[117] = h7_5_7 * 0.3333333333333334;
    res[118] = h7_5_8 * 0.5773502691896258;
    res[119] = h7_5_9 * 0.3333333333333334;
    res[120] = h7_6_4 * 0.3333333333333334;
    res[121] = h7_6_5 * 0.5773502691896258;
    res[122] = h7_6_6 * 0.5773502691896258;
    res[123] = h7_6_7 * 0.3333333333333334;
    res[124] = h7_6_8 * 0.5773502691896258;
    res[125] = h7_6_9 * 0.3333333333333334;
    res[126] = h7_7_4 * 0.19245008972987535;
    res[127] = h7_7_5 * 0.3333333333333334;
    res[128] = h7_7_6 * 0.3333333333333334;
    res[129] = h7_7_7 * 0.19245008972987535;
    res[130] = h7_7_8 * 0.3333333333333334;
    res[131] = h7_7_9 * 0.19245008972987535;
    res[132] = h7_8_4 * 0.3333333333333334;
    res[133] = h7_8_5 * 0.5773502691896258;
    res[134] = h7_8_6 * 0.5773502691896258;
    res[135] = h7_8_7 * 0.3333333333333334;
    res[136] = h7_8_8 * 0.5773502691896258;
    res[137] = h7_8_9 * 0.3333333333333334;
    res[138] = h7_9_4 * 0.19245008972987535;
    res[139] = h7_9_5 * 0.3333333333333334;
    res[140] = h7_9_6 * 0.3333333333333334;
    res[141] = h7_9_7 * 0.19245008972987535;
    res[142] = h7_9_8 * 0.3333333333333334;
    res[143] = h7_9_9 * 0.19245008972987535;
    res[144] = h8_4_4 * 0.3333333333333334;
    res[145] = h8_4_5 * 0.5773502691896258;
    res[146] = h8_4_6 * 0.5773502691896258;
    res[147] = h8_4_7 * 0.3333333333333334;
    res[148] = h8_4_8 * 0.5773502691896258;
    res[149] = h8_4_9 * 0.3333333333333334;
    res[150] = h8_5_4 * 0.5773502691896258;
    res[151] = h8_5_5;
    res[152] = h8_5_6;
    res[153] = h8_5_7 * 0.5773502691896258;
    res[154] = h8_5_8;
    res[155] = h8_5_9 * 0.5773502691896258;
    res[156] = h8_6_4 * 0.5773502691896258;
    res[157] = h8_6_5;
    res[158] = h8_6_6;
    res[159] = h8_6_7 * 0.5773502691896258;
    res[160] = h8_6_8;
    res[161] = h8_6_9 * 0.5773502691896258;
    res[162] = h8_7_4 * 0.3333333333333334;
    res[163] = h8_7_5 * 0.5773502691896258;
    res[164] = h8_7_6 * 0.5773502691896258;
    res[165] = h8_7_7 * 0.3333333333333334;
    res[166] = h8_7_8 * 0.5773502691896258;
    res[167] = h8_7_9 * 0.3333333333333334;
    res[168] = h8_8_4 * 0.5773502691896258;
    res[169] = h8_8_5;
    res[170] = h8_8_6;
    res[171] = h8_8_7 * 0.5773502691896258;
    res[172] = h8_8_8;
    res[173] = h8_8_9 * 0.5773502691896258;
    res[174] = h8_9_4 * 0.3333333333333334;
    res[175] = h8_9_5 * 0.5773502691896258;
    res[176] = h8_9_6 * 0.5773502691896258;
    res[177] = h8_9_7 * 0.3333333333333334;
    res[178] = h8_9_8 * 0.5773502691896258;
    res[179] = h8_9_9 * 0.3333333333333334;
    res[180] = h9_4_4 * 0.19245008972987535;
    res[181] = h9_4_5 * 0.3333333333333334;
    res[182] = h9_4_6 * 0.3333333333333334;
    res[183] = h9_4_7 * 0.19245008972987535;
    res[184] = h9_4_8 * 0.3333333333333334;
    res[185] = h9_4_9 * 0.19245008972987535;
    res[186] = h9_5_4 * 0.3333333333333334;
    res[187] = h9_5_5 * 0.5773502691896258;
    res[188] = h9_5_6 * 0.5773502691896258;
    res[189] = h9_5_7 * 0.3333333333333334;
    res[190] = h9_5_8 * 0.5773502691896258;
    res[191] = h9_5_9 * 0.3333333333333334;
    res[192] = h9_6_4 * 0.3333333333333334;
    res[193] = h9_6_5 * 0.5773502691896258;
    res[194] = h9_6_6 * 0.5773502691896258;
    res[195] = h9_6_7 * 0.3333333333333334;
    res[196] = h9_6_8 * 0.5773502691896258;
    res[197] = h9_6_9 * 0.3333333333333334;
    res[198] = h9_7_4 * 0.19245008972987535;
    res[199] = h9_7_5 * 0.3333333333333334;
    res[200] = h9_7_6 * 0.3333333333333334;
    res[201] = h9_7_7 * 0.19245008972987535;
    res[202] = h9_7_8 * 0.3333333333333334;
    res[203] = h9_7_9 * 0.19245008972987535;
    res[204] = h9_8_4 * 0.3333333333333334;
    res[205] = h9_8_5 * 0.5773502691896258;
    res[206] = h9_8_6 * 0.5773502691896258;
    res[207] = h9_8_7 * 0.3333333333333334;
    res[208] = h9_8_8 * 0.5773502691896258;
    res[209] = h9_8_9 * 0.3333333333333334;
    res[210] = h9_9_4 * 0.19245008972987535;
    res[211] = h9_9_5 * 0.3333333333333334;
    res[212] = h9_9_6 * 0.3333333333333334;
    res[213] = h9_9_7 * 0.19245008972987535;
    res[214] = h9_9_8 * 0.3333333333333334;
    res[215] = h9_9_9 * 0.19245008972987535;
}

// (ab|cd) over the bra primitive pairs [i0, i1) and ket primitive pairs [j0, j1) into
// res[216]; the contracted block also into acc_out when given (the bound kernels).
template <typename VT>
__device__ __forceinline__ void quartet_ddds(const PairTab &P, const BoysTab &B, int p, int q,
                                              int i0, int i1, int j0, int j1,
                                              double *__restrict__ res,
                                              double *__restrict__ acc_out = nullptr) {
    double acc[186];
    vrr_ddds<VT>(P, B, p, q, i0, i1, 1, j0, j1, 1, acc);
    if (acc_out) {
#pragma unroll
        for (int x = 0; x < 186; ++x) acc_out[x] = acc[x];
    }
    hrr_ddds(P, p, q, acc, res);
}

__device__ __forceinline__ void store_ddds(double *__restrict__ out, const int4 ib_, const int4 ik_,
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
    const long long kl_3_0 = pair_index(ik_.z + 3, ik_.w + 0);
    const long long kl_4_0 = pair_index(ik_.z + 4, ik_.w + 0);
    const long long kl_5_0 = pair_index(ik_.z + 5, ik_.w + 0);
    { const long long ij = ij_0_0, kl = kl_0_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[0]; }
    { const long long ij = ij_0_0, kl = kl_1_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[1]; }
    { const long long ij = ij_0_0, kl = kl_2_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[2]; }
    { const long long ij = ij_0_0, kl = kl_3_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[3]; }
    { const long long ij = ij_0_0, kl = kl_4_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[4]; }
    { const long long ij = ij_0_0, kl = kl_5_0;
      if ((!dab || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[5]; }
    { const long long ij = ij_0_1, kl = kl_0_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[6]; }
    { const long long ij = ij_0_1, kl = kl_1_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[7]; }
    { const long long ij = ij_0_1, kl = kl_2_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[8]; }
    { const long long ij = ij_0_1, kl = kl_3_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[9]; }
    { const long long ij = ij_0_1, kl = kl_4_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[10]; }
    { const long long ij = ij_0_1, kl = kl_5_0;
      if ((!dab || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[11]; }
    { const long long ij = ij_0_2, kl = kl_0_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[12]; }
    { const long long ij = ij_0_2, kl = kl_1_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[13]; }
    { const long long ij = ij_0_2, kl = kl_2_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[14]; }
    { const long long ij = ij_0_2, kl = kl_3_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[15]; }
    { const long long ij = ij_0_2, kl = kl_4_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[16]; }
    { const long long ij = ij_0_2, kl = kl_5_0;
      if ((!dab || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[17]; }
    { const long long ij = ij_0_3, kl = kl_0_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[18]; }
    { const long long ij = ij_0_3, kl = kl_1_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[19]; }
    { const long long ij = ij_0_3, kl = kl_2_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[20]; }
    { const long long ij = ij_0_3, kl = kl_3_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[21]; }
    { const long long ij = ij_0_3, kl = kl_4_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[22]; }
    { const long long ij = ij_0_3, kl = kl_5_0;
      if ((!dab || 0 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[23]; }
    { const long long ij = ij_0_4, kl = kl_0_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[24]; }
    { const long long ij = ij_0_4, kl = kl_1_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[25]; }
    { const long long ij = ij_0_4, kl = kl_2_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[26]; }
    { const long long ij = ij_0_4, kl = kl_3_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[27]; }
    { const long long ij = ij_0_4, kl = kl_4_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[28]; }
    { const long long ij = ij_0_4, kl = kl_5_0;
      if ((!dab || 0 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[29]; }
    { const long long ij = ij_0_5, kl = kl_0_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[30]; }
    { const long long ij = ij_0_5, kl = kl_1_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[31]; }
    { const long long ij = ij_0_5, kl = kl_2_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[32]; }
    { const long long ij = ij_0_5, kl = kl_3_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[33]; }
    { const long long ij = ij_0_5, kl = kl_4_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[34]; }
    { const long long ij = ij_0_5, kl = kl_5_0;
      if ((!dab || 0 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[35]; }
    { const long long ij = ij_1_0, kl = kl_0_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[36]; }
    { const long long ij = ij_1_0, kl = kl_1_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[37]; }
    { const long long ij = ij_1_0, kl = kl_2_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[38]; }
    { const long long ij = ij_1_0, kl = kl_3_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[39]; }
    { const long long ij = ij_1_0, kl = kl_4_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[40]; }
    { const long long ij = ij_1_0, kl = kl_5_0;
      if ((!dab || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[41]; }
    { const long long ij = ij_1_1, kl = kl_0_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[42]; }
    { const long long ij = ij_1_1, kl = kl_1_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[43]; }
    { const long long ij = ij_1_1, kl = kl_2_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[44]; }
    { const long long ij = ij_1_1, kl = kl_3_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[45]; }
    { const long long ij = ij_1_1, kl = kl_4_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[46]; }
    { const long long ij = ij_1_1, kl = kl_5_0;
      if ((!dab || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[47]; }
    { const long long ij = ij_1_2, kl = kl_0_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[48]; }
    { const long long ij = ij_1_2, kl = kl_1_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[49]; }
    { const long long ij = ij_1_2, kl = kl_2_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[50]; }
    { const long long ij = ij_1_2, kl = kl_3_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[51]; }
    { const long long ij = ij_1_2, kl = kl_4_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[52]; }
    { const long long ij = ij_1_2, kl = kl_5_0;
      if ((!dab || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[53]; }
    { const long long ij = ij_1_3, kl = kl_0_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[54]; }
    { const long long ij = ij_1_3, kl = kl_1_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[55]; }
    { const long long ij = ij_1_3, kl = kl_2_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[56]; }
    { const long long ij = ij_1_3, kl = kl_3_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[57]; }
    { const long long ij = ij_1_3, kl = kl_4_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[58]; }
    { const long long ij = ij_1_3, kl = kl_5_0;
      if ((!dab || 1 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[59]; }
    { const long long ij = ij_1_4, kl = kl_0_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[60]; }
    { const long long ij = ij_1_4, kl = kl_1_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[61]; }
    { const long long ij = ij_1_4, kl = kl_2_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[62]; }
    { const long long ij = ij_1_4, kl = kl_3_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[63]; }
    { const long long ij = ij_1_4, kl = kl_4_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[64]; }
    { const long long ij = ij_1_4, kl = kl_5_0;
      if ((!dab || 1 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[65]; }
    { const long long ij = ij_1_5, kl = kl_0_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[66]; }
    { const long long ij = ij_1_5, kl = kl_1_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[67]; }
    { const long long ij = ij_1_5, kl = kl_2_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[68]; }
    { const long long ij = ij_1_5, kl = kl_3_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[69]; }
    { const long long ij = ij_1_5, kl = kl_4_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[70]; }
    { const long long ij = ij_1_5, kl = kl_5_0;
      if ((!dab || 1 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[71]; }
    { const long long ij = ij_2_0, kl = kl_0_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[72]; }
    { const long long ij = ij_2_0, kl = kl_1_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[73]; }
    { const long long ij = ij_2_0, kl = kl_2_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[74]; }
    { const long long ij = ij_2_0, kl = kl_3_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[75]; }
    { const long long ij = ij_2_0, kl = kl_4_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[76]; }
    { const long long ij = ij_2_0, kl = kl_5_0;
      if ((!dab || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[77]; }
    { const long long ij = ij_2_1, kl = kl_0_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[78]; }
    { const long long ij = ij_2_1, kl = kl_1_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[79]; }
    { const long long ij = ij_2_1, kl = kl_2_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[80]; }
    { const long long ij = ij_2_1, kl = kl_3_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[81]; }
    { const long long ij = ij_2_1, kl = kl_4_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[82]; }
    { const long long ij = ij_2_1, kl = kl_5_0;
      if ((!dab || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[83]; }
    { const long long ij = ij_2_2, kl = kl_0_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[84]; }
    { const long long ij = ij_2_2, kl = kl_1_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[85]; }
    { const long long ij = ij_2_2, kl = kl_2_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[86]; }
    { const long long ij = ij_2_2, kl = kl_3_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[87]; }
    { const long long ij = ij_2_2, kl = kl_4_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[88]; }
    { const long long ij = ij_2_2, kl = kl_5_0;
      if ((!dab || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[89]; }
    { const long long ij = ij_2_3, kl = kl_0_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[90]; }
    { const long long ij = ij_2_3, kl = kl_1_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[91]; }
    { const long long ij = ij_2_3, kl = kl_2_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[92]; }
    { const long long ij = ij_2_3, kl = kl_3_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[93]; }
    { const long long ij = ij_2_3, kl = kl_4_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[94]; }
    { const long long ij = ij_2_3, kl = kl_5_0;
      if ((!dab || 2 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[95]; }
    { const long long ij = ij_2_4, kl = kl_0_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[96]; }
    { const long long ij = ij_2_4, kl = kl_1_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[97]; }
    { const long long ij = ij_2_4, kl = kl_2_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[98]; }
    { const long long ij = ij_2_4, kl = kl_3_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[99]; }
    { const long long ij = ij_2_4, kl = kl_4_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[100]; }
    { const long long ij = ij_2_4, kl = kl_5_0;
      if ((!dab || 2 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[101]; }
    { const long long ij = ij_2_5, kl = kl_0_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[102]; }
    { const long long ij = ij_2_5, kl = kl_1_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[103]; }
    { const long long ij = ij_2_5, kl = kl_2_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[104]; }
    { const long long ij = ij_2_5, kl = kl_3_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[105]; }
    { const long long ij = ij_2_5, kl = kl_4_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[106]; }
    { const long long ij = ij_2_5, kl = kl_5_0;
      if ((!dab || 2 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[107]; }
    { const long long ij = ij_3_0, kl = kl_0_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[108]; }
    { const long long ij = ij_3_0, kl = kl_1_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[109]; }
    { const long long ij = ij_3_0, kl = kl_2_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[110]; }
    { const long long ij = ij_3_0, kl = kl_3_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[111]; }
    { const long long ij = ij_3_0, kl = kl_4_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[112]; }
    { const long long ij = ij_3_0, kl = kl_5_0;
      if ((!dab || 3 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[113]; }
    { const long long ij = ij_3_1, kl = kl_0_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[114]; }
    { const long long ij = ij_3_1, kl = kl_1_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[115]; }
    { const long long ij = ij_3_1, kl = kl_2_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[116]; }
    { const long long ij = ij_3_1, kl = kl_3_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[117]; }
    { const long long ij = ij_3_1, kl = kl_4_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[118]; }
    { const long long ij = ij_3_1, kl = kl_5_0;
      if ((!dab || 3 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[119]; }
    { const long long ij = ij_3_2, kl = kl_0_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[120]; }
    { const long long ij = ij_3_2, kl = kl_1_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[121]; }
    { const long long ij = ij_3_2, kl = kl_2_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[122]; }
    { const long long ij = ij_3_2, kl = kl_3_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[123]; }
    { const long long ij = ij_3_2, kl = kl_4_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[124]; }
    { const long long ij = ij_3_2, kl = kl_5_0;
      if ((!dab || 3 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[125]; }
    { const long long ij = ij_3_3, kl = kl_0_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[126]; }
    { const long long ij = ij_3_3, kl = kl_1_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[127]; }
    { const long long ij = ij_3_3, kl = kl_2_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[128]; }
    { const long long ij = ij_3_3, kl = kl_3_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[129]; }
    { const long long ij = ij_3_3, kl = kl_4_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[130]; }
    { const long long ij = ij_3_3, kl = kl_5_0;
      if ((!dab || 3 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[131]; }
    { const long long ij = ij_3_4, kl = kl_0_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[132]; }
    { const long long ij = ij_3_4, kl = kl_1_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[133]; }
    { const long long ij = ij_3_4, kl = kl_2_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[134]; }
    { const long long ij = ij_3_4, kl = kl_3_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[135]; }
    { const long long ij = ij_3_4, kl = kl_4_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[136]; }
    { const long long ij = ij_3_4, kl = kl_5_0;
      if ((!dab || 3 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[137]; }
    { const long long ij = ij_3_5, kl = kl_0_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[138]; }
    { const long long ij = ij_3_5, kl = kl_1_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[139]; }
    { const long long ij = ij_3_5, kl = kl_2_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[140]; }
    { const long long ij = ij_3_5, kl = kl_3_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[141]; }
    { const long long ij = ij_3_5, kl = kl_4_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[142]; }
    { const long long ij = ij_3_5, kl = kl_5_0;
      if ((!dab || 3 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[143]; }
    { const long long ij = ij_4_0, kl = kl_0_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[144]; }
    { const long long ij = ij_4_0, kl = kl_1_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[145]; }
    { const long long ij = ij_4_0, kl = kl_2_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[146]; }
    { const long long ij = ij_4_0, kl = kl_3_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[147]; }
    { const long long ij = ij_4_0, kl = kl_4_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[148]; }
    { const long long ij = ij_4_0, kl = kl_5_0;
      if ((!dab || 4 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[149]; }
    { const long long ij = ij_4_1, kl = kl_0_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[150]; }
    { const long long ij = ij_4_1, kl = kl_1_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[151]; }
    { const long long ij = ij_4_1, kl = kl_2_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[152]; }
    { const long long ij = ij_4_1, kl = kl_3_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[153]; }
    { const long long ij = ij_4_1, kl = kl_4_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[154]; }
    { const long long ij = ij_4_1, kl = kl_5_0;
      if ((!dab || 4 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[155]; }
    { const long long ij = ij_4_2, kl = kl_0_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[156]; }
    { const long long ij = ij_4_2, kl = kl_1_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[157]; }
    { const long long ij = ij_4_2, kl = kl_2_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[158]; }
    { const long long ij = ij_4_2, kl = kl_3_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[159]; }
    { const long long ij = ij_4_2, kl = kl_4_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[160]; }
    { const long long ij = ij_4_2, kl = kl_5_0;
      if ((!dab || 4 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[161]; }
    { const long long ij = ij_4_3, kl = kl_0_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[162]; }
    { const long long ij = ij_4_3, kl = kl_1_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[163]; }
    { const long long ij = ij_4_3, kl = kl_2_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[164]; }
    { const long long ij = ij_4_3, kl = kl_3_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[165]; }
    { const long long ij = ij_4_3, kl = kl_4_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[166]; }
    { const long long ij = ij_4_3, kl = kl_5_0;
      if ((!dab || 4 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[167]; }
    { const long long ij = ij_4_4, kl = kl_0_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[168]; }
    { const long long ij = ij_4_4, kl = kl_1_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[169]; }
    { const long long ij = ij_4_4, kl = kl_2_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[170]; }
    { const long long ij = ij_4_4, kl = kl_3_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[171]; }
    { const long long ij = ij_4_4, kl = kl_4_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[172]; }
    { const long long ij = ij_4_4, kl = kl_5_0;
      if ((!dab || 4 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[173]; }
    { const long long ij = ij_4_5, kl = kl_0_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[174]; }
    { const long long ij = ij_4_5, kl = kl_1_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[175]; }
    { const long long ij = ij_4_5, kl = kl_2_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[176]; }
    { const long long ij = ij_4_5, kl = kl_3_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[177]; }
    { const long long ij = ij_4_5, kl = kl_4_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[178]; }
    { const long long ij = ij_4_5, kl = kl_5_0;
      if ((!dab || 4 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[179]; }
    { const long long ij = ij_5_0, kl = kl_0_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[180]; }
    { const long long ij = ij_5_0, kl = kl_1_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[181]; }
    { const long long ij = ij_5_0, kl = kl_2_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[182]; }
    { const long long ij = ij_5_0, kl = kl_3_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[183]; }
    { const long long ij = ij_5_0, kl = kl_4_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[184]; }
    { const long long ij = ij_5_0, kl = kl_5_0;
      if ((!dab || 5 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[185]; }
    { const long long ij = ij_5_1, kl = kl_0_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[186]; }
    { const long long ij = ij_5_1, kl = kl_1_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[187]; }
    { const long long ij = ij_5_1, kl = kl_2_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[188]; }
    { const long long ij = ij_5_1, kl = kl_3_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[189]; }
    { const long long ij = ij_5_1, kl = kl_4_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[190]; }
    { const long long ij = ij_5_1, kl = kl_5_0;
      if ((!dab || 5 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[191]; }
    { const long long ij = ij_5_2, kl = kl_0_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[192]; }
    { const long long ij = ij_5_2, kl = kl_1_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[193]; }
    { const long long ij = ij_5_2, kl = kl_2_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[194]; }
    { const long long ij = ij_5_2, kl = kl_3_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[195]; }
    { const long long ij = ij_5_2, kl = kl_4_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[196]; }
    { const long long ij = ij_5_2, kl = kl_5_0;
      if ((!dab || 5 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[197]; }
    { const long long ij = ij_5_3, kl = kl_0_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[198]; }
    { const long long ij = ij_5_3, kl = kl_1_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[199]; }
    { const long long ij = ij_5_3, kl = kl_2_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[200]; }
    { const long long ij = ij_5_3, kl = kl_3_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[201]; }
    { const long long ij = ij_5_3, kl = kl_4_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[202]; }
    { const long long ij = ij_5_3, kl = kl_5_0;
      if ((!dab || 5 >= 3) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[203]; }
    { const long long ij = ij_5_4, kl = kl_0_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[204]; }
    { const long long ij = ij_5_4, kl = kl_1_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[205]; }
    { const long long ij = ij_5_4, kl = kl_2_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[206]; }
    { const long long ij = ij_5_4, kl = kl_3_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[207]; }
    { const long long ij = ij_5_4, kl = kl_4_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[208]; }
    { const long long ij = ij_5_4, kl = kl_5_0;
      if ((!dab || 5 >= 4) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[209]; }
    { const long long ij = ij_5_5, kl = kl_0_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[210]; }
    { const long long ij = ij_5_5, kl = kl_1_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[211]; }
    { const long long ij = ij_5_5, kl = kl_2_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[212]; }
    { const long long ij = ij_5_5, kl = kl_3_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[213]; }
    { const long long ij = ij_5_5, kl = kl_4_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[214]; }
    { const long long ij = ij_5_5, kl = kl_5_0;
      if ((!dab || 5 >= 5) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[215]; }
}

// The quartet's share of J and K (molints_plan_jk, eri_common.cuh): every integral of the block,
// times f, into one orientation of each target; J_ab stays in the lane (one bra pair per chunk).
__device__ __forceinline__ void jk_ddds(const JKOut &jk, const int4 ib_, const int4 ik_, double f,
                                         const double *__restrict__ res, double *__restrict__ jab) {
    const long long n = jk.n;
    const double *__restrict__ D = jk.D;
    const double *__restrict__ Db = D + ib_.w * n, *__restrict__ Dc = D + ik_.z * n;
    double dcd[6], dbc[36], dbd[6], jcd[6], kbc[36], kbd[6];
#pragma unroll
    for (int k = 0; k < 6; ++k)
#pragma unroll
        for (int l = 0; l < 1; ++l) {
            dcd[k * 1 + l] = __ldg(&Dc[k * n + ik_.w + l]);
            jcd[k * 1 + l] = 0.0;
        }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            dbc[j * 6 + k] = __ldg(&Db[j * n + ik_.z + k]);
            kbc[j * 6 + k] = 0.0;
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
        double dab[6], dac[6], dad[1], kac[6], kad[1];
#pragma unroll
        for (int j = 0; j < 6; ++j) dab[j] = __ldg(&Da[ib_.w + j]);
#pragma unroll
        for (int k = 0; k < 6; ++k) { dac[k] = __ldg(&Da[ik_.z + k]); kac[k] = 0.0; }
#pragma unroll
        for (int l = 0; l < 1; ++l) { dad[l] = __ldg(&Da[ik_.w + l]); kad[l] = 0.0; }
        { const double v = f * res[(i * 6 + 0) * 6 + 0];
          jab[i * 6 + 0] = fma(dcd[0], v, jab[i * 6 + 0]);
          jcd[0] = fma(dab[0], v, jcd[0]);
          kac[0] = fma(dbd[0], v, kac[0]);
          kad[0] = fma(dbc[0], v, kad[0]);
          kbc[0] = fma(dad[0], v, kbc[0]);
          kbd[0] = fma(dac[0], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 6 + 1];
          jab[i * 6 + 0] = fma(dcd[1], v, jab[i * 6 + 0]);
          jcd[1] = fma(dab[0], v, jcd[1]);
          kac[1] = fma(dbd[0], v, kac[1]);
          kad[0] = fma(dbc[1], v, kad[0]);
          kbc[1] = fma(dad[0], v, kbc[1]);
          kbd[0] = fma(dac[1], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 6 + 2];
          jab[i * 6 + 0] = fma(dcd[2], v, jab[i * 6 + 0]);
          jcd[2] = fma(dab[0], v, jcd[2]);
          kac[2] = fma(dbd[0], v, kac[2]);
          kad[0] = fma(dbc[2], v, kad[0]);
          kbc[2] = fma(dad[0], v, kbc[2]);
          kbd[0] = fma(dac[2], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 6 + 3];
          jab[i * 6 + 0] = fma(dcd[3], v, jab[i * 6 + 0]);
          jcd[3] = fma(dab[0], v, jcd[3]);
          kac[3] = fma(dbd[0], v, kac[3]);
          kad[0] = fma(dbc[3], v, kad[0]);
          kbc[3] = fma(dad[0], v, kbc[3]);
          kbd[0] = fma(dac[3], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 6 + 4];
          jab[i * 6 + 0] = fma(dcd[4], v, jab[i * 6 + 0]);
          jcd[4] = fma(dab[0], v, jcd[4]);
          kac[4] = fma(dbd[0], v, kac[4]);
          kad[0] = fma(dbc[4], v, kad[0]);
          kbc[4] = fma(dad[0], v, kbc[4]);
          kbd[0] = fma(dac[4], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 0) * 6 + 5];
          jab[i * 6 + 0] = fma(dcd[5], v, jab[i * 6 + 0]);
          jcd[5] = fma(dab[0], v, jcd[5]);
          kac[5] = fma(dbd[0], v, kac[5]);
          kad[0] = fma(dbc[5], v, kad[0]);
          kbc[5] = fma(dad[0], v, kbc[5]);
          kbd[0] = fma(dac[5], v, kbd[0]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 0];
          jab[i * 6 + 1] = fma(dcd[0], v, jab[i * 6 + 1]);
          jcd[0] = fma(dab[1], v, jcd[0]);
          kac[0] = fma(dbd[1], v, kac[0]);
          kad[0] = fma(dbc[6], v, kad[0]);
          kbc[6] = fma(dad[0], v, kbc[6]);
          kbd[1] = fma(dac[0], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 1];
          jab[i * 6 + 1] = fma(dcd[1], v, jab[i * 6 + 1]);
          jcd[1] = fma(dab[1], v, jcd[1]);
          kac[1] = fma(dbd[1], v, kac[1]);
          kad[0] = fma(dbc[7], v, kad[0]);
          kbc[7] = fma(dad[0], v, kbc[7]);
          kbd[1] = fma(dac[1], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 2];
          jab[i * 6 + 1] = fma(dcd[2], v, jab[i * 6 + 1]);
          jcd[2] = fma(dab[1], v, jcd[2]);
          kac[2] = fma(dbd[1], v, kac[2]);
          kad[0] = fma(dbc[8], v, kad[0]);
          kbc[8] = fma(dad[0], v, kbc[8]);
          kbd[1] = fma(dac[2], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 3];
          jab[i * 6 + 1] = fma(dcd[3], v, jab[i * 6 + 1]);
          jcd[3] = fma(dab[1], v, jcd[3]);
          kac[3] = fma(dbd[1], v, kac[3]);
          kad[0] = fma(dbc[9], v, kad[0]);
          kbc[9] = fma(dad[0], v, kbc[9]);
          kbd[1] = fma(dac[3], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 4];
          jab[i * 6 + 1] = fma(dcd[4], v, jab[i * 6 + 1]);
          jcd[4] = fma(dab[1], v, jcd[4]);
          kac[4] = fma(dbd[1], v, kac[4]);
          kad[0] = fma(dbc[10], v, kad[0]);
          kbc[10] = fma(dad[0], v, kbc[10]);
          kbd[1] = fma(dac[4], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 1) * 6 + 5];
          jab[i * 6 + 1] = fma(dcd[5], v, jab[i * 6 + 1]);
          jcd[5] = fma(dab[1], v, jcd[5]);
          kac[5] = fma(dbd[1], v, kac[5]);
          kad[0] = fma(dbc[11], v, kad[0]);
          kbc[11] = fma(dad[0], v, kbc[11]);
          kbd[1] = fma(dac[5], v, kbd[1]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 0];
          jab[i * 6 + 2] = fma(dcd[0], v, jab[i * 6 + 2]);
          jcd[0] = fma(dab[2], v, jcd[0]);
          kac[0] = fma(dbd[2], v, kac[0]);
          kad[0] = fma(dbc[12], v, kad[0]);
          kbc[12] = fma(dad[0], v, kbc[12]);
          kbd[2] = fma(dac[0], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 1];
          jab[i * 6 + 2] = fma(dcd[1], v, jab[i * 6 + 2]);
          jcd[1] = fma(dab[2], v, jcd[1]);
          kac[1] = fma(dbd[2], v, kac[1]);
          kad[0] = fma(dbc[13], v, kad[0]);
          kbc[13] = fma(dad[0], v, kbc[13]);
          kbd[2] = fma(dac[1], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 2];
          jab[i * 6 + 2] = fma(dcd[2], v, jab[i * 6 + 2]);
          jcd[2] = fma(dab[2], v, jcd[2]);
          kac[2] = fma(dbd[2], v, kac[2]);
          kad[0] = fma(dbc[14], v, kad[0]);
          kbc[14] = fma(dad[0], v, kbc[14]);
          kbd[2] = fma(dac[2], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 3];
          jab[i * 6 + 2] = fma(dcd[3], v, jab[i * 6 + 2]);
          jcd[3] = fma(dab[2], v, jcd[3]);
          kac[3] = fma(dbd[2], v, kac[3]);
          kad[0] = fma(dbc[15], v, kad[0]);
          kbc[15] = fma(dad[0], v, kbc[15]);
          kbd[2] = fma(dac[3], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 4];
          jab[i * 6 + 2] = fma(dcd[4], v, jab[i * 6 + 2]);
          jcd[4] = fma(dab[2], v, jcd[4]);
          kac[4] = fma(dbd[2], v, kac[4]);
          kad[0] = fma(dbc[16], v, kad[0]);
          kbc[16] = fma(dad[0], v, kbc[16]);
          kbd[2] = fma(dac[4], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 2) * 6 + 5];
          jab[i * 6 + 2] = fma(dcd[5], v, jab[i * 6 + 2]);
          jcd[5] = fma(dab[2], v, jcd[5]);
          kac[5] = fma(dbd[2], v, kac[5]);
          kad[0] = fma(dbc[17], v, kad[0]);
          kbc[17] = fma(dad[0], v, kbc[17]);
          kbd[2] = fma(dac[5], v, kbd[2]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 0];
          jab[i * 6 + 3] = fma(dcd[0], v, jab[i * 6 + 3]);
          jcd[0] = fma(dab[3], v, jcd[0]);
          kac[0] = fma(dbd[3], v, kac[0]);
          kad[0] = fma(dbc[18], v, kad[0]);
          kbc[18] = fma(dad[0], v, kbc[18]);
          kbd[3] = fma(dac[0], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 1];
          jab[i * 6 + 3] = fma(dcd[1], v, jab[i * 6 + 3]);
          jcd[1] = fma(dab[3], v, jcd[1]);
          kac[1] = fma(dbd[3], v, kac[1]);
          kad[0] = fma(dbc[19], v, kad[0]);
          kbc[19] = fma(dad[0], v, kbc[19]);
          kbd[3] = fma(dac[1], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 2];
          jab[i * 6 + 3] = fma(dcd[2], v, jab[i * 6 + 3]);
          jcd[2] = fma(dab[3], v, jcd[2]);
          kac[2] = fma(dbd[3], v, kac[2]);
          kad[0] = fma(dbc[20], v, kad[0]);
          kbc[20] = fma(dad[0], v, kbc[20]);
          kbd[3] = fma(dac[2], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 3];
          jab[i * 6 + 3] = fma(dcd[3], v, jab[i * 6 + 3]);
          jcd[3] = fma(dab[3], v, jcd[3]);
          kac[3] = fma(dbd[3], v, kac[3]);
          kad[0] = fma(dbc[21], v, kad[0]);
          kbc[21] = fma(dad[0], v, kbc[21]);
          kbd[3] = fma(dac[3], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 4];
          jab[i * 6 + 3] = fma(dcd[4], v, jab[i * 6 + 3]);
          jcd[4] = fma(dab[3], v, jcd[4]);
          kac[4] = fma(dbd[3], v, kac[4]);
          kad[0] = fma(dbc[22], v, kad[0]);
          kbc[22] = fma(dad[0], v, kbc[22]);
          kbd[3] = fma(dac[4], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 3) * 6 + 5];
          jab[i * 6 + 3] = fma(dcd[5], v, jab[i * 6 + 3]);
          jcd[5] = fma(dab[3], v, jcd[5]);
          kac[5] = fma(dbd[3], v, kac[5]);
          kad[0] = fma(dbc[23], v, kad[0]);
          kbc[23] = fma(dad[0], v, kbc[23]);
          kbd[3] = fma(dac[5], v, kbd[3]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 0];
          jab[i * 6 + 4] = fma(dcd[0], v, jab[i * 6 + 4]);
          jcd[0] = fma(dab[4], v, jcd[0]);
          kac[0] = fma(dbd[4], v, kac[0]);
          kad[0] = fma(dbc[24], v, kad[0]);
          kbc[24] = fma(dad[0], v, kbc[24]);
          kbd[4] = fma(dac[0], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 1];
          jab[i * 6 + 4] = fma(dcd[1], v, jab[i * 6 + 4]);
          jcd[1] = fma(dab[4], v, jcd[1]);
          kac[1] = fma(dbd[4], v, kac[1]);
          kad[0] = fma(dbc[25], v, kad[0]);
          kbc[25] = fma(dad[0], v, kbc[25]);
          kbd[4] = fma(dac[1], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 2];
          jab[i * 6 + 4] = fma(dcd[2], v, jab[i * 6 + 4]);
          jcd[2] = fma(dab[4], v, jcd[2]);
          kac[2] = fma(dbd[4], v, kac[2]);
          kad[0] = fma(dbc[26], v, kad[0]);
          kbc[26] = fma(dad[0], v, kbc[26]);
          kbd[4] = fma(dac[2], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 3];
          jab[i * 6 + 4] = fma(dcd[3], v, jab[i * 6 + 4]);
          jcd[3] = fma(dab[4], v, jcd[3]);
          kac[3] = fma(dbd[4], v, kac[3]);
          kad[0] = fma(dbc[27], v, kad[0]);
          kbc[27] = fma(dad[0], v, kbc[27]);
          kbd[4] = fma(dac[3], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 4];
          jab[i * 6 + 4] = fma(dcd[4], v, jab[i * 6 + 4]);
          jcd[4] = fma(dab[4], v, jcd[4]);
          kac[4] = fma(dbd[4], v, kac[4]);
          kad[0] = fma(dbc[28], v, kad[0]);
          kbc[28] = fma(dad[0], v, kbc[28]);
          kbd[4] = fma(dac[4], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 4) * 6 + 5];
          jab[i * 6 + 4] = fma(dcd[5], v, jab[i * 6 + 4]);
          jcd[5] = fma(dab[4], v, jcd[5]);
          kac[5] = fma(dbd[4], v, kac[5]);
          kad[0] = fma(dbc[29], v, kad[0]);
          kbc[29] = fma(dad[0], v, kbc[29]);
          kbd[4] = fma(dac[5], v, kbd[4]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 0];
          jab[i * 6 + 5] = fma(dcd[0], v, jab[i * 6 + 5]);
          jcd[0] = fma(dab[5], v, jcd[0]);
          kac[0] = fma(dbd[5], v, kac[0]);
          kad[0] = fma(dbc[30], v, kad[0]);
          kbc[30] = fma(dad[0], v, kbc[30]);
          kbd[5] = fma(dac[0], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 1];
          jab[i * 6 + 5] = fma(dcd[1], v, jab[i * 6 + 5]);
          jcd[1] = fma(dab[5], v, jcd[1]);
          kac[1] = fma(dbd[5], v, kac[1]);
          kad[0] = fma(dbc[31], v, kad[0]);
          kbc[31] = fma(dad[0], v, kbc[31]);
          kbd[5] = fma(dac[1], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 2];
          jab[i * 6 + 5] = fma(dcd[2], v, jab[i * 6 + 5]);
          jcd[2] = fma(dab[5], v, jcd[2]);
          kac[2] = fma(dbd[5], v, kac[2]);
          kad[0] = fma(dbc[32], v, kad[0]);
          kbc[32] = fma(dad[0], v, kbc[32]);
          kbd[5] = fma(dac[2], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 3];
          jab[i * 6 + 5] = fma(dcd[3], v, jab[i * 6 + 5]);
          jcd[3] = fma(dab[5], v, jcd[3]);
          kac[3] = fma(dbd[5], v, kac[3]);
          kad[0] = fma(dbc[33], v, kad[0]);
          kbc[33] = fma(dad[0], v, kbc[33]);
          kbd[5] = fma(dac[3], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 4];
          jab[i * 6 + 5] = fma(dcd[4], v, jab[i * 6 + 5]);
          jcd[4] = fma(dab[5], v, jcd[4]);
          kac[4] = fma(dbd[5], v, kac[4]);
          kad[0] = fma(dbc[34], v, kad[0]);
          kbc[34] = fma(dad[0], v, kbc[34]);
          kbd[5] = fma(dac[4], v, kbd[5]); }
        { const double v = f * res[(i * 6 + 5) * 6 + 5];
          jab[i * 6 + 5] = fma(dcd[5], v, jab[i * 6 + 5]);
          jcd[5] = fma(dab[5], v, jcd[5]);
          kac[5] = fma(dbd[5], v, kac[5]);
          kad[0] = fma(dbc[35], v, kad[0]);
          kbc[35] = fma(dad[0], v, kbc[35]);
          kbd[5] = fma(dac[5], v, kbd[5]); }
#pragma unroll
        for (int k = 0; k < 6; ++k) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.z + k], kac[k]);
#pragma unroll
        for (int l = 0; l < 1; ++l) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.w + l], kad[l]);
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) {
#pragma unroll
        for (int k = 0; k < 6; ++k) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.z + k], kbc[j * 6 + k]);
#pragma unroll
        for (int l = 0; l < 1; ++l) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.w + l], kbd[j * 1 + l]);
    }
#pragma unroll
    for (int k = 0; k < 6; ++k)
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
__global__ void __launch_bounds__(128) eri_queue_ddds(const EriQueue Q) {
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
        double acc[186];
        double2 bp = make_double2(0.0, 0.0), bq = bp;
        if (live) {
            bp = __ldg(&Q.pairs.bnd[p]);
            bq = __ldg(&Q.pairs.bnd[q]);
        }
        if (!live || bp.x * bq.x < Q.screen_cut) {
#pragma unroll
            for (int x = 0; x < 186; ++x) acc[x] = 0.0;
        } else {
            const int nb = __ldg(&Q.pairs.info[p]).y, nk = __ldg(&Q.pairs.info[q]).y;
            if (MIXED && bp.y * bq.y < Q.fp32_cut)
                vrr_ddds<float>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
            else vrr_ddds<double>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
        }
        if (lg) {
            for (int off = W; off < 32; off <<= 1) {
#pragma unroll
                for (int x = 0; x < 186; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
            }
        }
        const bool lead = live && s == 0;
        if (!JK && Q.scratch) {
            // two-phase: each leader stores its quartet's whole block at its slot
            if (lead) {
                double res[216];
                hrr_ddds(Q.pairs, p, q, acc, res);
                double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                    (__ldg(&Q.chunk_slot[c]) + base + kq) * (long long)216;
#pragma unroll
                for (int x = 0; x < 216; ++x) dst[x] = res[x];
            }
        } else if (lead) {
            double res[216];
            hrr_ddds(Q.pairs, p, q, acc, res);
            if constexpr (JK) {
                const int4 ib_ = __ldg(&Q.pairs.info[p]), ik_ = __ldg(&Q.pairs.info[q]);
                jk_ddds(Q.jk, ib_, ik_, jk_weight(ib_.z == ib_.w, ik_.z == ik_.w, p == q), res, jab);
            } else {
                store_ddds(Q.out + __ldg(&Q.mol_out[ch.w]), __ldg(&Q.pairs.info[p]), __ldg(&Q.pairs.info[q]),
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


void launch_eri_ddds(const EriQueue &Q, int mixed, int grid, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid <= 0) return;
    constexpr size_t smem = 0;
    const bool jk = Q.jk.J != nullptr;
    if (mixed) { if (jk) eri_queue_ddds<1, 1><<<grid, 128, 0, s>>>(Q); else eri_queue_ddds<1, 0><<<grid, 128, smem, s>>>(Q); }
    else if (jk) eri_queue_ddds<0, 1><<<grid, 128, 0, s>>>(Q);
    else eri_queue_ddds<0, 0><<<grid, 128, smem, s>>>(Q);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_eri_ddds(int mixed) {

    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_ddds<1, 0>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_ddds<0, 0>, 128, 0);
    return n;
}

}  // namespace molints
