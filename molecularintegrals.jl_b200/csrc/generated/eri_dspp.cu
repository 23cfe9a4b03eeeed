// Generated by gen_eri.py -- class (ds|pp).  Do not edit.
// VRR entries: 116, contracted block: 54, HRR lines: 54, outputs: 54.
#include "../eri_common.cuh"

namespace molints {

// The contracted [e0|f0] block of bra pair p and ket pair q into acc[54], summed over
// the bra primitive pairs i0, i0 + istep, ... < i1 and the ket primitive pairs j0, j0 + jstep,
// ... < j1 of the two shell pairs.  VT is the VRR arithmetic type (double, or float for MIXED).
// The ket loop is outside: a warp shares its bra pair, so the inner bra loads are broadcasts
// and each lane's ket record is loaded once.  Steps above 1 split one quartet's primitive
// quartets over the lanes of a split group (their blocks are summed before the HRR).
template <typename VT>
__device__ __forceinline__ void vrr_dspp(const PairTab &P, const BoysTab &B, int p, int q,
                                          int i0, int i1, int istep, int j0, int j1, int jstep,
                                          double *__restrict__ acc) {
    const int4 ib_ = __ldg(&P.info[p]);
    const int4 ik_ = __ldg(&P.info[q]);
#pragma unroll
    for (int x = 0; x < 54; ++x) acc[x] = 0.0;
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
            double F[5];
            boys_scaled<4>(far, ze * r2, B, F);
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
            const VT v1_0_0 = PAx * v0_0_0 + WPx * v0_0_1;
            const VT v1_0_1 = PAx * v0_0_1 + WPx * v0_0_2;
            const VT v1_0_2 = PAx * v0_0_2 + WPx * v0_0_3;
            const VT v1_0_3 = PAx * v0_0_3 + WPx * v0_0_4;
            const VT v2_0_0 = PAy * v0_0_0 + WPy * v0_0_1;
            const VT v2_0_1 = PAy * v0_0_1 + WPy * v0_0_2;
            const VT v2_0_2 = PAy * v0_0_2 + WPy * v0_0_3;
            const VT v2_0_3 = PAy * v0_0_3 + WPy * v0_0_4;
            const VT v3_0_0 = PAz * v0_0_0 + WPz * v0_0_1;
            const VT v3_0_1 = PAz * v0_0_1 + WPz * v0_0_2;
            const VT v3_0_2 = PAz * v0_0_2 + WPz * v0_0_3;
            const VT v3_0_3 = PAz * v0_0_3 + WPz * v0_0_4;
            const VT v4_0_0 = PAx * v1_0_0 + WPx * v1_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v4_0_1 = PAx * v1_0_1 + WPx * v1_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v4_0_2 = PAx * v1_0_2 + WPx * v1_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v5_0_0 = PAx * v2_0_0 + WPx * v2_0_1;
            const VT v5_0_1 = PAx * v2_0_1 + WPx * v2_0_2;
            const VT v5_0_2 = PAx * v2_0_2 + WPx * v2_0_3;
            const VT v6_0_0 = PAx * v3_0_0 + WPx * v3_0_1;
            const VT v6_0_1 = PAx * v3_0_1 + WPx * v3_0_2;
            const VT v6_0_2 = PAx * v3_0_2 + WPx * v3_0_3;
            const VT v7_0_0 = PAy * v2_0_0 + WPy * v2_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v7_0_1 = PAy * v2_0_1 + WPy * v2_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v7_0_2 = PAy * v2_0_2 + WPy * v2_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
            const VT v8_0_0 = PAy * v3_0_0 + WPy * v3_0_1;
            const VT v8_0_1 = PAy * v3_0_1 + WPy * v3_0_2;
            const VT v8_0_2 = PAy * v3_0_2 + WPy * v3_0_3;
            const VT v9_0_0 = PAz * v3_0_0 + WPz * v3_0_1 + (VT)1.0 * oo2z * (v0_0_0 - rho_z * v0_0_1);
            const VT v9_0_1 = PAz * v3_0_1 + WPz * v3_0_2 + (VT)1.0 * oo2z * (v0_0_1 - rho_z * v0_0_2);
            const VT v9_0_2 = PAz * v3_0_2 + WPz * v3_0_3 + (VT)1.0 * oo2z * (v0_0_2 - rho_z * v0_0_3);
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
            if constexpr (sizeof(VT) == 8) {
                acc[0] += (double)v4_1_0;
                acc[1] += (double)v4_2_0;
                acc[2] += (double)v4_3_0;
                acc[3] = fma(QCx, v4_1_0, fma(WQx, v4_1_1, fma(2.0 * oo2ze, v1_1_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[3]))));
                acc[4] = fma(QCx, v4_2_0, fma(WQx, v4_2_1, fma(2.0 * oo2ze, v1_2_1, acc[4])));
                acc[5] = fma(QCx, v4_3_0, fma(WQx, v4_3_1, fma(2.0 * oo2ze, v1_3_1, acc[5])));
                acc[6] = fma(QCy, v4_2_0, fma(WQy, v4_2_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[6])));
                acc[7] = fma(QCy, v4_3_0, fma(WQy, v4_3_1, acc[7]));
                acc[8] = fma(QCz, v4_3_0, fma(WQz, v4_3_1, fma(1.0 * oo2e, (v4_0_0 - rho_e * v4_0_1), acc[8])));
                acc[9] += (double)v5_1_0;
                acc[10] += (double)v5_2_0;
                acc[11] += (double)v5_3_0;
                acc[12] = fma(QCx, v5_1_0, fma(WQx, v5_1_1, fma(1.0 * oo2ze, v2_1_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[12]))));
                acc[13] = fma(QCx, v5_2_0, fma(WQx, v5_2_1, fma(1.0 * oo2ze, v2_2_1, acc[13])));
                acc[14] = fma(QCx, v5_3_0, fma(WQx, v5_3_1, fma(1.0 * oo2ze, v2_3_1, acc[14])));
                acc[15] = fma(QCy, v5_2_0, fma(WQy, v5_2_1, fma(1.0 * oo2ze, v1_2_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[15]))));
                acc[16] = fma(QCy, v5_3_0, fma(WQy, v5_3_1, fma(1.0 * oo2ze, v1_3_1, acc[16])));
                acc[17] = fma(QCz, v5_3_0, fma(WQz, v5_3_1, fma(1.0 * oo2e, (v5_0_0 - rho_e * v5_0_1), acc[17])));
                acc[18] += (double)v6_1_0;
                acc[19] += (double)v6_2_0;
                acc[20] += (double)v6_3_0;
                acc[21] = fma(QCx, v6_1_0, fma(WQx, v6_1_1, fma(1.0 * oo2ze, v3_1_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[21]))));
                acc[22] = fma(QCx, v6_2_0, fma(WQx, v6_2_1, fma(1.0 * oo2ze, v3_2_1, acc[22])));
                acc[23] = fma(QCx, v6_3_0, fma(WQx, v6_3_1, fma(1.0 * oo2ze, v3_3_1, acc[23])));
                acc[24] = fma(QCy, v6_2_0, fma(WQy, v6_2_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[24])));
                acc[25] = fma(QCy, v6_3_0, fma(WQy, v6_3_1, acc[25]));
                acc[26] = fma(QCz, v6_3_0, fma(WQz, v6_3_1, fma(1.0 * oo2ze, v1_3_1, fma(1.0 * oo2e, (v6_0_0 - rho_e * v6_0_1), acc[26]))));
                acc[27] += (double)v7_1_0;
                acc[28] += (double)v7_2_0;
                acc[29] += (double)v7_3_0;
                acc[30] = fma(QCx, v7_1_0, fma(WQx, v7_1_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[30])));
                acc[31] = fma(QCx, v7_2_0, fma(WQx, v7_2_1, acc[31]));
                acc[32] = fma(QCx, v7_3_0, fma(WQx, v7_3_1, acc[32]));
                acc[33] = fma(QCy, v7_2_0, fma(WQy, v7_2_1, fma(2.0 * oo2ze, v2_2_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[33]))));
                acc[34] = fma(QCy, v7_3_0, fma(WQy, v7_3_1, fma(2.0 * oo2ze, v2_3_1, acc[34])));
                acc[35] = fma(QCz, v7_3_0, fma(WQz, v7_3_1, fma(1.0 * oo2e, (v7_0_0 - rho_e * v7_0_1), acc[35])));
                acc[36] += (double)v8_1_0;
                acc[37] += (double)v8_2_0;
                acc[38] += (double)v8_3_0;
                acc[39] = fma(QCx, v8_1_0, fma(WQx, v8_1_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[39])));
                acc[40] = fma(QCx, v8_2_0, fma(WQx, v8_2_1, acc[40]));
                acc[41] = fma(QCx, v8_3_0, fma(WQx, v8_3_1, acc[41]));
                acc[42] = fma(QCy, v8_2_0, fma(WQy, v8_2_1, fma(1.0 * oo2ze, v3_2_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[42]))));
                acc[43] = fma(QCy, v8_3_0, fma(WQy, v8_3_1, fma(1.0 * oo2ze, v3_3_1, acc[43])));
                acc[44] = fma(QCz, v8_3_0, fma(WQz, v8_3_1, fma(1.0 * oo2ze, v2_3_1, fma(1.0 * oo2e, (v8_0_0 - rho_e * v8_0_1), acc[44]))));
                acc[45] += (double)v9_1_0;
                acc[46] += (double)v9_2_0;
                acc[47] += (double)v9_3_0;
                acc[48] = fma(QCx, v9_1_0, fma(WQx, v9_1_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[48])));
                acc[49] = fma(QCx, v9_2_0, fma(WQx, v9_2_1, acc[49]));
                acc[50] = fma(QCx, v9_3_0, fma(WQx, v9_3_1, acc[50]));
                acc[51] = fma(QCy, v9_2_0, fma(WQy, v9_2_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[51])));
                acc[52] = fma(QCy, v9_3_0, fma(WQy, v9_3_1, acc[52]));
                acc[53] = fma(QCz, v9_3_0, fma(WQz, v9_3_1, fma(2.0 * oo2ze, v3_3_1, fma(1.0 * oo2e, (v9_0_0 - rho_e * v9_0_1), acc[53]))));
            } else {
                acc[0] += (double)v4_1_0;
                acc[1] += (double)v4_2_0;
                acc[2] += (double)v4_3_0;
                const VT v4_4_0 = QCx * v4_1_0 + WQx * v4_1_1 + (VT)2.0 * oo2ze * v1_1_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[3] += (double)v4_4_0;
                const VT v4_5_0 = QCx * v4_2_0 + WQx * v4_2_1 + (VT)2.0 * oo2ze * v1_2_1;
                acc[4] += (double)v4_5_0;
                const VT v4_6_0 = QCx * v4_3_0 + WQx * v4_3_1 + (VT)2.0 * oo2ze * v1_3_1;
                acc[5] += (double)v4_6_0;
                const VT v4_7_0 = QCy * v4_2_0 + WQy * v4_2_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[6] += (double)v4_7_0;
                const VT v4_8_0 = QCy * v4_3_0 + WQy * v4_3_1;
                acc[7] += (double)v4_8_0;
                const VT v4_9_0 = QCz * v4_3_0 + WQz * v4_3_1 + (VT)1.0 * oo2e * (v4_0_0 - rho_e * v4_0_1);
                acc[8] += (double)v4_9_0;
                acc[9] += (double)v5_1_0;
                acc[10] += (double)v5_2_0;
                acc[11] += (double)v5_3_0;
                const VT v5_4_0 = QCx * v5_1_0 + WQx * v5_1_1 + (VT)1.0 * oo2ze * v2_1_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[12] += (double)v5_4_0;
                const VT v5_5_0 = QCx * v5_2_0 + WQx * v5_2_1 + (VT)1.0 * oo2ze * v2_2_1;
                acc[13] += (double)v5_5_0;
                const VT v5_6_0 = QCx * v5_3_0 + WQx * v5_3_1 + (VT)1.0 * oo2ze * v2_3_1;
                acc[14] += (double)v5_6_0;
                const VT v5_7_0 = QCy * v5_2_0 + WQy * v5_2_1 + (VT)1.0 * oo2ze * v1_2_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[15] += (double)v5_7_0;
                const VT v5_8_0 = QCy * v5_3_0 + WQy * v5_3_1 + (VT)1.0 * oo2ze * v1_3_1;
                acc[16] += (double)v5_8_0;
                const VT v5_9_0 = QCz * v5_3_0 + WQz * v5_3_1 + (VT)1.0 * oo2e * (v5_0_0 - rho_e * v5_0_1);
                acc[17] += (double)v5_9_0;
                acc[18] += (double)v6_1_0;
                acc[19] += (double)v6_2_0;
                acc[20] += (double)v6_3_0;
                const VT v6_4_0 = QCx * v6_1_0 + WQx * v6_1_1 + (VT)1.0 * oo2ze * v3_1_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[21] += (double)v6_4_0;
                const VT v6_5_0 = QCx * v6_2_0 + WQx * v6_2_1 + (VT)1.0 * oo2ze * v3_2_1;
                acc[22] += (double)v6_5_0;
                const VT v6_6_0 = QCx * v6_3_0 + WQx * v6_3_1 + (VT)1.0 * oo2ze * v3_3_1;
                acc[23] += (double)v6_6_0;
                const VT v6_7_0 = QCy * v6_2_0 + WQy * v6_2_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[24] += (double)v6_7_0;
                const VT v6_8_0 = QCy * v6_3_0 + WQy * v6_3_1;
                acc[25] += (double)v6_8_0;
                const VT v6_9_0 = QCz * v6_3_0 + WQz * v6_3_1 + (VT)1.0 * oo2ze * v1_3_1 + (VT)1.0 * oo2e * (v6_0_0 - rho_e * v6_0_1);
                acc[26] += (double)v6_9_0;
                acc[27] += (double)v7_1_0;
                acc[28] += (double)v7_2_0;
                acc[29] += (double)v7_3_0;
                const VT v7_4_0 = QCx * v7_1_0 + WQx * v7_1_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[30] += (double)v7_4_0;
                const VT v7_5_0 = QCx * v7_2_0 + WQx * v7_2_1;
                acc[31] += (double)v7_5_0;
                const VT v7_6_0 = QCx * v7_3_0 + WQx * v7_3_1;
                acc[32] += (double)v7_6_0;
                const VT v7_7_0 = QCy * v7_2_0 + WQy * v7_2_1 + (VT)2.0 * oo2ze * v2_2_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[33] += (double)v7_7_0;
                const VT v7_8_0 = QCy * v7_3_0 + WQy * v7_3_1 + (VT)2.0 * oo2ze * v2_3_1;
                acc[34] += (double)v7_8_0;
                const VT v7_9_0 = QCz * v7_3_0 + WQz * v7_3_1 + (VT)1.0 * oo2e * (v7_0_0 - rho_e * v7_0_1);
                acc[35] += (double)v7_9_0;
                acc[36] += (double)v8_1_0;
                acc[37] += (double)v8_2_0;
                acc[38] += (double)v8_3_0;
                const VT v8_4_0 = QCx * v8_1_0 + WQx * v8_1_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[39] += (double)v8_4_0;
                const VT v8_5_0 = QCx * v8_2_0 + WQx * v8_2_1;
                acc[40] += (double)v8_5_0;
                const VT v8_6_0 = QCx * v8_3_0 + WQx * v8_3_1;
                acc[41] += (double)v8_6_0;
                const VT v8_7_0 = QCy * v8_2_0 + WQy * v8_2_1 + (VT)1.0 * oo2ze * v3_2_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[42] += (double)v8_7_0;
                const VT v8_8_0 = QCy * v8_3_0 + WQy * v8_3_1 + (VT)1.0 * oo2ze * v3_3_1;
                acc[43] += (double)v8_8_0;
                const VT v8_9_0 = QCz * v8_3_0 + WQz * v8_3_1 + (VT)1.0 * oo2ze * v2_3_1 + (VT)1.0 * oo2e * (v8_0_0 - rho_e * v8_0_1);
                acc[44] += (double)v8_9_0;
                acc[45] += (double)v9_1_0;
                acc[46] += (double)v9_2_0;
                acc[47] += (double)v9_3_0;
                const VT v9_4_0 = QCx * v9_1_0 + WQx * v9_1_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[48] += (double)v9_4_0;
                const VT v9_5_0 = QCx * v9_2_0 + WQx * v9_2_1;
                acc[49] += (double)v9_5_0;
                const VT v9_6_0 = QCx * v9_3_0 + WQx * v9_3_1;
                acc[50] += (double)v9_6_0;
                const VT v9_7_0 = QCy * v9_2_0 + WQy * v9_2_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[51] += (double)v9_7_0;
                const VT v9_8_0 = QCy * v9_3_0 + WQy * v9_3_1;
                acc[52] += (double)v9_8_0;
                const VT v9_9_0 = QCz * v9_3_0 + WQz * v9_3_1 + (VT)2.0 * oo2ze * v3_3_1 + (VT)1.0 * oo2e * (v9_0_0 - rho_e * v9_0_1);
                acc[53] += (double)v9_9_0;
            }
        }
    }
}

// Bra and ket HRR of the contracted block (src/HGP.jl:92-114), then the component norms:
// the normalised (ab|cd) of bra pair p and ket pair q into res[54] (ma, mb, mc, md
// row-major).
__device__ __forceinline__ void hrr_dspp(const PairTab &P, int p, int q, const double *__restrict__ acc,
                                          double *__restrict__ res) {
    const double4 gb = ldg4(&P.geo[p]);
    const double4 gk = ldg4(&P.geo[q]);
    const double ABx = gb.x, ABy = gb.y, ABz = gb.z;
    const double CDx = gk.x, CDy = gk.y, CDz = gk.z;
    (void)ABx; (void)ABy; (void)ABz; (void)CDx; (void)CDy; (void)CDz;
    const double k4_0_1_1 = acc[3] + CDx * acc[0];
    const double k4_0_1_2 = acc[4] + CDy * acc[0];
    const double k4_0_1_3 = acc[5] + CDz * acc[0];
    const double k4_0_2_1 = acc[4] + CDx * acc[1];
    const double k4_0_2_2 = acc[6] + CDy * acc[1];
    const double k4_0_2_3 = acc[7] + CDz * acc[1];
    const double k4_0_3_1 = acc[5] + CDx * acc[2];
    const double k4_0_3_2 = acc[7] + CDy * acc[2];
    const double k4_0_3_3 = acc[8] + CDz * acc[2];
    const double k5_0_1_1 = acc[12] + CDx * acc[9];
    const double k5_0_1_2 = acc[13] + CDy * acc[9];
    const double k5_0_1_3 = acc[14] + CDz * acc[9];
    const double k5_0_2_1 = acc[13] + CDx * acc[10];
    const double k5_0_2_2 = acc[15] + CDy * acc[10];
    const double k5_0_2_3 = acc[16] + CDz * acc[10];
    const double k5_0_3_1 = acc[14] + CDx * acc[11];
    const double k5_0_3_2 = acc[16] + CDy * acc[11];
    const double k5_0_3_3 = acc[17] + CDz * acc[11];
    const double k6_0_1_1 = acc[21] + CDx * acc[18];
    const double k6_0_1_2 = acc[22] + CDy * acc[18];
    const double k6_0_1_3 = acc[23] + CDz * acc[18];
    const double k6_0_2_1 = acc[22] + CDx * acc[19];
    const double k6_0_2_2 = acc[24] + CDy * acc[19];
    const double k6_0_2_3 = acc[25] + CDz * acc[19];
    const double k6_0_3_1 = acc[23] + CDx * acc[20];
    const double k6_0_3_2 = acc[25] + CDy * acc[20];
    const double k6_0_3_3 = acc[26] + CDz * acc[20];
    const double k7_0_1_1 = acc[30] + CDx * acc[27];
    const double k7_0_1_2 = acc[31] + CDy * acc[27];
    const double k7_0_1_3 = acc[32] + CDz * acc[27];
    const double k7_0_2_1 = acc[31] + CDx * acc[28];
    const double k7_0_2_2 = acc[33] + CDy * acc[28];
    const double k7_0_2_3 = acc[34] + CDz * acc[28];
    const double k7_0_3_1 = acc[32] + CDx * acc[29];
    const double k7_0_3_2 = acc[34] + CDy * acc[29];
    const double k7_0_3_3 = acc[35] + CDz * acc[29];
    const double k8_0_1_1 = acc[39] + CDx * acc[36];
    const double k8_0_1_2 = acc[40] + CDy * acc[36];
    const double k8_0_1_3 = acc[41] + CDz * acc[36];
    const double k8_0_2_1 = acc[40] + CDx * acc[37];
    const double k8_0_2_2 = acc[42] + CDy * acc[37];
    const double k8_0_2_3 = acc[43] + CDz * acc[37];
    const double k8_0_3_1 = acc[41] + CDx * acc[38];
    const double k8_0_3_2 = acc[43] + CDy * acc[38];
    const double k8_0_3_3 = acc[44] + CDz * acc[38];
    const double k9_0_1_1 = acc[48] + CDx * acc[45];
    const double k9_0_1_2 = acc[49] + CDy * acc[45];
    const double k9_0_1_3 = acc[50] + CDz * acc[45];
    const double k9_0_2_1 = acc[49] + CDx * acc[46];
    const double k9_0_2_2 = acc[51] + CDy * acc[46];
    const double k9_0_2_3 = acc[52] + CDz * acc[46];
    const double k9_0_3_1 = acc[50] + CDx * acc[47];
    const double k9_0_3_2 = acc[52] + CDy * acc[47];
    const double k9_0_3_3 = acc[53] + CDz * acc[47];
    res[0] = k4_0_1_1 * 0.5773502691896258;
    res[1] = k4_0_1_2 * 0.5773502691896258;
    res[2] = k4_0_1_3 * 0.5773502691896258;
    res[3] = k4_0_2_1 * 0.5773502691896258;
    res[4] = k4_0_2_2 * 0.5773502691896258;
    res[5] = k4_0_2_3 * 0.5773502691896258;
    res[6] = k4_0_3_1 * 0.5773502691896258;
    res[7] = k4_0_3_2 * 0.5773502691896258;
    res[8] = k4_0_3_3 * 0.5773502691896258;
    res[9] = k5_0_1_1;
    res[10] = k5_0_1_2;
    res[11] = k5_0_1_3;
    res[12] = k5_0_2_1;
    res[13] = k5_0_2_2;
    res[14] = k5_0_2_3;
    res[15] = k5_0_3_1;
    res[16] = k5_0_3_2;
    res[17] = k5_0_3_3;
    res[18] = k6_0_1_1;
    res[19] = k6_0_1_2;
    res[20] = k6_0_1_3;
    res[21] = k6_0_2_1;
    res[22] = k6_0_2_2;
    res[23] = k6_0_2_3;
    res[24] = k6_0_3_1;
    res[25] = k6_0_3_2;
    res[26] = k6_0_3_3;
    res[27] = k7_0_1_1 * 0.5773502691896258;
    res[28] = k7_0_1_2 * 0.5773502691896258;
    res[29] = k7_0_1_3 * 0.5773502691896258;
    res[30] = k7_0_2_1 * 0.5773502691896258;
    res[31] = k7_0_2_2 * 0.5773502691896258;
    res[32] = k7_0_2_3 * 0.5773502691896258;
    res[33] = k7_0_3_1 * 0.5773502691896258;
    res[34] = k7_0_3_2 * 0.5773502691896258;
    res[35] = k7_0_3_3 * 0.5773502691896258;
    res[36] = k8_0_1_1;
    res[37] = k8_0_1_2;
    res[38] = k8_0_1_3;
    res[39] = k8_0_2_1;
    res[40] = k8_0_2_2;
    res[41] = k8_0_2_3;
    res[42] = k8_0_3_1;
    res[43] = k8_0_3_2;
    res[44] = k8_0_3_3;
    res[45] = k9_0_1_1 * 0.5773502691896258;
    res[46] = k9_0_1_2 * 0.5773502691896258;
    res[47] = k9_0_1_3 * 0.5773502691896258;
    res[48] = k9_0_2_1 * 0.5773502691896258;
    res[49] = k9_0_2_2 * 0.5773502691896258;
    res[50] = k9_0_2_3 * 0.5773502691896258;
    res[51] = k9_0_3_1 * 0.5773502691896258;
    res[52] = k9_0_3_2 * 0.5773502691896258;
    res[53] = k9_0_3_3 * 0.5773502691896258;
}

// (ab|cd) over the bra primitive pairs [i0, i1) and ket primitive pairs [j0, j1) into
// res[54]; the contracted block also into acc_out when given (the bound kernels).
template <typename VT>
__device__ __forceinline__ void quartet_dspp(const PairTab &P, const BoysTab &B, int p, int q,
                                              int i0, int i1, int j0, int j1,
                                              double *__restrict__ res,
                                              double *__restrict__ acc_out = nullptr) {
    double acc[54];
    vrr_dspp<VT>(P, B, p, q, i0, i1, 1, j0, j1, 1, acc);
    if (acc_out) {
#pragma unroll
        for (int x = 0; x < 54; ++x) acc_out[x] = acc[x];
    }
    hrr_dspp(P, p, q, acc, res);
}

__device__ __forceinline__ void store_dspp(double *__restrict__ out, const int4 ib_, const int4 ik_,
                                            bool same, const double *__restrict__ res) {
    const bool dab = ib_.z == ib_.w, dcd = ik_.z == ik_.w;
    (void)dab; (void)dcd;
    const long long ij_0_0 = pair_index(ib_.z + 0, ib_.w + 0);
    const long long ij_1_0 = pair_index(ib_.z + 1, ib_.w + 0);
    const long long ij_2_0 = pair_index(ib_.z + 2, ib_.w + 0);
    const long long ij_3_0 = pair_index(ib_.z + 3, ib_.w + 0);
    const long long ij_4_0 = pair_index(ib_.z + 4, ib_.w + 0);
    const long long ij_5_0 = pair_index(ib_.z + 5, ib_.w + 0);
    const long long kl_0_0 = pair_index(ik_.z + 0, ik_.w + 0);
    const long long kl_0_1 = pair_index(ik_.z + 0, ik_.w + 1);
    const long long kl_0_2 = pair_index(ik_.z + 0, ik_.w + 2);
    const long long kl_1_0 = pair_index(ik_.z + 1, ik_.w + 0);
    const long long kl_1_1 = pair_index(ik_.z + 1, ik_.w + 1);
    const long long kl_1_2 = pair_index(ik_.z + 1, ik_.w + 2);
    const long long kl_2_0 = pair_index(ik_.z + 2, ik_.w + 0);
    const long long kl_2_1 = pair_index(ik_.z + 2, ik_.w + 1);
    const long long kl_2_2 = pair_index(ik_.z + 2, ik_.w + 2);
    { const long long ij = ij_0_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[0]; }
    { const long long ij = ij_0_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[1]; }
    { const long long ij = ij_0_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[2]; }
    { const long long ij = ij_0_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[3]; }
    { const long long ij = ij_0_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[4]; }
    { const long long ij = ij_0_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[5]; }
    { const long long ij = ij_0_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[6]; }
    { const long long ij = ij_0_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[7]; }
    { const long long ij = ij_0_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[8]; }
    { const long long ij = ij_1_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[9]; }
    { const long long ij = ij_1_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[10]; }
    { const long long ij = ij_1_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[11]; }
    { const long long ij = ij_1_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[12]; }
    { const long long ij = ij_1_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[13]; }
    { const long long ij = ij_1_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[14]; }
    { const long long ij = ij_1_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[15]; }
    { const long long ij = ij_1_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[16]; }
    { const long long ij = ij_1_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[17]; }
    { const long long ij = ij_2_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[18]; }
    { const long long ij = ij_2_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[19]; }
    { const long long ij = ij_2_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[20]; }
    { const long long ij = ij_2_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[21]; }
    { const long long ij = ij_2_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[22]; }
    { const long long ij = ij_2_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[23]; }
    { const long long ij = ij_2_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[24]; }
    { const long long ij = ij_2_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[25]; }
    { const long long ij = ij_2_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[26]; }
    { const long long ij = ij_3_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[27]; }
    { const long long ij = ij_3_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[28]; }
    { const long long ij = ij_3_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[29]; }
    { const long long ij = ij_3_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[30]; }
    { const long long ij = ij_3_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[31]; }
    { const long long ij = ij_3_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[32]; }
    { const long long ij = ij_3_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[33]; }
    { const long long ij = ij_3_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[34]; }
    { const long long ij = ij_3_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[35]; }
    { const long long ij = ij_4_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[36]; }
    { const long long ij = ij_4_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[37]; }
    { const long long ij = ij_4_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[38]; }
    { const long long ij = ij_4_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[39]; }
    { const long long ij = ij_4_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[40]; }
    { const long long ij = ij_4_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[41]; }
    { const long long ij = ij_4_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[42]; }
    { const long long ij = ij_4_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[43]; }
    { const long long ij = ij_4_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[44]; }
    { const long long ij = ij_5_0, kl = kl_0_0;
      if ((!dcd || 0 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[45]; }
    { const long long ij = ij_5_0, kl = kl_0_1;
      if ((!dcd || 0 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[46]; }
    { const long long ij = ij_5_0, kl = kl_0_2;
      if ((!dcd || 0 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[47]; }
    { const long long ij = ij_5_0, kl = kl_1_0;
      if ((!dcd || 1 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[48]; }
    { const long long ij = ij_5_0, kl = kl_1_1;
      if ((!dcd || 1 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[49]; }
    { const long long ij = ij_5_0, kl = kl_1_2;
      if ((!dcd || 1 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[50]; }
    { const long long ij = ij_5_0, kl = kl_2_0;
      if ((!dcd || 2 >= 0) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[51]; }
    { const long long ij = ij_5_0, kl = kl_2_1;
      if ((!dcd || 2 >= 1) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[52]; }
    { const long long ij = ij_5_0, kl = kl_2_2;
      if ((!dcd || 2 >= 2) && (!same || ij >= kl)) out[packed_index(ij, kl)] = res[53]; }
}

// The quartet's share of J and K (molints_plan_jk, eri_common.cuh): every integral of the block,
// times f, into one orientation of each target; J_ab stays in the lane (one bra pair per chunk).
__device__ __forceinline__ void jk_dspp(const JKOut &jk, const int4 ib_, const int4 ik_, double f,
                                         const double *__restrict__ res, double *__restrict__ jab) {
    const long long n = jk.n;
    const double *__restrict__ D = jk.D;
    const double *__restrict__ Db = D + ib_.w * n, *__restrict__ Dc = D + ik_.z * n;
    double dcd[9], dbc[3], dbd[3], jcd[9], kbc[3], kbd[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            dcd[k * 3 + l] = __ldg(&Dc[k * n + ik_.w + l]);
            jcd[k * 3 + l] = 0.0;
        }
#pragma unroll
    for (int j = 0; j < 1; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            dbc[j * 3 + k] = __ldg(&Db[j * n + ik_.z + k]);
            kbc[j * 3 + k] = 0.0;
        }
#pragma unroll
        for (int l = 0; l < 3; ++l) {
            dbd[j * 3 + l] = __ldg(&Db[j * n + ik_.w + l]);
            kbd[j * 3 + l] = 0.0;
        }
    }
#pragma unroll 1
    for (int i = 0; i < 6; ++i) {
        const double *__restrict__ Da = D + (ib_.z + i) * n;
        double dab[1], dac[3], dad[3], kac[3], kad[3];
#pragma unroll
        for (int j = 0; j < 1; ++j) dab[j] = __ldg(&Da[ib_.w + j]);
#pragma unroll
        for (int k = 0; k < 3; ++k) { dac[k] = __ldg(&Da[ik_.z + k]); kac[k] = 0.0; }
#pragma unroll
        for (int l = 0; l < 3; ++l) { dad[l] = __ldg(&Da[ik_.w + l]); kad[l] = 0.0; }
        { const double v = f * res[(i * 1 + 0) * 9 + 0];
          jab[i * 1 + 0] = fma(dcd[0], v, jab[i * 1 + 0]);
          jcd[0] = fma(dab[0], v, jcd[0]);
          kac[0] = fma(dbd[0], v, kac[0]);
          kad[0] = fma(dbc[0], v, kad[0]);
          kbc[0] = fma(dad[0], v, kbc[0]);
          kbd[0] = fma(dac[0], v, kbd[0]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 1];
          jab[i * 1 + 0] = fma(dcd[1], v, jab[i * 1 + 0]);
          jcd[1] = fma(dab[0], v, jcd[1]);
          kac[0] = fma(dbd[1], v, kac[0]);
          kad[1] = fma(dbc[0], v, kad[1]);
          kbc[0] = fma(dad[1], v, kbc[0]);
          kbd[1] = fma(dac[0], v, kbd[1]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 2];
          jab[i * 1 + 0] = fma(dcd[2], v, jab[i * 1 + 0]);
          jcd[2] = fma(dab[0], v, jcd[2]);
          kac[0] = fma(dbd[2], v, kac[0]);
          kad[2] = fma(dbc[0], v, kad[2]);
          kbc[0] = fma(dad[2], v, kbc[0]);
          kbd[2] = fma(dac[0], v, kbd[2]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 3];
          jab[i * 1 + 0] = fma(dcd[3], v, jab[i * 1 + 0]);
          jcd[3] = fma(dab[0], v, jcd[3]);
          kac[1] = fma(dbd[0], v, kac[1]);
          kad[0] = fma(dbc[1], v, kad[0]);
          kbc[1] = fma(dad[0], v, kbc[1]);
          kbd[0] = fma(dac[1], v, kbd[0]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 4];
          jab[i * 1 + 0] = fma(dcd[4], v, jab[i * 1 + 0]);
          jcd[4] = fma(dab[0], v, jcd[4]);
          kac[1] = fma(dbd[1], v, kac[1]);
          kad[1] = fma(dbc[1], v, kad[1]);
          kbc[1] = fma(dad[1], v, kbc[1]);
          kbd[1] = fma(dac[1], v, kbd[1]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 5];
          jab[i * 1 + 0] = fma(dcd[5], v, jab[i * 1 + 0]);
          jcd[5] = fma(dab[0], v, jcd[5]);
          kac[1] = fma(dbd[2], v, kac[1]);
          kad[2] = fma(dbc[1], v, kad[2]);
          kbc[1] = fma(dad[2], v, kbc[1]);
          kbd[2] = fma(dac[1], v, kbd[2]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 6];
          jab[i * 1 + 0] = fma(dcd[6], v, jab[i * 1 + 0]);
          jcd[6] = fma(dab[0], v, jcd[6]);
          kac[2] = fma(dbd[0], v, kac[2]);
          kad[0] = fma(dbc[2], v, kad[0]);
          kbc[2] = fma(dad[0], v, kbc[2]);
          kbd[0] = fma(dac[2], v, kbd[0]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 7];
          jab[i * 1 + 0] = fma(dcd[7], v, jab[i * 1 + 0]);
          jcd[7] = fma(dab[0], v, jcd[7]);
          kac[2] = fma(dbd[1], v, kac[2]);
          kad[1] = fma(dbc[2], v, kad[1]);
          kbc[2] = fma(dad[1], v, kbc[2]);
          kbd[1] = fma(dac[2], v, kbd[1]); }
        { const double v = f * res[(i * 1 + 0) * 9 + 8];
          jab[i * 1 + 0] = fma(dcd[8], v, jab[i * 1 + 0]);
          jcd[8] = fma(dab[0], v, jcd[8]);
          kac[2] = fma(dbd[2], v, kac[2]);
          kad[2] = fma(dbc[2], v, kad[2]);
          kbc[2] = fma(dad[2], v, kbc[2]);
          kbd[2] = fma(dac[2], v, kbd[2]); }
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.z + k], kac[k]);
#pragma unroll
        for (int l = 0; l < 3; ++l) atomicAdd(&jk.K[(ib_.z + i) * n + ik_.w + l], kad[l]);
    }
#pragma unroll
    for (int j = 0; j < 1; ++j) {
#pragma unroll
        for (int k = 0; k < 3; ++k) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.z + k], kbc[j * 3 + k]);
#pragma unroll
        for (int l = 0; l < 3; ++l) atomicAdd(&jk.K[(ib_.w + j) * n + ik_.w + l], kbd[j * 3 + l]);
    }
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int l = 0; l < 3; ++l) atomicAdd(&jk.J[(ik_.z + k) * n + ik_.w + l], 2.0 * jcd[k * 3 + l]);
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
__global__ void __launch_bounds__(128) eri_queue_dspp(const EriQueue Q) {
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
        double jab[JK ? 6 : 1];  // J/K digestion: the bra pair's J, over the chunk
        if constexpr (JK) {
#pragma unroll
            for (int x = 0; x < 6; ++x) jab[x] = 0.0;
        }
        for (int base = 0; base < cnt; base += W) {
        const int q = ch.y + base + kq;
        const bool live = base + kq < cnt;
        double acc[54];
        double2 bp = make_double2(0.0, 0.0), bq = bp;
        if (live) {
            bp = __ldg(&Q.pairs.bnd[p]);
            bq = __ldg(&Q.pairs.bnd[q]);
        }
        if (!live || bp.x * bq.x < Q.screen_cut) {
#pragma unroll
            for (int x = 0; x < 54; ++x) acc[x] = 0.0;
        } else {
            const int nb = __ldg(&Q.pairs.info[p]).y, nk = __ldg(&Q.pairs.info[q]).y;
            if (MIXED && bp.y * bq.y < Q.fp32_cut)
                vrr_dspp<float>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
            else vrr_dspp<double>(Q.pairs, Q.boys, p, q, is, nb, 1 << (lg - lgj), js, nk, 1 << lgj, acc);
        }
        if (lg) {
            for (int off = W; off < 32; off <<= 1) {
#pragma unroll
                for (int x = 0; x < 54; ++x) acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], off);
            }
        }
        const bool lead = live && s == 0;
        if (!JK && Q.scratch) {
            // two-phase: the leaders' HRR writes the blocks of the chunk's quartets straight
            // into shared memory, where they lie as in the scratch (consecutive slots); the warp
            // then copies them out as one contiguous run
            extern __shared__ double stg[];  // 4 * 32 * 54 doubles (launch_eri_dspp)
            double *sb = stg + (threadIdx.x >> 5) * (32 * 54);
            if (lead) hrr_dspp(Q.pairs, p, q, acc, sb + kq * 54);
            __syncwarp();
            const int nlive = min(W, cnt - base);
            double *__restrict__ dst = Q.scratch + __ldg(&Q.region[ch.w * kRegionFields]) +
                (__ldg(&Q.chunk_slot[c]) + base) * (long long)54;
            for (int t = lane; t < nlive * 54; t += 32) dst[t] = sb[t];
            __syncwarp();
        } else if (lead) {
            double res[54];
            hrr_dspp(Q.pairs, p, q, acc, res);
            if constexpr (JK) {
                const int4 ib_ = __ldg(&Q.pairs.info[p]), ik_ = __ldg(&Q.pairs.info[q]);
                jk_dspp(Q.jk, ib_, ik_, jk_weight(ib_.z == ib_.w, ik_.z == ik_.w, p == q), res, jab);
            } else {
                store_dspp(Q.out + __ldg(&Q.mol_out[ch.w]), __ldg(&Q.pairs.info[p]), __ldg(&Q.pairs.info[q]),
                            p == q, res);
            }
        }
        }
        if constexpr (JK) {
            // one addition per J_ab and chunk
            const int4 ib_ = __ldg(&Q.pairs.info[p]);
#pragma unroll
            for (int x = 0; x < 6; ++x) {
                double v = jab[x];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == 0) atomicAdd(&Q.jk.J[(long long)(ib_.z + x / 1) * Q.jk.n + ib_.w + x % 1], 2.0 * v);
            }
        }
    }
}


// The dynamic shared memory of the two-phase staging (55296 bytes), allowed once per device
// (before any graph capture: the occupancy query of plan creation calls it first).
static void eri_prepare_dspp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(eri_queue_dspp<0, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 55296);
        cudaFuncSetAttribute(eri_queue_dspp<1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 55296);
        done[dev] = true;
    }
}

void launch_eri_dspp(const EriQueue &Q, int mixed, int grid, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid <= 0) return;
    // two-phase plans stage the chunk's blocks in 55296 bytes of dynamic shared memory
    const size_t smem = Q.scratch && !Q.jk.J ? 55296 : 0;
    if (smem) eri_prepare_dspp();
    const bool jk = Q.jk.J != nullptr;
    if (mixed) { if (jk) eri_queue_dspp<1, 1><<<grid, 128, 0, s>>>(Q); else eri_queue_dspp<1, 0><<<grid, 128, smem, s>>>(Q); }
    else if (jk) eri_queue_dspp<0, 1><<<grid, 128, 0, s>>>(Q);
    else eri_queue_dspp<0, 0><<<grid, 128, smem, s>>>(Q);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_eri_dspp(int mixed) {
    eri_prepare_dspp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_dspp<1, 0>, 128, 0);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, eri_queue_dspp<0, 0>, 128, 0);
    return n;
}

}  // namespace molints
