// Generated by gen_rys.py -- Rys class (fd|fd).  Do not edit.
// roots 6, block 46 x 46, outputs 60 x 60, group 64 threads, 1 ket pairs a round,
// 9 primitive quartets per ket pair and batch, 103680 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_fdfd {
    static constexpr int LA = 3, LB = 2, LC = 3, LD = 2;
    static constexpr int E = 5, F = 5, NR = 6;
    static constexpr int NA = 46, NC = 46, NBLK = 2116;
    static constexpr int NB = 6, ND = 6;
    static constexpr int NAB = 60, NCD = 60;
    static constexpr int G = 64, W = 1, H = 1, PB = 9;
    static constexpr int S = 36, SI = 109, NCP = 47, NCDP = 61;
    static constexpr int SMEM_GROUP = 6480;
    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns
    template <typename T, typename A>
    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {
        acc[0] = fma(x[3] * y[0], z[0], acc[0]);
        acc[1] = fma(x[2] * y[1], z[0], acc[1]);
        acc[2] = fma(x[2] * y[0], z[1], acc[2]);
        acc[3] = fma(x[1] * y[2], z[0], acc[3]);
        acc[4] = fma(x[1] * y[0], z[2], acc[4]);
        acc[5] = fma(x[1] * y[1], z[1], acc[5]);
        acc[6] = fma(x[0] * y[3], z[0], acc[6]);
        acc[7] = fma(x[0] * y[2], z[1], acc[7]);
        acc[8] = fma(x[0] * y[1], z[2], acc[8]);
        acc[9] = fma(x[0] * y[0], z[3], acc[9]);
        acc[10] = fma(x[4] * y[0], z[0], acc[10]);
        acc[11] = fma(x[3] * y[1], z[0], acc[11]);
        acc[12] = fma(x[3] * y[0], z[1], acc[12]);
        acc[13] = fma(x[2] * y[2], z[0], acc[13]);
        acc[14] = fma(x[2] * y[1], z[1], acc[14]);
        acc[15] = fma(x[2] * y[0], z[2], acc[15]);
        acc[16] = fma(x[1] * y[3], z[0], acc[16]);
        acc[17] = fma(x[1] * y[2], z[1], acc[17]);
        acc[18] = fma(x[1] * y[1], z[2], acc[18]);
        acc[19] = fma(x[1] * y[0], z[3], acc[19]);
        acc[20] = fma(x[0] * y[4], z[0], acc[20]);
        acc[21] = fma(x[0] * y[3], z[1], acc[21]);
        acc[22] = fma(x[0] * y[2], z[2], acc[22]);
        acc[23] = fma(x[0] * y[1], z[3], acc[23]);
        acc[24] = fma(x[0] * y[0], z[4], acc[24]);
        acc[25] = fma(x[5] * y[0], z[0], acc[25]);
        acc[26] = fma(x[4] * y[1], z[0], acc[26]);
        acc[27] = fma(x[4] * y[0], z[1], acc[27]);
        acc[28] = fma(x[3] * y[2], z[0], acc[28]);
        acc[29] = fma(x[3] * y[1], z[1], acc[29]);
        acc[30] = fma(x[3] * y[0], z[2], acc[30]);
        acc[31] = fma(x[2] * y[3], z[0], acc[31]);
        acc[32] = fma(x[2] * y[2], z[1], acc[32]);
        acc[33] = fma(x[2] * y[1], z[2], acc[33]);
        acc[34] = fma(x[2] * y[0], z[3], acc[34]);
        acc[35] = fma(x[1] * y[4], z[0], acc[35]);
        acc[36] = fma(x[1] * y[3], z[1], acc[36]);
        acc[37] = fma(x[1] * y[2], z[2], acc[37]);
        acc[38] = fma(x[1] * y[1], z[3], acc[38]);
        acc[39] = fma(x[1] * y[0], z[4], acc[39]);
        acc[40] = fma(x[0] * y[5], z[0], acc[40]);
        acc[41] = fma(x[0] * y[4], z[1], acc[41]);
        acc[42] = fma(x[0] * y[3], z[2], acc[42]);
        acc[43] = fma(x[0] * y[2], z[3], acc[43]);
        acc[44] = fma(x[0] * y[1], z[4], acc[44]);
        acc[45] = fma(x[0] * y[0], z[5], acc[45]);
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[10], in[25]);
        const double h1 = fma(x, in[0], in[10]);
        const double h2 = fma(x, h1, h0);
        const double h3 = fma(y, in[10], in[26]);
        const double h4 = fma(y, in[0], in[11]);
        const double h5 = fma(x, h4, h3);
        const double h6 = fma(z, in[10], in[27]);
        const double h7 = fma(z, in[0], in[12]);
        const double h8 = fma(x, h7, h6);
        const double h9 = fma(y, in[11], in[28]);
        const double h10 = fma(y, h4, h9);
        const double h11 = fma(z, in[11], in[29]);
        const double h12 = fma(y, h7, h11);
        const double h13 = fma(z, in[12], in[30]);
        const double h14 = fma(z, h7, h13);
        const double h15 = fma(x, in[11], in[26]);
        const double h16 = fma(x, in[1], in[11]);
        const double h17 = fma(x, h16, h15);
        const double h18 = fma(y, in[1], in[13]);
        const double h19 = fma(x, h18, h9);
        const double h20 = fma(z, in[1], in[14]);
        const double h21 = fma(x, h20, h11);
        const double h22 = fma(y, in[13], in[31]);
        const double h23 = fma(y, h18, h22);
        const double h24 = fma(z, in[13], in[32]);
        const double h25 = fma(y, h20, h24);
        const double h26 = fma(z, in[14], in[33]);
        const double h27 = fma(z, h20, h26);
        const double h28 = fma(x, in[12], in[27]);
        const double h29 = fma(x, in[2], in[12]);
        const double h30 = fma(x, h29, h28);
        const double h31 = fma(y, in[12], in[29]);
        const double h32 = fma(y, in[2], in[14]);
        const double h33 = fma(x, h32, h31);
        const double h34 = fma(z, in[2], in[15]);
        const double h35 = fma(x, h34, h13);
        const double h36 = fma(y, in[14], in[32]);
        const double h37 = fma(y, h32, h36);
        const double h38 = fma(y, h34, h26);
        const double h39 = fma(z, in[15], in[34]);
        const double h40 = fma(z, h34, h39);
        const double h41 = fma(x, in[13], in[28]);
        const double h42 = fma(x, in[3], in[13]);
        const double h43 = fma(x, h42, h41);
        const double h44 = fma(y, in[3], in[16]);
        const double h45 = fma(x, h44, h22);
        const double h46 = fma(z, in[3], in[17]);
        const double h47 = fma(x, h46, h24);
        const double h48 = fma(y, in[16], in[35]);
        const double h49 = fma(y, h44, h48);
        const double h50 = fma(z, in[16], in[36]);
        const double h51 = fma(y, h46, h50);
        const double h52 = fma(z, in[17], in[37]);
        const double h53 = fma(z, h46, h52);
        const double h54 = fma(x, in[15], in[30]);
        const double h55 = fma(x, in[4], in[15]);
        const double h56 = fma(x, h55, h54);
        const double h57 = fma(y, in[15], in[33]);
        const double h58 = fma(y, in[4], in[18]);
        const double h59 = fma(x, h58, h57);
        const double h60 = fma(z, in[4], in[19]);
        const double h61 = fma(x, h60, h39);
        const double h62 = fma(y, in[18], in[37]);
        const double h63 = fma(y, h58, h62);
        const double h64 = fma(z, in[18], in[38]);
        const double h65 = fma(y, h60, h64);
        const double h66 = fma(z, in[19], in[39]);
        const double h67 = fma(z, h60, h66);
        const double h68 = fma(x, in[14], in[29]);
        const double h69 = fma(x, in[5], in[14]);
        const double h70 = fma(x, h69, h68);
        const double h71 = fma(y, in[5], in[17]);
        const double h72 = fma(x, h71, h36);
        const double h73 = fma(z, in[5], in[18]);
        const double h74 = fma(x, h73, h26);
        const double h75 = fma(y, in[17], in[36]);
        const double h76 = fma(y, h71, h75);
        const double h77 = fma(y, h73, h52);
        const double h78 = fma(z, h73, h64);
        const double h79 = fma(x, in[16], in[31]);
        const double h80 = fma(x, in[6], in[16]);
        const double h81 = fma(x, h80, h79);
        const double h82 = fma(y, in[6], in[20]);
        const double h83 = fma(x, h82, h48);
        const double h84 = fma(z, in[6], in[21]);
        const double h85 = fma(x, h84, h50);
        const double h86 = fma(y, in[20], in[40]);
        const double h87 = fma(y, h82, h86);
        const double h88 = fma(z, in[20], in[41]);
        const double h89 = fma(y, h84, h88);
        const double h90 = fma(z, in[21], in[42]);
        const double h91 = fma(z, h84, h90);
        const double h92 = fma(x, in[17], in[32]);
        const double h93 = fma(x, in[7], in[17]);
        const double h94 = fma(x, h93, h92);
        const double h95 = fma(y, in[7], in[21]);
        const double h96 = fma(x, h95, h75);
        const double h97 = fma(z, in[7], in[22]);
        const double h98 = fma(x, h97, h52);
        const double h99 = fma(y, in[21], in[41]);
        const double h100 = fma(y, h95, h99);
        const double h101 = fma(y, h97, h90);
        const double h102 = fma(z, in[22], in[43]);
        const double h103 = fma(z, h97, h102);
        const double h104 = fma(x, in[18], in[33]);
        const double h105 = fma(x, in[8], in[18]);
        const double h106 = fma(x, h105, h104);
        const double h107 = fma(y, in[8], in[22]);
        const double h108 = fma(x, h107, h62);
        const double h109 = fma(z, in[8], in[23]);
        const double h110 = fma(x, h109, h64);
        const double h111 = fma(y, in[22], in[42]);
        const double h112 = fma(y, h107, h111);
        const double h113 = fma(y, h109, h102);
        const double h114 = fma(z, in[23], in[44]);
        const double h115 = fma(z, h109, h114);
        const double h116 = fma(x, in[19], in[34]);
        const double h117 = fma(x, in[9], in[19]);
        const double h118 = fma(x, h117, h116);
        const double h119 = fma(y, in[19], in[38]);
        const double h120 = fma(y, in[9], in[23]);
        const double h121 = fma(x, h120, h119);
        const double h122 = fma(z, in[9], in[24]);
        const double h123 = fma(x, h122, h66);
        const double h124 = fma(y, in[23], in[43]);
        const double h125 = fma(y, h120, h124);
        const double h126 = fma(y, h122, h114);
        const double h127 = fma(z, in[24], in[45]);
        const double h128 = fma(z, h122, h127);
        out[0] = h2;
        out[47] = h5;
        out[94] = h8;
        out[141] = h10;
        out[188] = h12;
        out[235] = h14;
        out[282] = h17;
        out[329] = h19;
        out[376] = h21;
        out[423] = h23;
        out[470] = h25;
        out[517] = h27;
        out[564] = h30;
        out[611] = h33;
        out[658] = h35;
        out[705] = h37;
        out[752] = h38;
        out[799] = h40;
        out[846] = h43;
        out[893] = h45;
        out[940] = h47;
        out[987] = h49;
        out[1034] = h51;
        out[1081] = h53;
        out[1128] = h56;
        out[1175] = h59;
        out[1222] = h61;
        out[1269] = h63;
        out[1316] = h65;
        out[1363] = h67;
        out[1410] = h70;
        out[1457] = h72;
        out[1504] = h74;
        out[1551] = h76;
        out[1598] = h77;
        out[1645] = h78;
        out[1692] = h81;
        out[1739] = h83;
        out[1786] = h85;
        out[1833] = h87;
        out[1880] = h89;
        out[1927] = h91;
        out[1974] = h94;
        out[2021] = h96;
        out[2068] = h98;
        out[2115] = h100;
        out[2162] = h101;
        out[2209] = h103;
        out[2256] = h106;
        out[2303] = h108;
        out[2350] = h110;
        out[2397] = h112;
        out[2444] = h113;
        out[2491] = h115;
        out[2538] = h118;
        out[2585] = h121;
        out[2632] = h123;
        out[2679] = h125;
        out[2726] = h126;
        out[2773] = h128;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[10], in[25]);
        const double h1 = fma(x, in[0], in[10]);
        const double h2 = fma(x, h1, h0);
        const double h3 = fma(y, in[10], in[26]);
        const double h4 = fma(y, in[0], in[11]);
        const double h5 = fma(x, h4, h3);
        const double h6 = fma(z, in[10], in[27]);
        const double h7 = fma(z, in[0], in[12]);
        const double h8 = fma(x, h7, h6);
        const double h9 = fma(y, in[11], in[28]);
        const double h10 = fma(y, h4, h9);
        const double h11 = fma(z, in[11], in[29]);
        const double h12 = fma(y, h7, h11);
        const double h13 = fma(z, in[12], in[30]);
        const double h14 = fma(z, h7, h13);
        const double h15 = fma(x, in[11], in[26]);
        const double h16 = fma(x, in[1], in[11]);
        const double h17 = fma(x, h16, h15);
        const double h18 = fma(y, in[1], in[13]);
        const double h19 = fma(x, h18, h9);
        const double h20 = fma(z, in[1], in[14]);
        const double h21 = fma(x, h20, h11);
        const double h22 = fma(y, in[13], in[31]);
        const double h23 = fma(y, h18, h22);
        const double h24 = fma(z, in[13], in[32]);
        const double h25 = fma(y, h20, h24);
        const double h26 = fma(z, in[14], in[33]);
        const double h27 = fma(z, h20, h26);
        const double h28 = fma(x, in[12], in[27]);
        const double h29 = fma(x, in[2], in[12]);
        const double h30 = fma(x, h29, h28);
        const double h31 = fma(y, in[12], in[29]);
        const double h32 = fma(y, in[2], in[14]);
        const double h33 = fma(x, h32, h31);
        const double h34 = fma(z, in[2], in[15]);
        const double h35 = fma(x, h34, h13);
        const double h36 = fma(y, in[14], in[32]);
        const double h37 = fma(y, h32, h36);
        const double h38 = fma(y, h34, h26);
        const double h39 = fma(z, in[15], in[34]);
        const double h40 = fma(z, h34, h39);
        const double h41 = fma(x, in[13], in[28]);
        const double h42 = fma(x, in[3], in[13]);
        const double h43 = fma(x, h42, h41);
        const double h44 = fma(y, in[3], in[16]);
        const double h45 = fma(x, h44, h22);
        const double h46 = fma(z, in[3], in[17]);
        const double h47 = fma(x, h46, h24);
        const double h48 = fma(y, in[16], in[35]);
        const double h49 = fma(y, h44, h48);
        const double h50 = fma(z, in[16], in[36]);
        const double h51 = fma(y, h46, h50);
        const double h52 = fma(z, in[17], in[37]);
        const double h53 = fma(z, h46, h52);
        const double h54 = fma(x, in[15], in[30]);
        const double h55 = fma(x, in[4], in[15]);
        const double h56 = fma(x, h55, h54);
        const double h57 = fma(y, in[15], in[33]);
        const double h58 = fma(y, in[4], in[18]);
        const double h59 = fma(x, h58, h57);
        const double h60 = fma(z, in[4], in[19]);
        const double h61 = fma(x, h60, h39);
        const double h62 = fma(y, in[18], in[37]);
        const double h63 = fma(y, h58, h62);
        const double h64 = fma(z, in[18], in[38]);
        const double h65 = fma(y, h60, h64);
        const double h66 = fma(z, in[19], in[39]);
        const double h67 = fma(z, h60, h66);
        const double h68 = fma(x, in[14], in[29]);
        const double h69 = fma(x, in[5], in[14]);
        const double h70 = fma(x, h69, h68);
        const double h71 = fma(y, in[5], in[17]);
        const double h72 = fma(x, h71, h36);
        const double h73 = fma(z, in[5], in[18]);
        const double h74 = fma(x, h73, h26);
        const double h75 = fma(y, in[17], in[36]);
        const double h76 = fma(y, h71, h75);
        const double h77 = fma(y, h73, h52);
        const double h78 = fma(z, h73, h64);
        const double h79 = fma(x, in[16], in[31]);
        const double h80 = fma(x, in[6], in[16]);
        const double h81 = fma(x, h80, h79);
        const double h82 = fma(y, in[6], in[20]);
        const double h83 = fma(x, h82, h48);
        const double h84 = fma(z, in[6], in[21]);
        const double h85 = fma(x, h84, h50);
        const double h86 = fma(y, in[20], in[40]);
        const double h87 = fma(y, h82, h86);
        const double h88 = fma(z, in[20], in[41]);
        const double h89 = fma(y, h84, h88);
        const double h90 = fma(z, in[21], in[42]);
        const double h91 = fma(z, h84, h90);
        const double h92 = fma(x, in[17], in[32]);
        const double h93 = fma(x, in[7], in[17]);
        const double h94 = fma(x, h93, h92);
        const double h95 = fma(y, in[7], in[21]);
        const double h96 = fma(x, h95, h75);
        const double h97 = fma(z, in[7], in[22]);
        const double h98 = fma(x, h97, h52);
        const double h99 = fma(y, in[21], in[41]);
        const double h100 = fma(y, h95, h99);
        const double h101 = fma(y, h97, h90);
        const double h102 = fma(z, in[22], in[43]);
        const double h103 = fma(z, h97, h102);
        const double h104 = fma(x, in[18], in[33]);
        const double h105 = fma(x, in[8], in[18]);
        const double h106 = fma(x, h105, h104);
        const double h107 = fma(y, in[8], in[22]);
        const double h108 = fma(x, h107, h62);
        const double h109 = fma(z, in[8], in[23]);
        const double h110 = fma(x, h109, h64);
        const double h111 = fma(y, in[22], in[42]);
        const double h112 = fma(y, h107, h111);
        const double h113 = fma(y, h109, h102);
        const double h114 = fma(z, in[23], in[44]);
        const double h115 = fma(z, h109, h114);
        const double h116 = fma(x, in[19], in[34]);
        const double h117 = fma(x, in[9], in[19]);
        const double h118 = fma(x, h117, h116);
        const double h119 = fma(y, in[19], in[38]);
        const double h120 = fma(y, in[9], in[23]);
        const double h121 = fma(x, h120, h119);
        const double h122 = fma(z, in[9], in[24]);
        const double h123 = fma(x, h122, h66);
        const double h124 = fma(y, in[23], in[43]);
        const double h125 = fma(y, h120, h124);
        const double h126 = fma(y, h122, h114);
        const double h127 = fma(z, in[24], in[45]);
        const double h128 = fma(z, h122, h127);
        out[0] = h2 * (nrm * 0.14907119849998599);
        out[1] = h5 * (nrm * 0.2581988897471611);
        out[2] = h8 * (nrm * 0.2581988897471611);
        out[3] = h10 * (nrm * 0.14907119849998599);
        out[4] = h12 * (nrm * 0.2581988897471611);
        out[5] = h14 * (nrm * 0.14907119849998599);
        out[6] = h17 * (nrm * 0.3333333333333334);
        out[7] = h19 * (nrm * 0.5773502691896258);
        out[8] = h21 * (nrm * 0.5773502691896258);
        out[9] = h23 * (nrm * 0.3333333333333334);
        out[10] = h25 * (nrm * 0.5773502691896258);
        out[11] = h27 * (nrm * 0.3333333333333334);
        out[12] = h30 * (nrm * 0.3333333333333334);
        out[13] = h33 * (nrm * 0.5773502691896258);
        out[14] = h35 * (nrm * 0.5773502691896258);
        out[15] = h37 * (nrm * 0.3333333333333334);
        out[16] = h38 * (nrm * 0.5773502691896258);
        out[17] = h40 * (nrm * 0.3333333333333334);
        out[18] = h43 * (nrm * 0.3333333333333334);
        out[19] = h45 * (nrm * 0.5773502691896258);
        out[20] = h47 * (nrm * 0.5773502691896258);
        out[21] = h49 * (nrm * 0.3333333333333334);
        out[22] = h51 * (nrm * 0.5773502691896258);
        out[23] = h53 * (nrm * 0.3333333333333334);
        out[24] = h56 * (nrm * 0.3333333333333334);
        out[25] = h59 * (nrm * 0.5773502691896258);
        out[26] = h61 * (nrm * 0.5773502691896258);
        out[27] = h63 * (nrm * 0.3333333333333334);
        out[28] = h65 * (nrm * 0.5773502691896258);
        out[29] = h67 * (nrm * 0.3333333333333334);
        out[30] = h70 * (nrm * 0.5773502691896258);
        out[31] = h72 * (nrm * 1.0);
        out[32] = h74 * (nrm * 1.0);
        out[33] = h76 * (nrm * 0.5773502691896258);
        out[34] = h77 * (nrm * 1.0);
        out[35] = h78 * (nrm * 0.5773502691896258);
        out[36] = h81 * (nrm * 0.14907119849998599);
        out[37] = h83 * (nrm * 0.2581988897471611);
        out[38] = h85 * (nrm * 0.2581988897471611);
        out[39] = h87 * (nrm * 0.14907119849998599);
        out[40] = h89 * (nrm * 0.2581988897471611);
        out[41] = h91 * (nrm * 0.14907119849998599);
        out[42] = h94 * (nrm * 0.3333333333333334);
        out[43] = h96 * (nrm * 0.5773502691896258);
        out[44] = h98 * (nrm * 0.5773502691896258);
        out[45] = h100 * (nrm * 0.3333333333333334);
        out[46] = h101 * (nrm * 0.5773502691896258);
        out[47] = h103 * (nrm * 0.3333333333333334);
        out[48] = h106 * (nrm * 0.3333333333333334);
        out[49] = h108 * (nrm * 0.5773502691896258);
        out[50] = h110 * (nrm * 0.5773502691896258);
        out[51] = h112 * (nrm * 0.3333333333333334);
        out[52] = h113 * (nrm * 0.5773502691896258);
        out[53] = h115 * (nrm * 0.3333333333333334);
        out[54] = h118 * (nrm * 0.14907119849998599);
        out[55] = h121 * (nrm * 0.2581988897471611);
        out[56] = h123 * (nrm * 0.2581988897471611);
        out[57] = h125 * (nrm * 0.14907119849998599);
        out[58] = h126 * (nrm * 0.2581988897471611);
        out[59] = h128 * (nrm * 0.14907119849998599);
    }
};

__device__ const double kNormAB_fdfd[60] = {
    0.14907119849998599, 0.2581988897471611, 0.2581988897471611, 0.14907119849998599,
    0.2581988897471611, 0.14907119849998599, 0.3333333333333334, 0.5773502691896258,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.5773502691896258, 0.3333333333333334,
    0.5773502691896258, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.5773502691896258, 0.3333333333333334,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 1.0,
    1.0, 0.5773502691896258, 1.0, 0.5773502691896258,
    0.14907119849998599, 0.2581988897471611, 0.2581988897471611, 0.14907119849998599,
    0.2581988897471611, 0.14907119849998599, 0.3333333333333334, 0.5773502691896258,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.5773502691896258, 0.3333333333333334,
    0.5773502691896258, 0.3333333333333334, 0.14907119849998599, 0.2581988897471611,
    0.2581988897471611, 0.14907119849998599, 0.2581988897471611, 0.14907119849998599,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_fdfd[46] = { 3, 18, 258, 33, 513, 273, 48, 288, 528, 768, 4, 19, 259, 34, 274, 514, 49, 289, 529, 769, 64, 304, 544, 784, 1024, 5, 20, 260, 35, 275, 515, 50, 290, 530, 770, 65, 305, 545, 785, 1025, 80, 320, 560, 800, 1040, 1280 };

__device__ __forceinline__ RysClassTabs tabs_fdfd() {
    return RysClassTabs{kNormAB_fdfd, kCol_fdfd};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_fdfd(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_fdfd, MIXED>(Q, R, tabs_fdfd());
}

__global__ void __launch_bounds__(128) rys_bound_kernel_fdfd(PairTab P, RysTab R, int p0, int np,
                                                              double2 *pbound, const int *mol,
                                                              unsigned long long *qmax, double *qout, int full) {
    rys_bound_body<C_fdfd>(P, R, tabs_fdfd(), p0, np, pbound, mol, qmax, qout, full);
}

static void rys_prepare_fdfd() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_fdfd<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 103680);
        cudaFuncSetAttribute(rys_queue_fdfd<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 103680);
        cudaFuncSetAttribute(rys_bound_kernel_fdfd, cudaFuncAttributeMaxDynamicSharedMemorySize, 103680);
        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_fdfd(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_fdfd();
    constexpr int ng = 128 / C_fdfd::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_fdfd<1><<<grid, 128, 103680, s>>>(Q, R);
    else rys_queue_fdfd<0><<<grid, 128, 103680, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_fdfd(int mixed) {
    rys_prepare_fdfd();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fdfd<1>, 128, 103680);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fdfd<0>, 128, 103680);
    return n;
}

void launch_rys_bound_fdfd(const PairTab &P, const RysTab &R, int p0, int np, double2 *pbound,
                            const int *mol, unsigned long long *qmax, double *qout, int full, cudaStream_t s) {
    if (np <= 0) return;
    rys_prepare_fdfd();
    constexpr int ng = 128 / C_fdfd::G;
    rys_bound_kernel_fdfd<<<(np + ng - 1) / ng, 128, 103680, s>>>(P, R, p0, np, pbound, mol, qmax, qout,
                                                                             full);
}

}  // namespace molints
