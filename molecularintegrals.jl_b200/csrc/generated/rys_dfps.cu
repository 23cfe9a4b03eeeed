// Generated by gen_rys.py -- Rys class (df|ps).  Do not edit.
// roots 4, block 52 x 3, outputs 60 x 3, group 32 threads, 5 ket pairs a round,
// 1 primitive quartets per ket pair and batch, 57600 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_dfps {
    static constexpr int LA = 2, LB = 3, LC = 1, LD = 0;
    static constexpr int E = 5, F = 1, NR = 4;
    static constexpr int NA = 52, NC = 3, NBLK = 156;
    static constexpr int NB = 10, ND = 1;
    static constexpr int NAB = 60, NCD = 3;
    static constexpr int G = 32, W = 5, H = 2, PB = 1;
    static constexpr int S = 12, SI = 37, NCP = 3, NCDP = 3;
    static constexpr int SMEM_GROUP = 1800;
    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns
    template <typename T, typename A>
    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {
        acc[0] = fma(x[2] * y[0], z[0], acc[0]);
        acc[1] = fma(x[1] * y[1], z[0], acc[1]);
        acc[2] = fma(x[1] * y[0], z[1], acc[2]);
        acc[3] = fma(x[0] * y[2], z[0], acc[3]);
        acc[4] = fma(x[0] * y[1], z[1], acc[4]);
        acc[5] = fma(x[0] * y[0], z[2], acc[5]);
        acc[6] = fma(x[3] * y[0], z[0], acc[6]);
        acc[7] = fma(x[2] * y[1], z[0], acc[7]);
        acc[8] = fma(x[2] * y[0], z[1], acc[8]);
        acc[9] = fma(x[1] * y[2], z[0], acc[9]);
        acc[10] = fma(x[1] * y[0], z[2], acc[10]);
        acc[11] = fma(x[1] * y[1], z[1], acc[11]);
        acc[12] = fma(x[0] * y[3], z[0], acc[12]);
        acc[13] = fma(x[0] * y[2], z[1], acc[13]);
        acc[14] = fma(x[0] * y[1], z[2], acc[14]);
        acc[15] = fma(x[0] * y[0], z[3], acc[15]);
        acc[16] = fma(x[4] * y[0], z[0], acc[16]);
        acc[17] = fma(x[3] * y[1], z[0], acc[17]);
        acc[18] = fma(x[3] * y[0], z[1], acc[18]);
        acc[19] = fma(x[2] * y[2], z[0], acc[19]);
        acc[20] = fma(x[2] * y[1], z[1], acc[20]);
        acc[21] = fma(x[2] * y[0], z[2], acc[21]);
        acc[22] = fma(x[1] * y[3], z[0], acc[22]);
        acc[23] = fma(x[1] * y[2], z[1], acc[23]);
        acc[24] = fma(x[1] * y[1], z[2], acc[24]);
        acc[25] = fma(x[1] * y[0], z[3], acc[25]);
        acc[26] = fma(x[0] * y[4], z[0], acc[26]);
        acc[27] = fma(x[0] * y[3], z[1], acc[27]);
        acc[28] = fma(x[0] * y[2], z[2], acc[28]);
        acc[29] = fma(x[0] * y[1], z[3], acc[29]);
        acc[30] = fma(x[0] * y[0], z[4], acc[30]);
        acc[31] = fma(x[5] * y[0], z[0], acc[31]);
        acc[32] = fma(x[4] * y[1], z[0], acc[32]);
        acc[33] = fma(x[4] * y[0], z[1], acc[33]);
        acc[34] = fma(x[3] * y[2], z[0], acc[34]);
        acc[35] = fma(x[3] * y[1], z[1], acc[35]);
        acc[36] = fma(x[3] * y[0], z[2], acc[36]);
        acc[37] = fma(x[2] * y[3], z[0], acc[37]);
        acc[38] = fma(x[2] * y[2], z[1], acc[38]);
        acc[39] = fma(x[2] * y[1], z[2], acc[39]);
        acc[40] = fma(x[2] * y[0], z[3], acc[40]);
        acc[41] = fma(x[1] * y[4], z[0], acc[41]);
        acc[42] = fma(x[1] * y[3], z[1], acc[42]);
        acc[43] = fma(x[1] * y[2], z[2], acc[43]);
        acc[44] = fma(x[1] * y[1], z[3], acc[44]);
        acc[45] = fma(x[1] * y[0], z[4], acc[45]);
        acc[46] = fma(x[0] * y[5], z[0], acc[46]);
        acc[47] = fma(x[0] * y[4], z[1], acc[47]);
        acc[48] = fma(x[0] * y[3], z[2], acc[48]);
        acc[49] = fma(x[0] * y[2], z[3], acc[49]);
        acc[50] = fma(x[0] * y[1], z[4], acc[50]);
        acc[51] = fma(x[0] * y[0], z[5], acc[51]);
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[16], in[31]);
        const double h1 = fma(x, in[6], in[16]);
        const double h2 = fma(x, h1, h0);
        const double h3 = fma(x, in[0], in[6]);
        const double h4 = fma(x, h3, h1);
        const double h5 = fma(x, h4, h2);
        const double h6 = fma(y, in[16], in[32]);
        const double h7 = fma(y, in[6], in[17]);
        const double h8 = fma(x, h7, h6);
        const double h9 = fma(y, in[0], in[7]);
        const double h10 = fma(x, h9, h7);
        const double h11 = fma(x, h10, h8);
        const double h12 = fma(z, in[16], in[33]);
        const double h13 = fma(z, in[6], in[18]);
        const double h14 = fma(x, h13, h12);
        const double h15 = fma(z, in[0], in[8]);
        const double h16 = fma(x, h15, h13);
        const double h17 = fma(x, h16, h14);
        const double h18 = fma(y, in[17], in[34]);
        const double h19 = fma(y, in[7], in[19]);
        const double h20 = fma(x, h19, h18);
        const double h21 = fma(y, h10, h20);
        const double h22 = fma(z, in[18], in[36]);
        const double h23 = fma(z, in[8], in[21]);
        const double h24 = fma(x, h23, h22);
        const double h25 = fma(z, h16, h24);
        const double h26 = fma(z, in[17], in[35]);
        const double h27 = fma(y, h13, h26);
        const double h28 = fma(z, in[7], in[20]);
        const double h29 = fma(y, h15, h28);
        const double h30 = fma(x, h29, h27);
        const double h31 = fma(y, in[19], in[37]);
        const double h32 = fma(y, h19, h31);
        const double h33 = fma(y, h9, h19);
        const double h34 = fma(y, h33, h32);
        const double h35 = fma(z, in[19], in[38]);
        const double h36 = fma(y, h28, h35);
        const double h37 = fma(y, h29, h36);
        const double h38 = fma(z, in[20], in[39]);
        const double h39 = fma(y, h23, h38);
        const double h40 = fma(z, h29, h39);
        const double h41 = fma(z, in[21], in[40]);
        const double h42 = fma(z, h23, h41);
        const double h43 = fma(z, h15, h23);
        const double h44 = fma(z, h43, h42);
        const double h45 = fma(x, in[17], in[32]);
        const double h46 = fma(x, in[7], in[17]);
        const double h47 = fma(x, h46, h45);
        const double h48 = fma(x, in[1], in[7]);
        const double h49 = fma(x, h48, h46);
        const double h50 = fma(x, h49, h47);
        const double h51 = fma(y, in[1], in[9]);
        const double h52 = fma(x, h51, h19);
        const double h53 = fma(x, h52, h20);
        const double h54 = fma(x, h28, h26);
        const double h55 = fma(z, in[1], in[11]);
        const double h56 = fma(x, h55, h28);
        const double h57 = fma(x, h56, h54);
        const double h58 = fma(y, in[9], in[22]);
        const double h59 = fma(x, h58, h31);
        const double h60 = fma(y, h52, h59);
        const double h61 = fma(z, in[11], in[24]);
        const double h62 = fma(x, h61, h38);
        const double h63 = fma(z, h56, h62);
        const double h64 = fma(z, in[9], in[23]);
        const double h65 = fma(y, h55, h64);
        const double h66 = fma(x, h65, h36);
        const double h67 = fma(y, in[22], in[41]);
        const double h68 = fma(y, h58, h67);
        const double h69 = fma(y, h51, h58);
        const double h70 = fma(y, h69, h68);
        const double h71 = fma(z, in[22], in[42]);
        const double h72 = fma(y, h64, h71);
        const double h73 = fma(y, h65, h72);
        const double h74 = fma(z, in[23], in[43]);
        const double h75 = fma(y, h61, h74);
        const double h76 = fma(z, h65, h75);
        const double h77 = fma(z, in[24], in[44]);
        const double h78 = fma(z, h61, h77);
        const double h79 = fma(z, h55, h61);
        const double h80 = fma(z, h79, h78);
        const double h81 = fma(x, in[18], in[33]);
        const double h82 = fma(x, in[8], in[18]);
        const double h83 = fma(x, h82, h81);
        const double h84 = fma(x, in[2], in[8]);
        const double h85 = fma(x, h84, h82);
        const double h86 = fma(x, h85, h83);
        const double h87 = fma(y, in[18], in[35]);
        const double h88 = fma(y, in[8], in[20]);
        const double h89 = fma(x, h88, h87);
        const double h90 = fma(y, in[2], in[11]);
        const double h91 = fma(x, h90, h88);
        const double h92 = fma(x, h91, h89);
        const double h93 = fma(z, in[2], in[10]);
        const double h94 = fma(x, h93, h23);
        const double h95 = fma(x, h94, h24);
        const double h96 = fma(y, in[20], in[38]);
        const double h97 = fma(y, in[11], in[23]);
        const double h98 = fma(x, h97, h96);
        const double h99 = fma(y, h91, h98);
        const double h100 = fma(z, in[10], in[25]);
        const double h101 = fma(x, h100, h41);
        const double h102 = fma(z, h94, h101);
        const double h103 = fma(y, h93, h61);
        const double h104 = fma(x, h103, h39);
        const double h105 = fma(y, in[23], in[42]);
        const double h106 = fma(y, h97, h105);
        const double h107 = fma(y, h90, h97);
        const double h108 = fma(y, h107, h106);
        const double h109 = fma(y, h103, h75);
        const double h110 = fma(y, h100, h77);
        const double h111 = fma(z, h103, h110);
        const double h112 = fma(z, in[25], in[45]);
        const double h113 = fma(z, h100, h112);
        const double h114 = fma(z, h93, h100);
        const double h115 = fma(z, h114, h113);
        const double h116 = fma(x, in[19], in[34]);
        const double h117 = fma(x, in[9], in[19]);
        const double h118 = fma(x, h117, h116);
        const double h119 = fma(x, in[3], in[9]);
        const double h120 = fma(x, h119, h117);
        const double h121 = fma(x, h120, h118);
        const double h122 = fma(y, in[3], in[12]);
        const double h123 = fma(x, h122, h58);
        const double h124 = fma(x, h123, h59);
        const double h125 = fma(x, h64, h35);
        const double h126 = fma(z, in[3], in[13]);
        const double h127 = fma(x, h126, h64);
        const double h128 = fma(x, h127, h125);
        const double h129 = fma(y, in[12], in[26]);
        const double h130 = fma(x, h129, h67);
        const double h131 = fma(y, h123, h130);
        const double h132 = fma(z, in[13], in[28]);
        const double h133 = fma(x, h132, h74);
        const double h134 = fma(z, h127, h133);
        const double h135 = fma(z, in[12], in[27]);
        const double h136 = fma(y, h126, h135);
        const double h137 = fma(x, h136, h72);
        const double h138 = fma(y, in[26], in[46]);
        const double h139 = fma(y, h129, h138);
        const double h140 = fma(y, h122, h129);
        const double h141 = fma(y, h140, h139);
        const double h142 = fma(z, in[26], in[47]);
        const double h143 = fma(y, h135, h142);
        const double h144 = fma(y, h136, h143);
        const double h145 = fma(z, in[27], in[48]);
        const double h146 = fma(y, h132, h145);
        const double h147 = fma(z, h136, h146);
        const double h148 = fma(z, in[28], in[49]);
        const double h149 = fma(z, h132, h148);
        const double h150 = fma(z, h126, h132);
        const double h151 = fma(z, h150, h149);
        const double h152 = fma(x, in[20], in[35]);
        const double h153 = fma(x, in[11], in[20]);
        const double h154 = fma(x, h153, h152);
        const double h155 = fma(x, in[4], in[11]);
        const double h156 = fma(x, h155, h153);
        const double h157 = fma(x, h156, h154);
        const double h158 = fma(y, in[4], in[13]);
        const double h159 = fma(x, h158, h97);
        const double h160 = fma(x, h159, h98);
        const double h161 = fma(z, in[4], in[14]);
        const double h162 = fma(x, h161, h61);
        const double h163 = fma(x, h162, h62);
        const double h164 = fma(y, in[13], in[27]);
        const double h165 = fma(x, h164, h105);
        const double h166 = fma(y, h159, h165);
        const double h167 = fma(z, in[14], in[29]);
        const double h168 = fma(x, h167, h77);
        const double h169 = fma(z, h162, h168);
        const double h170 = fma(y, h161, h132);
        const double h171 = fma(x, h170, h75);
        const double h172 = fma(y, in[27], in[47]);
        const double h173 = fma(y, h164, h172);
        const double h174 = fma(y, h158, h164);
        const double h175 = fma(y, h174, h173);
        const double h176 = fma(y, h170, h146);
        const double h177 = fma(y, h167, h148);
        const double h178 = fma(z, h170, h177);
        const double h179 = fma(z, in[29], in[50]);
        const double h180 = fma(z, h167, h179);
        const double h181 = fma(z, h161, h167);
        const double h182 = fma(z, h181, h180);
        const double h183 = fma(x, in[21], in[36]);
        const double h184 = fma(x, in[10], in[21]);
        const double h185 = fma(x, h184, h183);
        const double h186 = fma(x, in[5], in[10]);
        const double h187 = fma(x, h186, h184);
        const double h188 = fma(x, h187, h185);
        const double h189 = fma(y, in[21], in[39]);
        const double h190 = fma(y, in[10], in[24]);
        const double h191 = fma(x, h190, h189);
        const double h192 = fma(y, in[5], in[14]);
        const double h193 = fma(x, h192, h190);
        const double h194 = fma(x, h193, h191);
        const double h195 = fma(z, in[5], in[15]);
        const double h196 = fma(x, h195, h100);
        const double h197 = fma(x, h196, h101);
        const double h198 = fma(y, in[24], in[43]);
        const double h199 = fma(y, in[14], in[28]);
        const double h200 = fma(x, h199, h198);
        const double h201 = fma(y, h193, h200);
        const double h202 = fma(z, in[15], in[30]);
        const double h203 = fma(x, h202, h112);
        const double h204 = fma(z, h196, h203);
        const double h205 = fma(y, h195, h167);
        const double h206 = fma(x, h205, h110);
        const double h207 = fma(y, in[28], in[48]);
        const double h208 = fma(y, h199, h207);
        const double h209 = fma(y, h192, h199);
        const double h210 = fma(y, h209, h208);
        const double h211 = fma(y, h205, h177);
        const double h212 = fma(y, h202, h179);
        const double h213 = fma(z, h205, h212);
        const double h214 = fma(z, in[30], in[51]);
        const double h215 = fma(z, h202, h214);
        const double h216 = fma(z, h195, h202);
        const double h217 = fma(z, h216, h215);
        out[0] = h5;
        out[3] = h11;
        out[6] = h17;
        out[9] = h21;
        out[12] = h25;
        out[15] = h30;
        out[18] = h34;
        out[21] = h37;
        out[24] = h40;
        out[27] = h44;
        out[30] = h50;
        out[33] = h53;
        out[36] = h57;
        out[39] = h60;
        out[42] = h63;
        out[45] = h66;
        out[48] = h70;
        out[51] = h73;
        out[54] = h76;
        out[57] = h80;
        out[60] = h86;
        out[63] = h92;
        out[66] = h95;
        out[69] = h99;
        out[72] = h102;
        out[75] = h104;
        out[78] = h108;
        out[81] = h109;
        out[84] = h111;
        out[87] = h115;
        out[90] = h121;
        out[93] = h124;
        out[96] = h128;
        out[99] = h131;
        out[102] = h134;
        out[105] = h137;
        out[108] = h141;
        out[111] = h144;
        out[114] = h147;
        out[117] = h151;
        out[120] = h157;
        out[123] = h160;
        out[126] = h163;
        out[129] = h166;
        out[132] = h169;
        out[135] = h171;
        out[138] = h175;
        out[141] = h176;
        out[144] = h178;
        out[147] = h182;
        out[150] = h188;
        out[153] = h194;
        out[156] = h197;
        out[159] = h201;
        out[162] = h204;
        out[165] = h206;
        out[168] = h210;
        out[171] = h211;
        out[174] = h213;
        out[177] = h217;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0] * (nrm * 1.0);
        out[1] = in[1] * (nrm * 1.0);
        out[2] = in[2] * (nrm * 1.0);
    }
};

__device__ const double kNormAB_dfps[60] = {
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.3333333333333334,
    0.3333333333333334, 0.5773502691896258, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.14907119849998599, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 1.0,
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.2581988897471611,
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 1.0, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.2581988897471611, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.14907119849998599,
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 1.0, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.2581988897471611, 0.14907119849998599, 0.3333333333333334,
    0.3333333333333334, 0.3333333333333334, 0.3333333333333334, 0.5773502691896258,
    0.14907119849998599, 0.3333333333333334, 0.3333333333333334, 0.14907119849998599,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_dfps[3] = { 1, 16, 256 };

__device__ __forceinline__ RysClassTabs tabs_dfps() {
    return RysClassTabs{kNormAB_dfps, kCol_dfps};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_dfps(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_dfps, MIXED>(Q, R, tabs_dfps());
}

static void rys_prepare_dfps() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_dfps<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 57600);
        cudaFuncSetAttribute(rys_queue_dfps<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 57600);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_dfps(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_dfps();
    constexpr int ng = 128 / C_dfps::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_dfps<1><<<grid, 128, 57600, s>>>(Q, R);
    else rys_queue_dfps<0><<<grid, 128, 57600, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_dfps(int mixed) {
    rys_prepare_dfps();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dfps<1>, 128, 57600);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dfps<0>, 128, 57600);
    return n;
}

}  // namespace molints
