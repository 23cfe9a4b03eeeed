// Generated by gen_rys.py -- Rys class (dd|pp).  Do not edit.
// roots 4, block 31 x 9, outputs 36 x 9, group 32 threads, 3 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 62208 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_ddpp {
    static constexpr int LA = 2, LB = 2, LC = 1, LD = 1;
    static constexpr int E = 4, F = 2, NR = 4;
    static constexpr int NA = 31, NC = 9, NBLK = 279;
    static constexpr int NB = 6, ND = 3;
    static constexpr int NAB = 36, NCD = 9;
    static constexpr int G = 32, W = 3, H = 1, PB = 2;
    static constexpr int S = 15, SI = 45, NCP = 9, NCDP = 9;
    static constexpr int SMEM_GROUP = 1944;
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
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[6], in[16]);
        const double h1 = fma(x, in[0], in[6]);
        const double h2 = fma(x, h1, h0);
        const double h3 = fma(y, in[6], in[17]);
        const double h4 = fma(y, in[0], in[7]);
        const double h5 = fma(x, h4, h3);
        const double h6 = fma(z, in[6], in[18]);
        const double h7 = fma(z, in[0], in[8]);
        const double h8 = fma(x, h7, h6);
        const double h9 = fma(y, in[7], in[19]);
        const double h10 = fma(y, h4, h9);
        const double h11 = fma(z, in[7], in[20]);
        const double h12 = fma(y, h7, h11);
        const double h13 = fma(z, in[8], in[21]);
        const double h14 = fma(z, h7, h13);
        const double h15 = fma(x, in[7], in[17]);
        const double h16 = fma(x, in[1], in[7]);
        const double h17 = fma(x, h16, h15);
        const double h18 = fma(y, in[1], in[9]);
        const double h19 = fma(x, h18, h9);
        const double h20 = fma(z, in[1], in[11]);
        const double h21 = fma(x, h20, h11);
        const double h22 = fma(y, in[9], in[22]);
        const double h23 = fma(y, h18, h22);
        const double h24 = fma(z, in[9], in[23]);
        const double h25 = fma(y, h20, h24);
        const double h26 = fma(z, in[11], in[24]);
        const double h27 = fma(z, h20, h26);
        const double h28 = fma(x, in[8], in[18]);
        const double h29 = fma(x, in[2], in[8]);
        const double h30 = fma(x, h29, h28);
        const double h31 = fma(y, in[8], in[20]);
        const double h32 = fma(y, in[2], in[11]);
        const double h33 = fma(x, h32, h31);
        const double h34 = fma(z, in[2], in[10]);
        const double h35 = fma(x, h34, h13);
        const double h36 = fma(y, in[11], in[23]);
        const double h37 = fma(y, h32, h36);
        const double h38 = fma(y, h34, h26);
        const double h39 = fma(z, in[10], in[25]);
        const double h40 = fma(z, h34, h39);
        const double h41 = fma(x, in[9], in[19]);
        const double h42 = fma(x, in[3], in[9]);
        const double h43 = fma(x, h42, h41);
        const double h44 = fma(y, in[3], in[12]);
        const double h45 = fma(x, h44, h22);
        const double h46 = fma(z, in[3], in[13]);
        const double h47 = fma(x, h46, h24);
        const double h48 = fma(y, in[12], in[26]);
        const double h49 = fma(y, h44, h48);
        const double h50 = fma(z, in[12], in[27]);
        const double h51 = fma(y, h46, h50);
        const double h52 = fma(z, in[13], in[28]);
        const double h53 = fma(z, h46, h52);
        const double h54 = fma(x, in[11], in[20]);
        const double h55 = fma(x, in[4], in[11]);
        const double h56 = fma(x, h55, h54);
        const double h57 = fma(y, in[4], in[13]);
        const double h58 = fma(x, h57, h36);
        const double h59 = fma(z, in[4], in[14]);
        const double h60 = fma(x, h59, h26);
        const double h61 = fma(y, in[13], in[27]);
        const double h62 = fma(y, h57, h61);
        const double h63 = fma(y, h59, h52);
        const double h64 = fma(z, in[14], in[29]);
        const double h65 = fma(z, h59, h64);
        const double h66 = fma(x, in[10], in[21]);
        const double h67 = fma(x, in[5], in[10]);
        const double h68 = fma(x, h67, h66);
        const double h69 = fma(y, in[10], in[24]);
        const double h70 = fma(y, in[5], in[14]);
        const double h71 = fma(x, h70, h69);
        const double h72 = fma(z, in[5], in[15]);
        const double h73 = fma(x, h72, h39);
        const double h74 = fma(y, in[14], in[28]);
        const double h75 = fma(y, h70, h74);
        const double h76 = fma(y, h72, h64);
        const double h77 = fma(z, in[15], in[30]);
        const double h78 = fma(z, h72, h77);
        out[0] = h2;
        out[9] = h5;
        out[18] = h8;
        out[27] = h10;
        out[36] = h12;
        out[45] = h14;
        out[54] = h17;
        out[63] = h19;
        out[72] = h21;
        out[81] = h23;
        out[90] = h25;
        out[99] = h27;
        out[108] = h30;
        out[117] = h33;
        out[126] = h35;
        out[135] = h37;
        out[144] = h38;
        out[153] = h40;
        out[162] = h43;
        out[171] = h45;
        out[180] = h47;
        out[189] = h49;
        out[198] = h51;
        out[207] = h53;
        out[216] = h56;
        out[225] = h58;
        out[234] = h60;
        out[243] = h62;
        out[252] = h63;
        out[261] = h65;
        out[270] = h68;
        out[279] = h71;
        out[288] = h73;
        out[297] = h75;
        out[306] = h76;
        out[315] = h78;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[0], in[3]);
        const double h1 = fma(y, in[0], in[4]);
        const double h2 = fma(z, in[0], in[5]);
        const double h3 = fma(x, in[1], in[4]);
        const double h4 = fma(y, in[1], in[6]);
        const double h5 = fma(z, in[1], in[7]);
        const double h6 = fma(x, in[2], in[5]);
        const double h7 = fma(y, in[2], in[7]);
        const double h8 = fma(z, in[2], in[8]);
        out[0] = h0 * (nrm * 1.0);
        out[1] = h1 * (nrm * 1.0);
        out[2] = h2 * (nrm * 1.0);
        out[3] = h3 * (nrm * 1.0);
        out[4] = h4 * (nrm * 1.0);
        out[5] = h5 * (nrm * 1.0);
        out[6] = h6 * (nrm * 1.0);
        out[7] = h7 * (nrm * 1.0);
        out[8] = h8 * (nrm * 1.0);
    }
};

__device__ const double kNormAB_ddpp[36] = {
    0.3333333333333334, 0.5773502691896258, 0.5773502691896258, 0.3333333333333334,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 1.0,
    1.0, 0.5773502691896258, 1.0, 0.5773502691896258,
    0.5773502691896258, 1.0, 1.0, 0.5773502691896258,
    1.0, 0.5773502691896258, 0.3333333333333334, 0.5773502691896258,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 0.3333333333333334,
    0.5773502691896258, 1.0, 1.0, 0.5773502691896258,
    1.0, 0.5773502691896258, 0.3333333333333334, 0.5773502691896258,
    0.5773502691896258, 0.3333333333333334, 0.5773502691896258, 0.3333333333333334,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_ddpp[9] = { 1, 16, 256, 2, 17, 257, 32, 272, 512 };

__device__ __forceinline__ RysClassTabs tabs_ddpp() {
    return RysClassTabs{kNormAB_ddpp, kCol_ddpp};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_ddpp(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_ddpp, MIXED>(Q, R, tabs_ddpp());
}

static void rys_prepare_ddpp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_ddpp<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 62208);
        cudaFuncSetAttribute(rys_queue_ddpp<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 62208);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_ddpp(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_ddpp();
    constexpr int ng = 128 / C_ddpp::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_ddpp<1><<<grid, 128, 62208, s>>>(Q, R);
    else rys_queue_ddpp<0><<<grid, 128, 62208, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_ddpp(int mixed) {
    rys_prepare_ddpp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_ddpp<1>, 128, 62208);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_ddpp<0>, 128, 62208);
    return n;
}

}  // namespace molints
