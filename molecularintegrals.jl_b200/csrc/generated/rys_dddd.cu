// Generated by gen_rys.py -- Rys class (dd|dd).  Do not edit.
// roots 5, block 31 x 31, outputs 36 x 36, group 32 threads, 1 ket pairs a round,
// 6 primitive quartets per ket pair and batch, 78336 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_dddd {
    static constexpr int LA = 2, LB = 2, LC = 2, LD = 2;
    static constexpr int E = 4, F = 4, NR = 5;
    static constexpr int NA = 31, NC = 31, NBLK = 961;
    static constexpr int NB = 6, ND = 6;
    static constexpr int NAB = 36, NCD = 36;
    static constexpr int G = 32, W = 1, H = 1, PB = 6;
    static constexpr int S = 25, SI = 75, NCP = 31, NCDP = 37;
    static constexpr int SMEM_GROUP = 2448;
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
        out[31] = h5;
        out[62] = h8;
        out[93] = h10;
        out[124] = h12;
        out[155] = h14;
        out[186] = h17;
        out[217] = h19;
        out[248] = h21;
        out[279] = h23;
        out[310] = h25;
        out[341] = h27;
        out[372] = h30;
        out[403] = h33;
        out[434] = h35;
        out[465] = h37;
        out[496] = h38;
        out[527] = h40;
        out[558] = h43;
        out[589] = h45;
        out[620] = h47;
        out[651] = h49;
        out[682] = h51;
        out[713] = h53;
        out[744] = h56;
        out[775] = h58;
        out[806] = h60;
        out[837] = h62;
        out[868] = h63;
        out[899] = h65;
        out[930] = h68;
        out[961] = h71;
        out[992] = h73;
        out[1023] = h75;
        out[1054] = h76;
        out[1085] = h78;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
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
        out[0] = h2 * (nrm * 0.3333333333333334);
        out[1] = h5 * (nrm * 0.5773502691896258);
        out[2] = h8 * (nrm * 0.5773502691896258);
        out[3] = h10 * (nrm * 0.3333333333333334);
        out[4] = h12 * (nrm * 0.5773502691896258);
        out[5] = h14 * (nrm * 0.3333333333333334);
        out[6] = h17 * (nrm * 0.5773502691896258);
        out[7] = h19 * (nrm * 1.0);
        out[8] = h21 * (nrm * 1.0);
        out[9] = h23 * (nrm * 0.5773502691896258);
        out[10] = h25 * (nrm * 1.0);
        out[11] = h27 * (nrm * 0.5773502691896258);
        out[12] = h30 * (nrm * 0.5773502691896258);
        out[13] = h33 * (nrm * 1.0);
        out[14] = h35 * (nrm * 1.0);
        out[15] = h37 * (nrm * 0.5773502691896258);
        out[16] = h38 * (nrm * 1.0);
        out[17] = h40 * (nrm * 0.5773502691896258);
        out[18] = h43 * (nrm * 0.3333333333333334);
        out[19] = h45 * (nrm * 0.5773502691896258);
        out[20] = h47 * (nrm * 0.5773502691896258);
        out[21] = h49 * (nrm * 0.3333333333333334);
        out[22] = h51 * (nrm * 0.5773502691896258);
        out[23] = h53 * (nrm * 0.3333333333333334);
        out[24] = h56 * (nrm * 0.5773502691896258);
        out[25] = h58 * (nrm * 1.0);
        out[26] = h60 * (nrm * 1.0);
        out[27] = h62 * (nrm * 0.5773502691896258);
        out[28] = h63 * (nrm * 1.0);
        out[29] = h65 * (nrm * 0.5773502691896258);
        out[30] = h68 * (nrm * 0.3333333333333334);
        out[31] = h71 * (nrm * 0.5773502691896258);
        out[32] = h73 * (nrm * 0.5773502691896258);
        out[33] = h75 * (nrm * 0.3333333333333334);
        out[34] = h76 * (nrm * 0.5773502691896258);
        out[35] = h78 * (nrm * 0.3333333333333334);
    }
};

__device__ const double kNormAB_dddd[36] = {
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
__device__ const uint16_t kCol_dddd[31] = { 2, 17, 257, 32, 272, 512, 3, 18, 258, 33, 513, 273, 48, 288, 528, 768, 4, 19, 259, 34, 274, 514, 49, 289, 529, 769, 64, 304, 544, 784, 1024 };

__device__ __forceinline__ RysClassTabs tabs_dddd() {
    return RysClassTabs{kNormAB_dddd, kCol_dddd};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_dddd(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_dddd, MIXED>(Q, R, tabs_dddd());
}

__global__ void __launch_bounds__(128) rys_bound_kernel_dddd(PairTab P, RysTab R, int p0, int np,
                                                              double2 *pbound, const int *mol,
                                                              unsigned long long *qmax, double *qout, int full) {
    rys_bound_body<C_dddd>(P, R, tabs_dddd(), p0, np, pbound, mol, qmax, qout, full);
}

static void rys_prepare_dddd() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_dddd<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 78336);
        cudaFuncSetAttribute(rys_queue_dddd<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 78336);
        cudaFuncSetAttribute(rys_bound_kernel_dddd, cudaFuncAttributeMaxDynamicSharedMemorySize, 78336);
        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_dddd(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_dddd();
    constexpr int ng = 128 / C_dddd::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_dddd<1><<<grid, 128, 78336, s>>>(Q, R);
    else rys_queue_dddd<0><<<grid, 128, 78336, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_dddd(int mixed) {
    rys_prepare_dddd();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dddd<1>, 128, 78336);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dddd<0>, 128, 78336);
    return n;
}

void launch_rys_bound_dddd(const PairTab &P, const RysTab &R, int p0, int np, double2 *pbound,
                            const int *mol, unsigned long long *qmax, double *qout, int full, cudaStream_t s) {
    if (np <= 0) return;
    rys_prepare_dddd();
    constexpr int ng = 128 / C_dddd::G;
    rys_bound_kernel_dddd<<<(np + ng - 1) / ng, 128, 78336, s>>>(P, R, p0, np, pbound, mol, qmax, qout,
                                                                             full);
}

}  // namespace molints
