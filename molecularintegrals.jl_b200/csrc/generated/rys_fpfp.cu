// Generated by gen_rys.py -- Rys class (fp|fp).  Do not edit.
// roots 5, block 25 x 25, outputs 30 x 30, group 32 threads, 1 ket pairs a round,
// 4 primitive quartets per ket pair and batch, 53760 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_fpfp {
    static constexpr int LA = 3, LB = 1, LC = 3, LD = 1;
    static constexpr int E = 4, F = 4, NR = 5;
    static constexpr int NA = 25, NC = 25, NBLK = 625;
    static constexpr int NB = 3, ND = 3;
    static constexpr int NAB = 30, NCD = 30;
    static constexpr int G = 32, W = 1, H = 1, PB = 4;
    static constexpr int S = 25, SI = 75, NCP = 25, NCDP = 31;
    static constexpr int SMEM_GROUP = 1680;
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
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[0], in[10]);
        const double h1 = fma(y, in[0], in[11]);
        const double h2 = fma(z, in[0], in[12]);
        const double h3 = fma(x, in[1], in[11]);
        const double h4 = fma(y, in[1], in[13]);
        const double h5 = fma(z, in[1], in[14]);
        const double h6 = fma(x, in[2], in[12]);
        const double h7 = fma(y, in[2], in[14]);
        const double h8 = fma(z, in[2], in[15]);
        const double h9 = fma(x, in[3], in[13]);
        const double h10 = fma(y, in[3], in[16]);
        const double h11 = fma(z, in[3], in[17]);
        const double h12 = fma(x, in[4], in[15]);
        const double h13 = fma(y, in[4], in[18]);
        const double h14 = fma(z, in[4], in[19]);
        const double h15 = fma(x, in[5], in[14]);
        const double h16 = fma(y, in[5], in[17]);
        const double h17 = fma(z, in[5], in[18]);
        const double h18 = fma(x, in[6], in[16]);
        const double h19 = fma(y, in[6], in[20]);
        const double h20 = fma(z, in[6], in[21]);
        const double h21 = fma(x, in[7], in[17]);
        const double h22 = fma(y, in[7], in[21]);
        const double h23 = fma(z, in[7], in[22]);
        const double h24 = fma(x, in[8], in[18]);
        const double h25 = fma(y, in[8], in[22]);
        const double h26 = fma(z, in[8], in[23]);
        const double h27 = fma(x, in[9], in[19]);
        const double h28 = fma(y, in[9], in[23]);
        const double h29 = fma(z, in[9], in[24]);
        out[0] = h0;
        out[25] = h1;
        out[50] = h2;
        out[75] = h3;
        out[100] = h4;
        out[125] = h5;
        out[150] = h6;
        out[175] = h7;
        out[200] = h8;
        out[225] = h9;
        out[250] = h10;
        out[275] = h11;
        out[300] = h12;
        out[325] = h13;
        out[350] = h14;
        out[375] = h15;
        out[400] = h16;
        out[425] = h17;
        out[450] = h18;
        out[475] = h19;
        out[500] = h20;
        out[525] = h21;
        out[550] = h22;
        out[575] = h23;
        out[600] = h24;
        out[625] = h25;
        out[650] = h26;
        out[675] = h27;
        out[700] = h28;
        out[725] = h29;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[0], in[10]);
        const double h1 = fma(y, in[0], in[11]);
        const double h2 = fma(z, in[0], in[12]);
        const double h3 = fma(x, in[1], in[11]);
        const double h4 = fma(y, in[1], in[13]);
        const double h5 = fma(z, in[1], in[14]);
        const double h6 = fma(x, in[2], in[12]);
        const double h7 = fma(y, in[2], in[14]);
        const double h8 = fma(z, in[2], in[15]);
        const double h9 = fma(x, in[3], in[13]);
        const double h10 = fma(y, in[3], in[16]);
        const double h11 = fma(z, in[3], in[17]);
        const double h12 = fma(x, in[4], in[15]);
        const double h13 = fma(y, in[4], in[18]);
        const double h14 = fma(z, in[4], in[19]);
        const double h15 = fma(x, in[5], in[14]);
        const double h16 = fma(y, in[5], in[17]);
        const double h17 = fma(z, in[5], in[18]);
        const double h18 = fma(x, in[6], in[16]);
        const double h19 = fma(y, in[6], in[20]);
        const double h20 = fma(z, in[6], in[21]);
        const double h21 = fma(x, in[7], in[17]);
        const double h22 = fma(y, in[7], in[21]);
        const double h23 = fma(z, in[7], in[22]);
        const double h24 = fma(x, in[8], in[18]);
        const double h25 = fma(y, in[8], in[22]);
        const double h26 = fma(z, in[8], in[23]);
        const double h27 = fma(x, in[9], in[19]);
        const double h28 = fma(y, in[9], in[23]);
        const double h29 = fma(z, in[9], in[24]);
        out[0] = h0 * (nrm * 0.2581988897471611);
        out[1] = h1 * (nrm * 0.2581988897471611);
        out[2] = h2 * (nrm * 0.2581988897471611);
        out[3] = h3 * (nrm * 0.5773502691896258);
        out[4] = h4 * (nrm * 0.5773502691896258);
        out[5] = h5 * (nrm * 0.5773502691896258);
        out[6] = h6 * (nrm * 0.5773502691896258);
        out[7] = h7 * (nrm * 0.5773502691896258);
        out[8] = h8 * (nrm * 0.5773502691896258);
        out[9] = h9 * (nrm * 0.5773502691896258);
        out[10] = h10 * (nrm * 0.5773502691896258);
        out[11] = h11 * (nrm * 0.5773502691896258);
        out[12] = h12 * (nrm * 0.5773502691896258);
        out[13] = h13 * (nrm * 0.5773502691896258);
        out[14] = h14 * (nrm * 0.5773502691896258);
        out[15] = h15 * (nrm * 1.0);
        out[16] = h16 * (nrm * 1.0);
        out[17] = h17 * (nrm * 1.0);
        out[18] = h18 * (nrm * 0.2581988897471611);
        out[19] = h19 * (nrm * 0.2581988897471611);
        out[20] = h20 * (nrm * 0.2581988897471611);
        out[21] = h21 * (nrm * 0.5773502691896258);
        out[22] = h22 * (nrm * 0.5773502691896258);
        out[23] = h23 * (nrm * 0.5773502691896258);
        out[24] = h24 * (nrm * 0.5773502691896258);
        out[25] = h25 * (nrm * 0.5773502691896258);
        out[26] = h26 * (nrm * 0.5773502691896258);
        out[27] = h27 * (nrm * 0.2581988897471611);
        out[28] = h28 * (nrm * 0.2581988897471611);
        out[29] = h29 * (nrm * 0.2581988897471611);
    }
};

__device__ const double kNormAB_fpfp[30] = {
    0.2581988897471611, 0.2581988897471611, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 1.0,
    1.0, 1.0, 0.2581988897471611, 0.2581988897471611,
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 0.2581988897471611,
    0.2581988897471611, 0.2581988897471611,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_fpfp[25] = { 3, 18, 258, 33, 513, 273, 48, 288, 528, 768, 4, 19, 259, 34, 274, 514, 49, 289, 529, 769, 64, 304, 544, 784, 1024 };

__device__ __forceinline__ RysClassTabs tabs_fpfp() {
    return RysClassTabs{kNormAB_fpfp, kCol_fpfp};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_fpfp(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_fpfp, MIXED>(Q, R, tabs_fpfp());
}

__global__ void __launch_bounds__(128) rys_bound_kernel_fpfp(PairTab P, RysTab R, int p0, int np,
                                                              double2 *pbound, const int *mol,
                                                              unsigned long long *qmax, double *qout, int full) {
    rys_bound_body<C_fpfp>(P, R, tabs_fpfp(), p0, np, pbound, mol, qmax, qout, full);
}

static void rys_prepare_fpfp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_fpfp<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 53760);
        cudaFuncSetAttribute(rys_queue_fpfp<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 53760);
        cudaFuncSetAttribute(rys_bound_kernel_fpfp, cudaFuncAttributeMaxDynamicSharedMemorySize, 53760);
        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_fpfp(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_fpfp();
    constexpr int ng = 128 / C_fpfp::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_fpfp<1><<<grid, 128, 53760, s>>>(Q, R);
    else rys_queue_fpfp<0><<<grid, 128, 53760, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_fpfp(int mixed) {
    rys_prepare_fpfp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fpfp<1>, 128, 53760);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fpfp<0>, 128, 53760);
    return n;
}

void launch_rys_bound_fpfp(const PairTab &P, const RysTab &R, int p0, int np, double2 *pbound,
                            const int *mol, unsigned long long *qmax, double *qout, int full, cudaStream_t s) {
    if (np <= 0) return;
    rys_prepare_fpfp();
    constexpr int ng = 128 / C_fpfp::G;
    rys_bound_kernel_fpfp<<<(np + ng - 1) / ng, 128, 53760, s>>>(P, R, p0, np, pbound, mol, qmax, qout,
                                                                             full);
}

}  // namespace molints
