// Generated by gen_rys.py -- Rys class (fp|fs).  Do not edit.
// roots 4, block 25 x 10, outputs 30 x 10, group 32 threads, 3 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 63360 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_fpfs {
    static constexpr int LA = 3, LB = 1, LC = 3, LD = 0;
    static constexpr int E = 4, F = 3, NR = 4;
    static constexpr int NA = 25, NC = 10, NBLK = 250;
    static constexpr int NB = 3, ND = 1;
    static constexpr int NAB = 30, NCD = 10;
    static constexpr int G = 32, W = 3, H = 1, PB = 2;
    static constexpr int S = 20, SI = 61, NCP = 11, NCDP = 11;
    static constexpr int SMEM_GROUP = 1980;
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
        out[11] = h1;
        out[22] = h2;
        out[33] = h3;
        out[44] = h4;
        out[55] = h5;
        out[66] = h6;
        out[77] = h7;
        out[88] = h8;
        out[99] = h9;
        out[110] = h10;
        out[121] = h11;
        out[132] = h12;
        out[143] = h13;
        out[154] = h14;
        out[165] = h15;
        out[176] = h16;
        out[187] = h17;
        out[198] = h18;
        out[209] = h19;
        out[220] = h20;
        out[231] = h21;
        out[242] = h22;
        out[253] = h23;
        out[264] = h24;
        out[275] = h25;
        out[286] = h26;
        out[297] = h27;
        out[308] = h28;
        out[319] = h29;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0] * (nrm * 0.2581988897471611);
        out[1] = in[1] * (nrm * 0.5773502691896258);
        out[2] = in[2] * (nrm * 0.5773502691896258);
        out[3] = in[3] * (nrm * 0.5773502691896258);
        out[4] = in[4] * (nrm * 0.5773502691896258);
        out[5] = in[5] * (nrm * 1.0);
        out[6] = in[6] * (nrm * 0.2581988897471611);
        out[7] = in[7] * (nrm * 0.5773502691896258);
        out[8] = in[8] * (nrm * 0.5773502691896258);
        out[9] = in[9] * (nrm * 0.2581988897471611);
    }
};

__device__ const double kNormAB_fpfs[30] = {
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
__device__ const uint16_t kCol_fpfs[10] = { 3, 18, 258, 33, 513, 273, 48, 288, 528, 768 };

__device__ __forceinline__ RysClassTabs tabs_fpfs() {
    return RysClassTabs{kNormAB_fpfs, kCol_fpfs};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_fpfs(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_fpfs, MIXED>(Q, R, tabs_fpfs());
}

static void rys_prepare_fpfs() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_fpfs<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 63360);
        cudaFuncSetAttribute(rys_queue_fpfs<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 63360);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_fpfs(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_fpfs();
    constexpr int ng = 128 / C_fpfs::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_fpfs<1><<<grid, 128, 63360, s>>>(Q, R);
    else rys_queue_fpfs<0><<<grid, 128, 63360, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_fpfs(int mixed) {
    rys_prepare_fpfs();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fpfs<1>, 128, 63360);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fpfs<0>, 128, 63360);
    return n;
}

}  // namespace molints
