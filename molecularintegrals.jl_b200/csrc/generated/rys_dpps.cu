// Generated by gen_rys.py -- Rys class (dp|ps).  Do not edit.
// roots 3, block 16 x 3, outputs 18 x 3, group 32 threads, 5 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 24000 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_dpps {
    static constexpr int LA = 2, LB = 1, LC = 1, LD = 0;
    static constexpr int E = 3, F = 1, NR = 3;
    static constexpr int NA = 16, NC = 3, NBLK = 48;
    static constexpr int NB = 3, ND = 1;
    static constexpr int NAB = 18, NCD = 3;
    static constexpr int G = 32, W = 5, H = 2, PB = 2;
    static constexpr int S = 8, SI = 25, NCP = 3, NCDP = 3;
    static constexpr int SMEM_GROUP = 750;
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
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        const double h0 = fma(x, in[0], in[6]);
        const double h1 = fma(y, in[0], in[7]);
        const double h2 = fma(z, in[0], in[8]);
        const double h3 = fma(x, in[1], in[7]);
        const double h4 = fma(y, in[1], in[9]);
        const double h5 = fma(z, in[1], in[11]);
        const double h6 = fma(x, in[2], in[8]);
        const double h7 = fma(y, in[2], in[11]);
        const double h8 = fma(z, in[2], in[10]);
        const double h9 = fma(x, in[3], in[9]);
        const double h10 = fma(y, in[3], in[12]);
        const double h11 = fma(z, in[3], in[13]);
        const double h12 = fma(x, in[4], in[11]);
        const double h13 = fma(y, in[4], in[13]);
        const double h14 = fma(z, in[4], in[14]);
        const double h15 = fma(x, in[5], in[10]);
        const double h16 = fma(y, in[5], in[14]);
        const double h17 = fma(z, in[5], in[15]);
        out[0] = h0;
        out[3] = h1;
        out[6] = h2;
        out[9] = h3;
        out[12] = h4;
        out[15] = h5;
        out[18] = h6;
        out[21] = h7;
        out[24] = h8;
        out[27] = h9;
        out[30] = h10;
        out[33] = h11;
        out[36] = h12;
        out[39] = h13;
        out[42] = h14;
        out[45] = h15;
        out[48] = h16;
        out[51] = h17;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0] * (nrm * 1.0);
        out[1] = in[1] * (nrm * 1.0);
        out[2] = in[2] * (nrm * 1.0);
    }
};

__device__ const double kNormAB_dpps[18] = {
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 1.0,
    1.0, 1.0, 1.0, 1.0,
    1.0, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    1.0, 1.0, 1.0, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_dpps[3] = { 1, 16, 256 };

__device__ __forceinline__ RysClassTabs tabs_dpps() {
    return RysClassTabs{kNormAB_dpps, kCol_dpps};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_dpps(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_dpps, MIXED>(Q, R, tabs_dpps());
}

static void rys_prepare_dpps() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_dpps<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 24000);
        cudaFuncSetAttribute(rys_queue_dpps<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 24000);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_dpps(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_dpps();
    constexpr int ng = 128 / C_dpps::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_dpps<1><<<grid, 128, 24000, s>>>(Q, R);
    else rys_queue_dpps<0><<<grid, 128, 24000, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_dpps(int mixed) {
    rys_prepare_dpps();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dpps<1>, 128, 24000);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dpps<0>, 128, 24000);
    return n;
}

}  // namespace molints
