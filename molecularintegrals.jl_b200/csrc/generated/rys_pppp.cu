// Generated by gen_rys.py -- Rys class (pp|pp).  Do not edit.
// roots 3, block 9 x 9, outputs 9 x 9, group 32 threads, 3 ket pairs a round,
// 3 primitive quartets per ket pair and batch, 23328 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_pppp {
    static constexpr int LA = 1, LB = 1, LC = 1, LD = 1;
    static constexpr int E = 2, F = 2, NR = 3;
    static constexpr int NA = 9, NC = 9, NBLK = 81;
    static constexpr int NB = 3, ND = 3;
    static constexpr int NAB = 9, NCD = 9;
    static constexpr int G = 32, W = 3, H = 1, PB = 3;
    static constexpr int S = 9, SI = 27, NCP = 9, NCDP = 9;
    static constexpr int SMEM_GROUP = 729;
    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns
    template <typename T, typename A>
    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {
        acc[0] = fma(x[1] * y[0], z[0], acc[0]);
        acc[1] = fma(x[0] * y[1], z[0], acc[1]);
        acc[2] = fma(x[0] * y[0], z[1], acc[2]);
        acc[3] = fma(x[2] * y[0], z[0], acc[3]);
        acc[4] = fma(x[1] * y[1], z[0], acc[4]);
        acc[5] = fma(x[1] * y[0], z[1], acc[5]);
        acc[6] = fma(x[0] * y[2], z[0], acc[6]);
        acc[7] = fma(x[0] * y[1], z[1], acc[7]);
        acc[8] = fma(x[0] * y[0], z[2], acc[8]);
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
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
        out[0] = h0;
        out[9] = h1;
        out[18] = h2;
        out[27] = h3;
        out[36] = h4;
        out[45] = h5;
        out[54] = h6;
        out[63] = h7;
        out[72] = h8;
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

__device__ const double kNormAB_pppp[9] = {
    1.0, 1.0, 1.0, 1.0,
    1.0, 1.0, 1.0, 1.0,
    1.0,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_pppp[9] = { 1, 16, 256, 2, 17, 257, 32, 272, 512 };

__device__ __forceinline__ RysClassTabs tabs_pppp() {
    return RysClassTabs{kNormAB_pppp, kCol_pppp};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_pppp(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_pppp, MIXED>(Q, R, tabs_pppp());
}

static void rys_prepare_pppp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_pppp<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 23328);
        cudaFuncSetAttribute(rys_queue_pppp<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 23328);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_pppp(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_pppp();
    constexpr int ng = 128 / C_pppp::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_pppp<1><<<grid, 128, 23328, s>>>(Q, R);
    else rys_queue_pppp<0><<<grid, 128, 23328, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_pppp(int mixed) {
    rys_prepare_pppp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_pppp<1>, 128, 23328);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_pppp<0>, 128, 23328);
    return n;
}

}  // namespace molints
