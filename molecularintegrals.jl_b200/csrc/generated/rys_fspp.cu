// Generated by gen_rys.py -- Rys class (fs|pp).  Do not edit.
// roots 3, block 10 x 9, outputs 10 x 9, group 32 threads, 3 ket pairs a round,
// 3 primitive quartets per ket pair and batch, 31968 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_fspp {
    static constexpr int LA = 3, LB = 0, LC = 1, LD = 1;
    static constexpr int E = 3, F = 2, NR = 3;
    static constexpr int NA = 10, NC = 9, NBLK = 90;
    static constexpr int NB = 1, ND = 3;
    static constexpr int NAB = 10, NCD = 9;
    static constexpr int G = 32, W = 3, H = 1, PB = 3;
    static constexpr int S = 12, SI = 37, NCP = 9, NCDP = 9;
    static constexpr int SMEM_GROUP = 999;
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
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0];
        out[9] = in[1];
        out[18] = in[2];
        out[27] = in[3];
        out[36] = in[4];
        out[45] = in[5];
        out[54] = in[6];
        out[63] = in[7];
        out[72] = in[8];
        out[81] = in[9];
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

__device__ const double kNormAB_fspp[10] = {
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 1.0, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.2581988897471611,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_fspp[9] = { 1, 16, 256, 2, 17, 257, 32, 272, 512 };

__device__ __forceinline__ RysClassTabs tabs_fspp() {
    return RysClassTabs{kNormAB_fspp, kCol_fspp};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_fspp(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_fspp, MIXED>(Q, R, tabs_fspp());
}

static void rys_prepare_fspp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_fspp<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 31968);
        cudaFuncSetAttribute(rys_queue_fspp<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 31968);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_fspp(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_fspp();
    constexpr int ng = 128 / C_fspp::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_fspp<1><<<grid, 128, 31968, s>>>(Q, R);
    else rys_queue_fspp<0><<<grid, 128, 31968, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_fspp(int mixed) {
    rys_prepare_fspp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fspp<1>, 128, 31968);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fspp<0>, 128, 31968);
    return n;
}

}  // namespace molints
