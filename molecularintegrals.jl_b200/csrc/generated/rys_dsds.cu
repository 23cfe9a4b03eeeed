// Generated by gen_rys.py -- Rys class (ds|ds).  Do not edit.
// roots 3, block 6 x 6, outputs 6 x 6, group 32 threads, 5 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 25920 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_dsds {
    static constexpr int LA = 2, LB = 0, LC = 2, LD = 0;
    static constexpr int E = 2, F = 2, NR = 3;
    static constexpr int NA = 6, NC = 6, NBLK = 36;
    static constexpr int NB = 1, ND = 1;
    static constexpr int NAB = 6, NCD = 6;
    static constexpr int G = 32, W = 5, H = 1, PB = 2;
    static constexpr int S = 9, SI = 27, NCP = 7, NCDP = 7;
    static constexpr int SMEM_GROUP = 810;
    // stage 2: acc[row] += x[ax] y[ay] z[az] for the column's table columns
    template <typename T, typename A>
    __device__ __forceinline__ static void col_update(const T *x, const T *y, const T *z, A *acc) {
        acc[0] = fma(x[2] * y[0], z[0], acc[0]);
        acc[1] = fma(x[1] * y[1], z[0], acc[1]);
        acc[2] = fma(x[1] * y[0], z[1], acc[2]);
        acc[3] = fma(x[0] * y[2], z[0], acc[3]);
        acc[4] = fma(x[0] * y[1], z[1], acc[4]);
        acc[5] = fma(x[0] * y[0], z[2], acc[5]);
    }
    // bra HRR of one column (row stride NCP), ket HRR of one row times the component norms
    __device__ __forceinline__ static void bra_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0];
        out[7] = in[1];
        out[14] = in[2];
        out[21] = in[3];
        out[28] = in[4];
        out[35] = in[5];
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
        (void)x; (void)y; (void)z; (void)nrm;
        out[0] = in[0] * (nrm * 0.5773502691896258);
        out[1] = in[1] * (nrm * 1.0);
        out[2] = in[2] * (nrm * 1.0);
        out[3] = in[3] * (nrm * 0.5773502691896258);
        out[4] = in[4] * (nrm * 1.0);
        out[5] = in[5] * (nrm * 0.5773502691896258);
    }
};

__device__ const double kNormAB_dsds[6] = {
    0.5773502691896258, 1.0, 1.0, 0.5773502691896258,
    1.0, 0.5773502691896258,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_dsds[6] = { 2, 17, 257, 32, 272, 512 };

__device__ __forceinline__ RysClassTabs tabs_dsds() {
    return RysClassTabs{kNormAB_dsds, kCol_dsds};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_dsds(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_dsds, MIXED>(Q, R, tabs_dsds());
}

static void rys_prepare_dsds() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_dsds<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 25920);
        cudaFuncSetAttribute(rys_queue_dsds<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 25920);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_dsds(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_dsds();
    constexpr int ng = 128 / C_dsds::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_dsds<1><<<grid, 128, 25920, s>>>(Q, R);
    else rys_queue_dsds<0><<<grid, 128, 25920, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_dsds(int mixed) {
    rys_prepare_dsds();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dsds<1>, 128, 25920);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dsds<0>, 128, 25920);
    return n;
}

}  // namespace molints
