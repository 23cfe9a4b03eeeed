// Generated by gen_rys.py -- Rys class (fs|fs).  Do not edit.
// roots 4, block 10 x 10, outputs 10 x 10, group 32 threads, 3 ket pairs a round,
// 2 primitive quartets per ket pair and batch, 37632 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_fsfs {
    static constexpr int LA = 3, LB = 0, LC = 3, LD = 0;
    static constexpr int E = 3, F = 3, NR = 4;
    static constexpr int NA = 10, NC = 10, NBLK = 100;
    static constexpr int NB = 1, ND = 1;
    static constexpr int NAB = 10, NCD = 10;
    static constexpr int G = 32, W = 3, H = 1, PB = 2;
    static constexpr int S = 16, SI = 49, NCP = 11, NCDP = 11;
    static constexpr int SMEM_GROUP = 1176;
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
        out[11] = in[1];
        out[22] = in[2];
        out[33] = in[3];
        out[44] = in[4];
        out[55] = in[5];
        out[66] = in[6];
        out[77] = in[7];
        out[88] = in[8];
        out[99] = in[9];
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

__device__ const double kNormAB_fsfs[10] = {
    0.2581988897471611, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    0.5773502691896258, 1.0, 0.2581988897471611, 0.5773502691896258,
    0.5773502691896258, 0.2581988897471611,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_fsfs[10] = { 3, 18, 258, 33, 513, 273, 48, 288, 528, 768 };

__device__ __forceinline__ RysClassTabs tabs_fsfs() {
    return RysClassTabs{kNormAB_fsfs, kCol_fsfs};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_fsfs(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_fsfs, MIXED>(Q, R, tabs_fsfs());
}

static void rys_prepare_fsfs() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_fsfs<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 37632);
        cudaFuncSetAttribute(rys_queue_fsfs<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 37632);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_fsfs(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_fsfs();
    constexpr int ng = 128 / C_fsfs::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_fsfs<1><<<grid, 128, 37632, s>>>(Q, R);
    else rys_queue_fsfs<0><<<grid, 128, 37632, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_fsfs(int mixed) {
    rys_prepare_fsfs();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fsfs<1>, 128, 37632);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_fsfs<0>, 128, 37632);
    return n;
}

}  // namespace molints
