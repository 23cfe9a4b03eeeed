// Generated by gen_rys.py -- Rys class (dp|dp).  Do not edit.
// roots 4, block 16 x 16, outputs 18 x 18, group 32 threads, 2 ket pairs a round,
// 3 primitive quartets per ket pair and batch, 41472 B shared per block.
#include "../rys_common.cuh"

namespace molints {

struct C_dpdp {
    static constexpr int LA = 2, LB = 1, LC = 2, LD = 1;
    static constexpr int E = 3, F = 3, NR = 4;
    static constexpr int NA = 16, NC = 16, NBLK = 256;
    static constexpr int NB = 3, ND = 3;
    static constexpr int NAB = 18, NCD = 18;
    static constexpr int G = 32, W = 2, H = 1, PB = 3;
    static constexpr int S = 16, SI = 49, NCP = 17, NCDP = 19;
    static constexpr int SMEM_GROUP = 1296;
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
        out[17] = h1;
        out[34] = h2;
        out[51] = h3;
        out[68] = h4;
        out[85] = h5;
        out[102] = h6;
        out[119] = h7;
        out[136] = h8;
        out[153] = h9;
        out[170] = h10;
        out[187] = h11;
        out[204] = h12;
        out[221] = h13;
        out[238] = h14;
        out[255] = h15;
        out[272] = h16;
        out[289] = h17;
    }
    __device__ __forceinline__ static void ket_hrr(const double *__restrict__ in, double x, double y, double z, double nrm, double *__restrict__ out) {
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
        out[0] = h0 * (nrm * 0.5773502691896258);
        out[1] = h1 * (nrm * 0.5773502691896258);
        out[2] = h2 * (nrm * 0.5773502691896258);
        out[3] = h3 * (nrm * 1.0);
        out[4] = h4 * (nrm * 1.0);
        out[5] = h5 * (nrm * 1.0);
        out[6] = h6 * (nrm * 1.0);
        out[7] = h7 * (nrm * 1.0);
        out[8] = h8 * (nrm * 1.0);
        out[9] = h9 * (nrm * 0.5773502691896258);
        out[10] = h10 * (nrm * 0.5773502691896258);
        out[11] = h11 * (nrm * 0.5773502691896258);
        out[12] = h12 * (nrm * 1.0);
        out[13] = h13 * (nrm * 1.0);
        out[14] = h14 * (nrm * 1.0);
        out[15] = h15 * (nrm * 0.5773502691896258);
        out[16] = h16 * (nrm * 0.5773502691896258);
        out[17] = h17 * (nrm * 0.5773502691896258);
    }
};

__device__ const double kNormAB_dpdp[18] = {
    0.5773502691896258, 0.5773502691896258, 0.5773502691896258, 1.0,
    1.0, 1.0, 1.0, 1.0,
    1.0, 0.5773502691896258, 0.5773502691896258, 0.5773502691896258,
    1.0, 1.0, 1.0, 0.5773502691896258,
    0.5773502691896258, 0.5773502691896258,
};

// column components cx | cy << 4 | cz << 8
__device__ const uint16_t kCol_dpdp[16] = { 2, 17, 257, 32, 272, 512, 3, 18, 258, 33, 513, 273, 48, 288, 528, 768 };

__device__ __forceinline__ RysClassTabs tabs_dpdp() {
    return RysClassTabs{kNormAB_dpdp, kCol_dpdp};
}

template <int MIXED>
__global__ void __launch_bounds__(128) rys_queue_dpdp(const EriQueue Q, const RysTab R) {
    rys_queue_body<C_dpdp, MIXED>(Q, R, tabs_dpdp());
}

static void rys_prepare_dpdp() {
    static bool done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !done[dev]) {
        cudaFuncSetAttribute(rys_queue_dpdp<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, 41472);
        cudaFuncSetAttribute(rys_queue_dpdp<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, 41472);

        done[dev] = true;
    }
}

// grid_max: resident blocks on the device; the grid is cut to the chunks' groups.
void launch_rys_dpdp(const EriQueue &Q, const RysTab &R, int mixed, int grid_max, cudaStream_t s) {
    if (Q.nchunks <= 0 || grid_max <= 0) return;
    rys_prepare_dpdp();
    constexpr int ng = 128 / C_dpdp::G;
    const int grid = (int)std::min<long long>(grid_max, ((long long)Q.nchunks + ng - 1) / ng);
    if (mixed) rys_queue_dpdp<1><<<grid, 128, 41472, s>>>(Q, R);
    else rys_queue_dpdp<0><<<grid, 128, 41472, s>>>(Q, R);
}

// Resident blocks of 128 threads per SM for the queue kernel (sizes the persistent grid).
int occupancy_rys_dpdp(int mixed) {
    rys_prepare_dpdp();
    int n = 0;
    if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dpdp<1>, 128, 41472);
    else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, rys_queue_dpdp<0>, 128, 41472);
    return n;
}

}  // namespace molints
