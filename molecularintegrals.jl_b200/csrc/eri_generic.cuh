// eri_generic.cuh -- the work list of the generic kernel (eri_generic.cu).
#pragma once
#include "eri_common.cuh"

namespace molints {

// Outputs of one unit of the generic kernel: a quartet of more ((gf|fp) and (gp|ff), 4500, and up) is several
// units, each of which sets the quartet's items up again.
constexpr int kGenTile = 4096;

// The primitive quartets of a shell quartet, the last shell's primitive fastest.  Unsigned: shells have
// up to 255 primitives, and 255^4 + 96 (a kernel's step) is below 2^32 where 164^4 x 3 roots, of a
// (gs|ss) quartet, is above 2^31.
struct GenPrims {
    int a, b, c, d;
};
__host__ __device__ inline unsigned gen_prim_count(const int *np) {
    return (unsigned)np[0] * (unsigned)np[1] * (unsigned)np[2] * (unsigned)np[3];
}
__host__ __device__ inline GenPrims gen_prim(unsigned k, const int *np) {
    GenPrims p;
    p.d = (int)(k % (unsigned)np[3]); k /= (unsigned)np[3];
    p.c = (int)(k % (unsigned)np[2]); k /= (unsigned)np[2];
    p.b = (int)(k % (unsigned)np[1]);
    p.a = (int)(k / (unsigned)np[1]);
    return p;
}

// The shell quartets with a g shell, as units of at most kGenTile outputs.
struct GenQuartets {
    const int4 *quartet;          // per unit: global shells (I, J, K, L), reference order
    const int2 *mol_tile;         // per unit: molecule, tile of the quartet's outputs
    long long n;                  // units
    int *counter;                 // next unit; zero at launch
    const double *xyz;            // shells: centre
    const int *L, *nprim, *poff, *fn_off;  // angular momentum, primitives, first function in molecule
    const double *expn, *ncoef;   // primitive exponents, normalised coefficients
    const long long *mol_out;     // packed offset of each molecule
    double *out;
    RysTab rys;
};
void launch_eri_generic(const GenQuartets &G, int num_sms, cudaStream_t s);

}  // namespace molints
