// eri_generic.cuh -- the work list of the generic kernel (eri_generic.cu).
#pragma once
#include "eri_common.cuh"

namespace molints {

// Outputs of one unit of the generic kernel: a quartet of more (from (gg|fd) up) is several units.
constexpr int kGenTile = 4096;

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
