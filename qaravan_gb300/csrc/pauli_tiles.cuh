// Host interface of the tiled Pauli-sum kernels (pauli_tiles.cu).
#pragma once

#include "qgb_common.cuh"

namespace qgb_host {

struct PauliTerm {
    uint64_t x, z;  // X and Z masks over the state's bits (Y sets both)
    int ny;         // number of Y factors
    int slot;       // output slot
    double coeff;
};

// partials[(b * nterms + slot) * *nblk + blk], *nblk <= max_blocks per state.
// QGB_EDECLINE: the caller runs its general kernel.
int pauli_tiles_expect(const void* sv, int dtype, int n, const PauliTerm* terms, int nterms, int64_t batch,
                       int64_t stride, int max_blocks, double* partials, int* nblk, cudaStream_t st);
int pauli_tiles_apply(const void* sv, void* out, int dtype, int n, const PauliTerm* terms, int nterms, int64_t batch,
                      int64_t stride, cudaStream_t st);

}  // namespace qgb_host
