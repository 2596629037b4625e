// The operator table of the sparse-MPO mixes (contract.cu, mixed.cu).
#pragma once

#include "nc_common.cuh"

namespace nc {
namespace {

constexpr int MIX_MAX_NNZ = 64;
constexpr int MIX_MAX_D = 4;
constexpr int MIX_T = 256;
constexpr int MIX_MAX_STAGE = 384;     // channels x d of a staged mix at most

// Matrices grouped by `to` (or `from`) index, in their own order within a group.
struct MixTable {
    cplx W[MIX_MAX_NNZ * MIX_MAX_D * MIX_MAX_D];
    int other[MIX_MAX_NNZ];          // the other index of each matrix
    int first[MIX_MAX_STAGE + 1];    // group k: matrices first[k] .. first[k+1] - 1
};
__device__ __forceinline__ void mix_table(MixTable& t, int nnz, int d, int groups, bool by_to, const uint32_t* __restrict__ idx,
                                          const cplx* __restrict__ W) {
    __shared__ int at[MIX_MAX_NNZ];
    for (int n = threadIdx.x; n < nnz; n += blockDim.x) {
        const int mine = (int)idx[2 * n + (by_to ? 1 : 0)];
        int pos = 0;   // matrices with a smaller key, or the same key and earlier
        for (int q = 0; q < nnz; ++q) {
            const int k = (int)idx[2 * q + (by_to ? 1 : 0)];
            pos += (k < mine || (k == mine && q < n)) ? 1 : 0;
        }
        at[n] = pos;
        t.other[pos] = (int)idx[2 * n + (by_to ? 0 : 1)] - 1;
    }
    for (int k = threadIdx.x; k <= groups; k += blockDim.x) {
        int pos = 0;
        for (int q = 0; q < nnz; ++q) pos += ((int)idx[2 * q + (by_to ? 1 : 0)] - 1 < k) ? 1 : 0;
        t.first[k] = pos;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < nnz * d * d; i += blockDim.x) t.W[at[i / (d * d)] * d * d + i % (d * d)] = W[i];
    __syncthreads();
}

}  // namespace
}  // namespace nc
