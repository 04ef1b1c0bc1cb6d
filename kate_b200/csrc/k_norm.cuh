// ||psi||^2 of a complex64 state, summed by the kernel that holds the
// amplitudes: k_norm2_c64 (k_measure.cu) or a run's last block pass
// (k_block_c64.cu).
#pragma once

#include <cuda_runtime.h>

#include "launch.hpp"

namespace kate {

// renorm_scratch_bytes() of device memory, zeroed once.
struct NormScratch {
    double* part;     // RN_GRID per-CTA sums
    double* out;      // ||psi||^2, 1 / ||psi||
    unsigned* count;  // finished CTAs
};
inline NormScratch norm_scratch(void* scratch) {
    double* part = (double*)scratch;
    double* out = part + RN_GRID;
    return {part, out, (unsigned*)(out + 2)};
}

// Every thread of the N-thread CTA calls it with its sum. Each CTA adds its
// threads' sums in a fixed tree and writes its partial; the last CTA to finish
// adds the partials in a fixed order (deterministic), writes out[0] and
// out[1], and resets the counter for the next run.
template <int N>
__device__ __forceinline__ void finish_norm(double acc, const NormScratch& S) {
    __shared__ double red[N];
    __shared__ bool last;
    const uint32_t t = threadIdx.x;
    red[t] = acc;
    __syncthreads();
    for (int w = N / 2; w > 0; w >>= 1) {
        if (t < (uint32_t)w) red[t] += red[t + w];
        __syncthreads();
    }
    if (t == 0) {
        S.part[blockIdx.x] = red[0];
        __threadfence();
        last = atomicAdd(S.count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // Partials by the whole CTA, in a fixed order (one thread adding 592 of
    // them one after another took 20 us, most of the kernel at 21 qubits).
    __threadfence();
    double tot = 0.0;
    for (uint32_t c = t; c < gridDim.x; c += N) tot += __ldcg(S.part + c);
    red[t] = tot;
    __syncthreads();
    for (int w = N / 2; w > 0; w >>= 1) {
        if (t < (uint32_t)w) red[t] += red[t + w];
        __syncthreads();
    }
    if (t == 0) {
        tot = red[0];
        S.out[0] = tot;
        S.out[1] = tot > 0.0 ? 1.0 / sqrt(tot) : 1.0;
        *S.count = 0;
    }
}

}  // namespace kate
