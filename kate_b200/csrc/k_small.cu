// Whole circuits on states of fewer than 12 qubits: one launch of one CTA
// holds the state in shared memory from the initial state through every
// pass's register-staged program (k_stage.cuh) to the stored state and, for
// complex128 when asked for, the amplitude sums of the measurement.
//
// The state fits a fraction of one SM, so a run is a chain of dependent
// steps in one CTA and is bound by their latency: program dispatch, the FP64
// pipe's and the barriers at stage boundaries. A thread holds 4 amplitudes (8
// at 11 qubits, the most thread bits the programs address being 8), which
// gives the four schedulers eight warps at 10 qubits and keeps the unrolled
// ops in the instruction cache; with the tile kernel's 16 per thread two
// warps issued one instruction in five cycles, and a 10-qubit circuit of 290
// gates took 48 us.
// What this kernel removes is everything between the steps: with a generic
// kernel per 96 gates (one sweep of the tile, with its index arithmetic and
// a barrier, per gate), a memset, a one-element kernel, a measurement kernel
// and two copies, a 10-qubit circuit of 290 gates took 392 us on the GPU.
// Programs are copied into shared memory one pass ahead (two table buffers).
// Arithmetic is FP64 for complex64 states too; they are rounded once, when
// the state is stored.
#include "k_stage.cuh"
#include "launch.hpp"

namespace kate {

namespace {

using namespace stage;

// Program tables of one pass, as run_program reads them.
struct SmallTables {
    SOp ops[KATE_MAX_SOPS];
    double2 mats[KATE_MAX_MATS];
    uint16_t stab[KATE_MAX_STAGES][44];
};
static_assert(sizeof(SmallTables) % 16 == 0, "two of them follow each other");

__device__ __forceinline__ void copy16(void* dst, const unsigned char* src, int bytes, uint32_t t, uint32_t nt) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int i = (int)t * 16; i < bytes; i += (int)nt * 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + (uint32_t)i), "l"(src + i) : "memory");
}

__device__ __forceinline__ void prefetch(SmallTables& T, const BatchProg& P, const unsigned char* blob, uint32_t t,
                                         uint32_t nt) {
    copy16(T.ops, blob + P.ops_off, P.nops * (int)sizeof(SOp), t, nt);
    copy16(T.mats, blob + P.mats_off, P.nmats * 16, t, nt);
    copy16(T.stab, blob + P.stab_off, (P.nstages * 88 + 15) & ~15, t, nt);
}

// m: the programs' tile bits; 2^m / N threads run them. With fewer than 32 of
// these the warp's other lanes repeat them, so that every lane takes every
// barrier: the same values to the same places, since a stage stores only once
// the whole warp has loaded (run_program).
// init: 0 the state as it is, 1 |0...0>, 2 the product state PI.
// SM: whether a program has shared-memory ops (without them the program loop
// makes no call, and nothing is kept in memory around one).
template <bool SM, int N>
__global__ void __launch_bounds__(256)
    k_small(void* __restrict__ st, int c64, int n, int m, const BatchProg* __restrict__ progs, int p0, int p1,
            const unsigned char* __restrict__ blob, const DevOp* __restrict__ sops, const double2* __restrict__ pool,
            int init, const __grid_constant__ ProductInit PI, double2* __restrict__ sums) {
    extern __shared__ __align__(16) unsigned char small_raw[];
    SmallTables* T = reinterpret_cast<SmallTables*>(small_raw);
    double2* tile = reinterpret_cast<double2*>(T + 2);
    const uint32_t tb = (uint32_t)__cvta_generic_to_shared(tile);
    const uint32_t t = threadIdx.x, nt = blockDim.x, tp = t & ((1u << m) / N - 1u);
    const uint32_t size = 1u << m, dim = 1u << n;
    if (p0 < p1) prefetch(T[0], progs[p0], blob, t, nt);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    for (uint32_t x = t; x < size; x += nt) {
        double2 v = make_double2(0.0, 0.0);
        if (x < dim) {
            if (init == 0) {
                if (c64) {
                    const float2 f = reinterpret_cast<const float2*>(st)[x];
                    v = make_double2(f.x, f.y);
                } else {
                    v = reinterpret_cast<const double2*>(st)[x];
                }
            } else if (init == 1) {
                if (x == 0) v.x = 1.0;
            } else {
                v.x = 1.0;
                for (int q = 0; q < n; q++) {
                    const int b = (int)((x >> q) & 1u);
                    v = cmul(v, make_double2(PI.v[b][q][0], PI.v[b][q][1]));
                }
            }
        }
        tile[ops::swz(x)] = v;
    }
    for (int p = p0; p < p1; p++) {
        const int cur = (p - p0) & 1;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        // Program p and the tile are in place, and the other tables (of
        // program p - 1) are free.
        __syncthreads();
        if (p + 1 < p1) prefetch(T[cur ^ 1], progs[p + 1], blob, t, nt);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        run_program<double2, SM, 5, 0, N>(T[cur], progs[p].nops, tb, tile, 0, sops, progs[p].sop0, pool, tp, nullptr,
                                         nullptr, m, (int)nt, (int)t);
    }
    __syncthreads();
    for (uint32_t x = t; x < dim; x += nt) {
        const double2 v = tile[ops::swz(x)];
        if (c64) reinterpret_cast<float2*>(st)[x] = make_float2((float)v.x, (float)v.y);
        else reinterpret_cast<double2*>(st)[x] = v;
    }
    if (sums) {
        // Output 1 + 2b + v: the sum of the amplitudes with bit b = v, by 16
        // threads in a fixed order; outputs 1 and 2 make the total, output 0.
        const uint32_t half = dim / 2, i = t & 15u;
        for (uint32_t o0 = 0; o0 < 2u * (uint32_t)n; o0 += nt / 16) {
            const uint32_t o = o0 + (t >> 4), b = o >> 1;
            double2 s = make_double2(0.0, 0.0);
            if (o < 2u * (uint32_t)n)
                for (uint32_t k = i; k < half; k += 16)
                    s = dadd(s, tile[ops::swz(ins0(k, (int)b) | ((o & 1u) << b))]);
#pragma unroll
            for (int d = 8; d > 0; d >>= 1)
                s = dadd(s, make_double2(__shfl_down_sync(0xffffffffu, s.x, d, 16),
                                         __shfl_down_sync(0xffffffffu, s.y, d, 16)));
            if (i == 0 && o < 2u * (uint32_t)n) sums[1 + o] = s;
            if (o0 == 0) {
                const double2 r = make_double2(__shfl_down_sync(0xffffffffu, s.x, 16),
                                               __shfl_down_sync(0xffffffffu, s.y, 16));
                if (t == 0) sums[0] = dadd(s, r);
            }
        }
    }
}

size_t small_smem(int m) { return 2 * sizeof(SmallTables) + ((size_t)16 << m); }

}  // namespace

cudaError_t small_prepare(int device) {
    static bool done[64] = {false};
    if (device >= 0 && device < 64 && done[device]) return cudaSuccess;
    const int smem = (int)small_smem(KATE_TILE_BITS - 1);
    cudaError_t e = cudaSuccess;
    for (auto f : {k_small<false, 4>, k_small<true, 4>, k_small<false, 8>, k_small<true, 8>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess && device >= 0 && device < 64) done[device] = true;
    return e;
}

cudaError_t launch_small(void* st, int prec, int n, int reg_bits, const BatchProg* progs, int p0, int p1,
                         const void* blob, const DevOp* sops, const void* pool, bool smem_ops, int init,
                         const ProductInit& PI, void* sums, cudaStream_t s) {
    if (n < 1 || n >= KATE_TILE_BITS || (reg_bits != 2 && reg_bits != 3) || n - reg_bits > 8)
        return cudaErrorInvalidValue;
    const int m = n > reg_bits ? n : reg_bits + 1;
    const unsigned nt = m - reg_bits < 5 ? 32u : 1u << (m - reg_bits);
    const auto f = reg_bits == 2 ? (smem_ops ? k_small<true, 4> : k_small<false, 4>)
                                 : (smem_ops ? k_small<true, 8> : k_small<false, 8>);
    f<<<1, nt, small_smem(m), s>>>(st, prec, n, m, progs, p0, p1, (const unsigned char*)blob, sops,
                                   (const double2*)pool, init, PI, (double2*)sums);
    return cudaGetLastError();
}

}  // namespace kate
