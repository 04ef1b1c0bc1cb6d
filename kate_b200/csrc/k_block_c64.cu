// Complex64 group pass with 5-qubit dense blocks on the tensor cores
// (tcgen05, kind::f16 with BF16 operands, split-BF16 products, FP32
// accumulation in TMEM); the block arithmetic is in k_block.cuh.
//
// Each CTA (256 threads; two CTAs per SM, ~97 KiB of shared memory each) is
// two groups of 128 threads, each with a 4096-amplitude coset tile of its own
// in a grid-stride loop: staging buffer, barrier, mbarrier and TMEM columns.
// A tile's blocks are a chain of latencies (operands to TMEM, products, their
// completion, results back), so what counts is how many tiles are on their
// way per SM: four groups overlap each other's chains and tile copies
// (16-byte cp.async of amplitude pairs; tile bit 0 is physical bit 0): a
// two-block pass over 2^30 amplitudes takes 3.6 ms, against 4.9 with the CTA
// working on one tile and a second buffer prefetching the next (2.6 at the
// copy rate). The
// block matrices (B operands, hi and lo) are staged in shared memory once per
// CTA. A run from |0...0> reads nothing in its first pass. A run's last pass
// also sums ||psi||^2 of what it stores (FP64, per thread, then per CTA; the
// CTA that finishes last adds the CTAs' sums in their order), which saves the
// renormalisation's read of the state (a 21-qubit run 170 -> 166 us, 26 qubits
// 3.36 -> 3.21 ms, 30 qubits 96.0 -> 94.2 ms). All waits are
// bounded: on timeout the kernel records an error flag for the host and
// returns after its copies in flight completed, freeing its TMEM.
#include <cuda_runtime.h>

#include "k_block.cuh"
#include "k_common.cuh"
#include "k_norm.cuh"
#include "launch.hpp"

namespace kate {

namespace {

using namespace blk;

constexpr int G = 128, NG = NT / G;                                             // groups per CTA
constexpr uint32_t OFF_B = 0;                                                   // blocks' B images
constexpr uint32_t OFF_S = OFF_B + KATE_C64_MAX_BLOCKS * KATE_BLOCK_IMG_BYTES;  // a staging tile per group
constexpr uint32_t OFF_MISC = OFF_S + NG * S_BYTES;  // groups' words, images' mbarrier, TMEM slot
constexpr uint32_t SMEM_BYTES = OFF_MISC + 64 + 1024;  // + alignment slack

template <bool NORM>
__global__ void __launch_bounds__(NT, 2)
    k_block_c64(float2* __restrict__ st, const __grid_constant__ BlockProg P, const uint8_t* __restrict__ bimg,
                int from_zero, int* __restrict__ err, NormScratch N) {
    extern __shared__ uint8_t smem_raw[];
    let_next_start();
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // 1024-byte aligned operand region
    uint8_t* gbase = smem_raw + (base - raw);
    const uint32_t t = threadIdx.x, grp = t / G;
    constexpr uint32_t GS = sizeof(GroupSync);
    GroupSync* groups = reinterpret_cast<GroupSync*>(gbase + OFF_MISC);
    const uint32_t sync = base + OFF_MISC + GS * grp, mbar_img = base + OFF_MISC + GS * NG;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + OFF_MISC + GS * NG + 8);
    if (t == 0) {
        for (int i = 0; i <= NG; i++)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(base + OFF_MISC + GS * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < NG; i++) groups[i].gave_up = 0;
    }
    tmem_alloc(tmem_slot, NG * TMEM_COLS);
    __syncthreads();
    // Block matrices: B images into shared memory once, by the bulk-copy engine.
    uint32_t phase_img = 0;
    if (!load_images(P.nblocks, [&](int b) { return bimg + P.bimg[b]; }, base + OFF_B, mbar_img, phase_img) &&
        t == 0)
        for (int i = 0; i < NG; i++) groups[i].gave_up = 1;
    Pass<G> X;
    setup(P, X);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot + grp * TMEM_COLS;

    const uint64_t ncos = 1ull << P.ncb;
    float2* S = reinterpret_cast<float2*>(gbase + OFF_S + grp * S_BYTES);
    const uint32_t sb = base + OFF_S + grp * S_BYTES;
    uint32_t phase = 0;
    double norm = 0.0;
    wait_for_previous();  // everything above reads only what no pass writes
    for (uint64_t c = (uint64_t)blockIdx.x * NG + grp; c < ncos; c += (uint64_t)gridDim.x * NG) {
        const uint64_t cb = coset_base(P, c);
        if (from_zero) {
            if (cb) {
                store_zero<false>(X, st, cb);
                continue;
            }
            zero_tile<G>(S, true);
        } else {
            load_tile<false>(st, cb, sb, X);
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        }
        group_bar<G>();
        if (!apply_blocks(P, X, S, base + OFF_B, tmem, sync, phase)) break;
        store_tile<false, NORM>(P, X, st, cb, S, norm);
        group_bar<G>();
    }
    if (groups[grp].gave_up && t % G == 0) atomicExch(err, 1);
    tmem_free(*tmem_slot, NG * TMEM_COLS);
    if constexpr (NORM) finish_norm<NT>(norm, N);
}

}  // namespace

int block_c64_grid(int n, int device) {
    static int cached[64] = {0};
    if (device < 0 || device >= 64) device = 0;
    if (!cached[device]) {
        for (auto* k : {k_block_c64<false>, k_block_c64<true>}) {
            cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_BYTES);
            cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        }
        int sms = 148, smem_sm = 0, reserved = 0;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
        cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
        // Registers allow two CTAs (__launch_bounds__); shared memory decides.
        int occ = smem_sm / (int)(SMEM_BYTES + reserved);
        if (occ < 1) occ = 1;
        if (occ > 2) occ = 2;
        cached[device] = sms * occ < RN_GRID ? sms * occ : RN_GRID;
    }
    const uint64_t nctas = ((1ull << (n - TB)) + NG - 1) / NG;
    return (int)(nctas < (uint64_t)cached[device] ? nctas : (uint64_t)cached[device]);
}

cudaError_t launch_block_c64(void* st, const BlockProg& prog, const void* bimg, bool from_zero, int* err, int grid,
                             void* norm, cudaStream_t s) {
    if (prog.m != TB || prog.nblocks < 1 || prog.nblocks > KATE_C64_MAX_BLOCKS) return cudaErrorInvalidValue;
    if (prog.tphys[0] != 0) return cudaErrorInvalidValue;  // amplitude pairs must be contiguous
    return launch_after(norm ? k_block_c64<true> : k_block_c64<false>, grid, NT, SMEM_BYTES, s, (float2*)st, prog,
                        (const uint8_t*)bimg, (int)from_zero, err, norm ? norm_scratch(norm) : NormScratch{});
}

}  // namespace kate
