// Complex64 tensor-core blocks: the device code shared by the simulator's
// pass kernel (k_block_c64.cu) and the batch kernel's block tasks
// (k_batch.cu). A pass applies up to KATE_C64_MAX_BLOCKS dense 5-qubit blocks
// (BlockProg, device_types.h) to 4096-amplitude coset tiles staged in shared
// memory. A group of G threads works on a tile (128, two groups per CTA, in
// the simulator's pass kernel and in the batch kernel's tasks of two tiles and
// more; the whole CTA, 256, in its tasks of a single tile); per block:
//   1. every thread builds its part of the MMA A operand from the staging
//      tile: row r = t & 127 (the values of the 7 non-block tile bits), all
//      32 block indices or (G = 256) the 16 of K half t >> 7, re/im
//      interleaved, as a BF16 hi part and the BF16 remainder (lo), and writes
//      it to TMEM (tcgen05.st; the A operand of tcgen05.mma may live in TMEM:
//      lane r, one 32-bit column per re/im pair);
//   2. one elected thread issues 4 K-steps x 3 products (A_hi.B_hi,
//      A_hi.B_lo, A_lo.B_hi; M = 128, N = 64, K = 16; A from TMEM, B from
//      shared memory) into one TMEM accumulator and commits to an mbarrier;
//   3. every thread reads its row's results back from TMEM and writes them
//      to the staging tile at the amplitudes' tile positions.
// Then the tile is written back with the pass's remap permutation (16-byte
// stores of amplitude pairs). All waits are bounded. Staging offsets are
// linear over GF(2) in the index, so every one is a per-thread base XOR a
// combination of a few values that are the same for all threads (one
// three-input XOR per access).
//
// Accuracy: hi + lo keeps ~16 bits of each FP32 operand and the dropped
// lo.lo product is ~2^-16 relative, so one block's relative error is about
// 1e-5 per amplitude; infidelity stays orders of magnitude below 1e-6 over a
// circuit (checked against complex128 by the tests and the bench).
#pragma once

#include <cuda_runtime.h>

#include "device_types.h"

namespace kate {
namespace blk {

constexpr int NT = 256;
constexpr int TB = KATE_TILE_BITS;  // 12 tile bits
constexpr int TS = 1 << TB;
constexpr uint32_t S_BYTES = TS * 8;  // one staging tile (float2)
// TMEM columns per tile: the FP32 accumulator (N = 64), then the A
// operand's hi and lo parts (128 lanes x 64 BF16 = 32 columns each).
constexpr uint32_t TMEM_COLS = 128;
constexpr uint32_t TM_AHI = 64, TM_ALO = 96;
#ifndef KATE_BLOCK_WAIT_LIMIT
#define KATE_BLOCK_WAIT_LIMIT (1L << 24)
#endif
constexpr long WAIT_LIMIT = KATE_BLOCK_WAIT_LIMIT;  // polls of an mbarrier before a wait gives up
// The pass's staging-tile swizzle (BlockProg::smask, chosen on the host):
// element e sits at e ^ sum_k parity(e & f[k]) << k. Linear over GF(2), so
// offsets of XOR-combined indices XOR.
struct Swz {
    uint32_t f0, f1, f2, f3;
    __device__ __forceinline__ uint32_t operator()(uint32_t e) const {
        return e ^ ((uint32_t)__popc(e & f0) & 1u) ^ (((uint32_t)__popc(e & f1) & 1u) << 1) ^
               (((uint32_t)__popc(e & f2) & 1u) << 2) ^ (((uint32_t)__popc(e & f3) & 1u) << 3);
    }
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Two floats rounded to BF16 (nearest even) and packed: lo in bits 0..15,
// hi in bits 16..31.
__device__ __forceinline__ uint32_t bf16x2_rn(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

// UMMA shared-memory descriptor, K-major, 128-byte swizzle: 8-row groups
// 1024 bytes apart (SBO), version 1.
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;            // leading byte offset (16 B; unused for swizzled K-major)
    d |= (uint64_t)(1024u >> 4) << 32;  // stride byte offset
    d |= (uint64_t)1u << 46;            // descriptor version for sm_100
    d |= (uint64_t)2u << 61;            // SWIZZLE_128B
    return d;
}

// Instruction descriptor: D F32, A/B BF16, both K-major, N = 64, M = 128.
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

// D (TMEM) += A (TMEM) x B (shared memory descriptor).
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(bdesc), "r"(IDESC), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

// 16 consecutive TMEM columns of this warp's 32 lanes from 16 registers per thread.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    for (long it = 0; it < WAIT_LIMIT; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Copies the pass's block operand images (nblocks x KATE_BLOCK_IMG_BYTES,
// contiguous per block, 16-byte aligned in global memory) into shared memory
// at `dst` (block b at dst + b * KATE_BLOCK_IMG_BYTES) with the bulk-copy
// engine: thread 0 announces the bytes on mbarrier `mbar` and issues one
// cp.async.bulk per image; every thread waits (bounded) for the phase
// `phase`, which it then flips. src(b) gives block b's global image.
// Returns false when the wait gave up.
template <typename Src>
__device__ __forceinline__ bool load_images(int nblocks, Src src, uint32_t dst, uint32_t mbar, uint32_t& phase) {
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar),
                     "r"((uint32_t)nblocks * KATE_BLOCK_IMG_BYTES)
                     : "memory");
        for (int b = 0; b < nblocks; b++)
            asm volatile(
                "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    dst + (uint32_t)b * KATE_BLOCK_IMG_BYTES),
                "l"(src(b)), "r"((uint32_t)KATE_BLOCK_IMG_BYTES), "r"(mbar)
                : "memory");
    }
    const bool ok = mbar_wait(mbar, phase);
    phase ^= 1u;
    return ok;
}

// TMEM allocation of one CTA, `cols` columns (a power of two, 32..512;
// warp 0 allocates; every thread reads the base after the barrier the
// caller places). `slot` is a shared-memory word.
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t cols) {
    if ((threadIdx.x >> 5) == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)),
                     "r"(cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}

// Frees the CTA's TMEM; every thread calls it (it synchronises the CTA).
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if ((threadIdx.x >> 5) == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols) : "memory");
    }
}

// A group's words in shared memory: the mbarrier of its products, and whether
// a wait of its threads gave up. Threads of other groups touch neither while
// the group works: between the barrier that ends a tile's last block, after
// which the group's threads read the flag, and the next tile's products,
// before which none of them can set it, lies another barrier of the group, so
// all of them read the same. (The groups of a CTA have no barrier in common.
// With one flag for both, a thread could see the other group's where its
// neighbours did not yet, and they would wait for one another at different
// barriers, without a bound.)
struct GroupSync {
    uint64_t mbar;
    int gave_up, pad;
};
constexpr uint32_t GAVE_UP = 8;  // its offset

// Barrier of the G threads that work on one tile: the CTA, or named barrier
// 1 + (the group's index).
template <int G>
__device__ __forceinline__ void group_bar() {
    if constexpr (G == NT) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + threadIdx.x / G), "n"(G) : "memory");
}

// Combinations of four basis values: combo(c, j) = XOR of the c's of the set
// bits of j, of which v[] holds those of bits 0, 1 and of bits 2, 3.
struct Combo4 {
    uint32_t v[6];  // b0, b1, b0 ^ b1, b2, b3, b2 ^ b3
    __device__ __forceinline__ void set(uint32_t b0, uint32_t b1, uint32_t b2, uint32_t b3) {
        v[0] = b0, v[1] = b1, v[2] = b0 ^ b1, v[3] = b2, v[4] = b3, v[5] = b2 ^ b3;
    }
    __device__ __forceinline__ uint32_t at(uint32_t base, int j) const {  // j a compile-time constant
        const uint32_t lo = (j & 3) ? v[(j & 3) - 1] : 0u, hi = (j >> 2) ? v[2 + (j >> 2)] : 0u;
        return base ^ lo ^ hi;
    }
};

// A pass's addressing for one thread of a G-thread group, built by setup()
// from a BlockProg. Copy j of thread t moves the amplitude pair e, e + 1 with
// e = 2t + 2G j (tile bit 0 is physical bit 0).
template <int G>
struct Pass {
    static constexpr int JB = G == 128 ? 4 : 3;  // bits of j
    static constexpr int NJ = 1 << JB;
    uint32_t row[KATE_C64_MAX_BLOCKS];   // swizzled offset of this thread's A row
    Combo4 blk[KATE_C64_MAX_BLOCKS];     // of block-index bits 0..3
    uint32_t blk4[KATE_C64_MAX_BLOCKS];  // of block-index bit 4
    uint64_t dT, dB[4];                  // global offsets of t and of each bit of j within a coset
    uint32_t cp_base, wb_base, o1;       // staging offsets: copy-in, write-back, write-back's second amplitude
    Combo4 cp, wb;                       // of the bits of j
    bool pairs;                          // amplitude pairs stay in one 16-byte staging slot
    __device__ __forceinline__ uint64_t dH(int j) const {
        uint64_t d = 0;
#pragma unroll
        for (int i = 0; i < JB; i++)
            if ((j >> i) & 1) d += dB[i];
        return d;
    }
};

template <int G>
__device__ __forceinline__ void setup(const BlockProg& P, Pass<G>& X) {
    constexpr int JB = Pass<G>::JB, TBITS = TB - 1 - JB;
    const uint32_t t = threadIdx.x & (uint32_t)(G - 1);
    const Swz sswz{P.smask[0], P.smask[1], P.smask[2], P.smask[3]};
    X.pairs = P.smask[0] == 0;
#pragma unroll
    for (int blk = 0; blk < KATE_C64_MAX_BLOCKS; blk++) {
        X.row[blk] = X.blk4[blk] = 0;
        X.blk[blk].set(0, 0, 0, 0);
        if (blk >= P.nblocks) continue;
        uint32_t bmask = 0;
        for (int i = 0; i < 5; i++) bmask |= 1u << P.btb[blk][i];
        const uint32_t r = t & 127u;  // TMEM lane 32 (warp & 3) + lane
        uint32_t d = 0;
        for (int i = 0, q = 0; i < TB; i++)
            if (!((bmask >> i) & 1u)) d |= ((r >> q++) & 1u) << i;
        X.row[blk] = sswz(d);
        X.blk[blk].set(sswz(1u << P.btb[blk][0]), sswz(1u << P.btb[blk][1]), sswz(1u << P.btb[blk][2]),
                       sswz(1u << P.btb[blk][3]));
        X.blk4[blk] = sswz(1u << P.btb[blk][4]);
    }
    uint64_t dT = 0;
    uint32_t pT = 0;
    for (int i = 0; i < TBITS; i++) {
        dT |= (uint64_t)((t >> i) & 1u) << P.tphys[i + 1];
        pT |= ((t >> i) & 1u) << P.outsrc[i + 1];
    }
    X.dT = dT;
    uint32_t c[4] = {0, 0, 0, 0}, w[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 4; i++) {
        X.dB[i] = 0;
        if (i >= JB) continue;
        X.dB[i] = 1ull << P.tphys[1 + TBITS + i];
        c[i] = sswz(2u * (uint32_t)G << i);
        w[i] = sswz(1u << P.outsrc[1 + TBITS + i]);
    }
    X.cp.set(c[0], c[1], c[2], c[3]);
    X.wb.set(w[0], w[1], w[2], w[3]);
    X.cp_base = sswz(2u * t);
    X.wb_base = sswz(pT);
    X.o1 = sswz(1u << P.outsrc[0]);
}

__device__ __forceinline__ uint64_t coset_base(const BlockProg& P, uint64_t c) {
    uint64_t b = 0;
    for (int i = 0; i < P.ncb; i++) b |= ((c >> i) & 1ull) << P.cphys[i];
    return b;
}

// Issues the copy of the tile at global base `cb` into the staging tile at
// shared address `sb` (no commit: the caller commits the group). Pairs go
// through L2 only (cp.async.cg). L2ONLY: the state may have been written by
// other SMs earlier in the same launch, so an unpaired swizzle's 8-byte
// copies (which cp.async can only route through L1) become L2 loads and
// shared stores, visible after the caller's barrier.
template <bool L2ONLY, int G>
__device__ __forceinline__ void load_tile(const float2* st, uint64_t cb, uint32_t sb, const Pass<G>& X) {
    const float2* src = st + cb + X.dT;
    if (X.pairs) {
#pragma unroll
        for (int j = 0; j < Pass<G>::NJ; j++) {
            const uint32_t d = sb + X.cp.at(X.cp_base, j) * 8u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src + X.dH(j)) : "memory");
        }
    } else if (L2ONLY) {
#pragma unroll 8
        for (int j = 0; j < Pass<G>::NJ; j++) {
            const uint32_t e0 = X.cp.at(X.cp_base, j);
            const float4 v = __ldcg(reinterpret_cast<const float4*>(src + X.dH(j)));
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(sb + e0 * 8u), "f"(v.x), "f"(v.y) : "memory");
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(sb + (e0 ^ 1u) * 8u), "f"(v.z), "f"(v.w)
                         : "memory");
        }
    } else {
        // The pair's two amplitudes land in different 8-byte slots.
#pragma unroll
        for (int j = 0; j < Pass<G>::NJ; j++) {
            const uint32_t e0 = X.cp.at(X.cp_base, j);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sb + e0 * 8u), "l"(src + X.dH(j))
                         : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sb + (e0 ^ 1u) * 8u),
                         "l"(src + X.dH(j) + 1)
                         : "memory");
        }
    }
}

// Fills the staging tile with the tile of |0...0>: zeros, and 1 at element
// 0 when `one` (coset 0; element 0 sits at staging offset 0 since the
// swizzle is linear).
template <int G>
__device__ __forceinline__ void zero_tile(float2* S, bool one) {
    const uint32_t t = threadIdx.x & (uint32_t)(G - 1);
    float4* s4 = reinterpret_cast<float4*>(S);
    for (uint32_t i = t; i < (uint32_t)TS / 2; i += G) s4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    group_bar<G>();
    if (one && t == 0) S[0] = make_float2(1.f, 0.f);
}

// Applies the pass's blocks to the staging tile S (its copy complete and
// visible to every thread of the group), in the 128 TMEM columns from tmem
// (accumulator, then the A parts). B images at shared address bimg (block b
// at bimg + b * KATE_BLOCK_IMG_BYTES, 1024-byte aligned). sync: shared address
// of the group's GroupSync. Returns false, to every thread of the group, when
// one of its waits for the products gave up; the tile is then undefined.
template <int G>
__device__ __forceinline__ bool apply_blocks(const BlockProg& P, const Pass<G>& X, float2* S, uint32_t bimg,
                                             uint32_t tmem, uint32_t sync, uint32_t& phase) {
    const uint32_t t = threadIdx.x & (uint32_t)(G - 1);
    const uint32_t lanes = tmem + (((threadIdx.x >> 5) & 3u) << 21);  // this warp's 32 lanes
    constexpr uint32_t NH = NT / G;                                   // K halves per thread
    for (int blk = 0; blk < P.nblocks; blk++) {
        const Combo4 C = blk == 0 ? X.blk[0] : X.blk[KATE_C64_MAX_BLOCKS - 1];
        const uint32_t row = blk == 0 ? X.row[0] : X.row[KATE_C64_MAX_BLOCKS - 1];
        const uint32_t b4 = blk == 0 ? X.blk4[0] : X.blk4[KATE_C64_MAX_BLOCKS - 1];
        const bool wide = P.btb[blk][0] == 0 && X.pairs;  // block index bit 0 = tile bit 0: 16-byte pairs
        // 1. A operands (hi, lo) from the staging tile into TMEM: block
        //    indices 16h..16h+15 are TMEM columns 16h..16h+15 of the A parts.
#pragma unroll
        for (uint32_t hh = 0; hh < NH; hh++) {
            const uint32_t h = G == NT ? t >> 7 : hh;
            const uint32_t base = h ? row ^ b4 : row;
            uint32_t hw[16], lw[16];
            auto split = [&](int e, float2 a) {
                const uint32_t hp = bf16x2_rn(a.x, a.y);
                const float hre = __uint_as_float(hp << 16), him = __uint_as_float(hp & 0xffff0000u);
                hw[e] = hp;
                lw[e] = bf16x2_rn(a.x - hre, a.y - him);
            };
            if (wide) {
#pragma unroll
                for (int e = 0; e < 16; e += 2) {
                    const float4 v = *reinterpret_cast<const float4*>(&S[C.at(base, e)]);
                    split(e, make_float2(v.x, v.y));
                    split(e + 1, make_float2(v.z, v.w));
                }
            } else {
#pragma unroll
                for (int e = 0; e < 16; e++) split(e, S[C.at(base, e)]);
            }
            tmem_st16(lanes + TM_AHI + h * 16u, hw);
            tmem_st16(lanes + TM_ALO + h * 16u, lw);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        group_bar<G>();
        // 2. Tensor-core products into TMEM.
        if (t == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t bb = bimg + (uint32_t)blk * KATE_BLOCK_IMG_BYTES;
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const uint32_t k = (uint32_t)s * 32u;  // K = 16 BF16 = 32 bytes per step (B)
                const uint32_t kc = (uint32_t)s * 8u;  // K = 16 BF16 = 8 TMEM columns per step (A)
                const uint64_t b_hi = sw128_desc(bb + k), b_lo = sw128_desc(bb + KATE_BLOCK_IMG_BYTES / 2 + k);
                mma_bf16_ts(tmem, tmem + TM_AHI + kc, b_hi, s > 0 ? 1u : 0u);
                mma_bf16_ts(tmem, tmem + TM_AHI + kc, b_lo, 1u);
                mma_bf16_ts(tmem, tmem + TM_ALO + kc, b_hi, 1u);
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(sync)
                         : "memory");
        }
        // Every thread waits for the products itself (try_wait suspends the
        // waiting thread), so no barrier sits between the products and the
        // read-back. A wait that gives up raises the flag; the read-back and
        // the next block still run (their values are then unused), so that
        // every thread takes the same barriers to the look at the flag.
        if (!mbar_wait(sync, phase)) asm volatile("st.shared.u32 [%0], 1;" ::"r"(sync + GAVE_UP) : "memory");
        phase ^= 1u;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // 3. Results: row t & 127, block indices 16h..16h+15 in columns
        //    32h..32h+31 of the accumulator.
#pragma unroll
        for (uint32_t hh = 0; hh < NH; hh++) {
            const uint32_t h = G == NT ? t >> 7 : hh;
            const uint32_t base = h ? row ^ b4 : row;
            uint32_t d[32];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                "[%32];"
                : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]),
                  "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]),
                  "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]),
                  "=r"(d[22]), "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]),
                  "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
                : "r"(lanes + h * 32u));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (wide) {
#pragma unroll
                for (int e = 0; e < 16; e += 2)
                    *reinterpret_cast<float4*>(&S[C.at(base, e)]) =
                        make_float4(__uint_as_float(d[2 * e]), __uint_as_float(d[2 * e + 1]),
                                    __uint_as_float(d[2 * e + 2]), __uint_as_float(d[2 * e + 3]));
            } else {
#pragma unroll
                for (int e = 0; e < 16; e++)
                    S[C.at(base, e)] = make_float2(__uint_as_float(d[2 * e]), __uint_as_float(d[2 * e + 1]));
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        group_bar<G>();
    }
    // Once per tile (once per block, the look took 30 ns of each). The vote
    // tells the compiler that the answer is the same for the warp; without it
    // the loop over tiles loses its uniform registers and spills.
    uint32_t stop;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(stop) : "r"(sync + GAVE_UP) : "memory");
    return !__any_sync(0xffffffffu, stop != 0);
}

// Writes the staging tile back with the remap permutation, an amplitude pair
// per store. st_cg: stores that bypass L1 (the state is read by other SMs
// later in the same launch). NORM: adds |a|^2 of this thread's amplitudes to
// `norm`.
template <bool CG, bool NORM, int G>
__device__ __forceinline__ void store_tile(const BlockProg& P, const Pass<G>& X, float2* st, uint64_t cb,
                                           const float2* S, double& norm) {
    float2* dst = st + cb + X.dT;
    auto put = [&](float2* p, float4 v) {
        if (NORM)
            norm += ((double)v.x * v.x + (double)v.y * v.y) + ((double)v.z * v.z + (double)v.w * v.w);
        if (CG) __stcg(reinterpret_cast<float4*>(p), v);
        else *reinterpret_cast<float4*>(p) = v;
    };
    if (P.outsrc[0] == 0 && X.pairs) {
        // Output bit 0 keeps input bit 0: the pair is one 16-byte slot.
#pragma unroll
        for (int j = 0; j < Pass<G>::NJ; j++)
            put(dst + X.dH(j), *reinterpret_cast<const float4*>(&S[X.wb.at(X.wb_base, j)]));
    } else {
#pragma unroll
        for (int j = 0; j < Pass<G>::NJ; j++) {
            const uint32_t e0 = X.wb.at(X.wb_base, j);
            const float2 v0 = S[e0], v1 = S[e0 ^ X.o1];
            put(dst + X.dH(j), make_float4(v0.x, v0.y, v1.x, v1.y));
        }
    }
}

// Zeros to every amplitude of a coset (a run from |0...0>: cosets other than
// the first stay zero under any blocks).
template <bool CG, int G>
__device__ __forceinline__ void store_zero(const Pass<G>& X, float2* st, uint64_t cb) {
    float2* dst = st + cb + X.dT;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < Pass<G>::NJ; j++) {
        float4* p = reinterpret_cast<float4*>(dst + X.dH(j));
        if (CG) __stcg(p, z);
        else *p = z;
    }
}

}  // namespace blk
}  // namespace kate
