// Persistent batch kernel: many independent circuits in one launch.
//
// CTAs take tasks from a global queue (one atomicAdd per task). A task
// first waits, with a time-bounded spin, until the tasks of its circuit that
// it depends on have finished (per-circuit counters), then runs:
//   BT_SMALL  the whole circuit in shared memory: |0...0>, every pass
//             program back to back on the same tile, <Z_q>; the state never
//             touches HBM;
//   BT_PASS   one group pass program over a range of cosets: 16-byte
//             cp.async loads (L2 only: other SMs wrote the state earlier in
//             this launch), the register-staged program, stores that bypass
//             L1. The first pass of a circuit starts from |0...0> in shared
//             memory instead of loading;
//   BT_ZRED   <Z_q> partial sums over a range of amplitudes, added to the
//             circuit's outputs with FP64 atomics (and, for sampling, each
//             chunk's probability sum);
//   BT_PREFIX exclusive prefix of a circuit's chunk sums;
//   BT_SAMPLE inverse-CDF sampling of the shots falling in a chunk range.
// Finished tasks bump their circuit's counter after a memory fence. Tasks
// are queued in level order per circuit, so a task waits only on tasks
// dequeued before it: every CTA can finish the task it runs, whatever the
// number of resident CTAs.
// C2 is the amplitude type: float2 (complex64, FP32 arithmetic) or double2
// (complex128, FP64 arithmetic). <Z> sums are FP64.
#include <cuda_runtime.h>

#include "k_block.cuh"
#include "k_stage.cuh"
#include "launch.hpp"

namespace kate {

namespace {

using namespace stage;


__device__ __forceinline__ unsigned long long now_ns() {
    unsigned long long v;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
    return v;
}

__device__ __forceinline__ double2 ldst(const double2* p) { return __ldcg(p); }
__device__ __forceinline__ double2 ldst(const float2* p) {
    const float2 v = __ldcg(p);
    return make_double2(v.x, v.y);
}

// Block-wide sums of per-thread values v[0..nb): result in red[NB * 8 + b].
template <int NB>
__device__ void block_sums(const double (&v)[NB], int nb, double* red) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int b = 0; b < NB; b++) {
        if (b >= nb) break;
        double x = v[b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) red[warp * NB + b] = x;
    }
    __syncthreads();
    if (t < nb) {
        double s = 0.0;
        for (int w = 0; w < NT / 32; w++) s += red[w * NB + t];
        red[NB * (NT / 32) + t] = s;
    }
    __syncthreads();
}

__device__ __forceinline__ ProgView view(const BatchProg& P, const unsigned char* blob) {
    ProgView v;
    v.m = P.m;
    v.ncb = P.ncb;
    v.nops = P.nstages >= 0 ? P.nops : 0;  // generic programs run from global memory
    v.nmats = P.nstages >= 0 ? P.nmats : 0;
    v.nstages = P.nstages >= 0 ? P.nstages : 0;
    v.sop0 = P.sop0;
    v.tphys = P.tphys;
    v.outsrc = P.outsrc;
    v.cphys = P.cphys;
    v.ops = reinterpret_cast<const SOp*>(blob + P.ops_off);
    v.mats = reinterpret_cast<const double(*)[2]>(blob + P.mats_off);
    v.stab = reinterpret_cast<const uint16_t(*)[44]>(blob + P.stab_off);
    return v;
}

// Dynamic shared memory of the batch kernel: two tiles, then the program
// tables or, for a tensor-core block task, the block region: the B operand
// images (1024-byte aligned), the BlockProg.
extern __shared__ __align__(16) unsigned char batch_smem_raw[];
constexpr uint32_t BLK_IMG = KATE_C64_MAX_BLOCKS * KATE_BLOCK_IMG_BYTES;
constexpr uint32_t BLK_PROG = (sizeof(BlockProg) + 15) & ~15u;
constexpr uint32_t BLK_REGION = 1024 + BLK_IMG + BLK_PROG;
static_assert(sizeof(BlockProg) % 8 == 0, "BlockProg is copied as 8-byte words");
// Per CTA, for the whole launch (complex64 batches with block programs):
// the groups' words and their mbarriers' phases, the TMEM columns.
__shared__ blk::GroupSync blk_group[2];
__shared__ uint64_t blk_mbar_img;
__shared__ uint32_t blk_tmem, blk_phase[2], blk_phase_img;

// Waits (time-bounded) until `need` tasks of the circuit have finished; every
// thread returns the same answer, after a barrier. *abort (shared) is set
// when the wait gave up.
__device__ __forceinline__ bool wait_dep(const int* done, int need, int* err, unsigned long long wait_ns, int* abort) {
    if (threadIdx.x == 0 && need > 0) {
        const unsigned long long t0 = now_ns();
        while (*((volatile const int*)done) < need) {
            if (now_ns() - t0 > wait_ns || *((volatile int*)err)) {
                *abort = 1;
                atomicExch(err, 1);
                break;
            }
            __nanosleep(256);
        }
        __threadfence();
    }
    __syncthreads();
    return *abort == 0;
}

// The task queue as a CTA sees it. A CTA takes its next task in the last step
// of the current one, by one thread and in two parts: the index (an atomic)
// and, once that is there, the descriptor's copy into shared memory, so that
// neither round trip is on the CTA's path (192 complex64 circuits of 10 to 20
// qubits: 5.5 ms; 6.1 ms with both between two tasks and the dependency waited
// for before a task's tables and operand images were in place). Not earlier: a
// task taken while the current one still waits or runs for long is kept from
// the other CTAs (5.6 ms when it was taken at the current one's start, and 48
// requests to the server took 11.6 ms in place of 8.7).
// Of the unfinished tasks the one taken first is always some CTA's current
// one (a CTA runs its tasks in the order it took them) and waits only on
// tasks taken before it: nothing can wait in a circle.
__shared__ __align__(16) BatchTask q_task[2];  // this task and the next
__shared__ int q_idx[2];
__shared__ const BatchTask* q_tasks;
__shared__ int *q_head, *q_err;
__shared__ int q_n;
constexpr uint32_t TAKER = NT - 32;  // the thread that takes the next task
static_assert(sizeof(BatchTask) == 32, "a descriptor is two 16-byte copies");

__device__ __forceinline__ int take_index() {
    // After a failed wait anywhere, every CTA stops at its next task.
    return *((volatile int*)q_err) ? q_n : atomicAdd(q_head, 1);
}
__device__ __forceinline__ void fetch_task(int i, uint32_t slot) {
    q_idx[slot] = i;
    if (i < q_n) {
        const uint32_t d = (uint32_t)__cvta_generic_to_shared(&q_task[slot]);
        const char* src = reinterpret_cast<const char*>(q_tasks + i);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 16u), "l"(src + 16) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// A complex64 tensor-core block pass over cosets [c0, c1) of one circuit
// (the BatchProg's BPROG_BLOCK program): the BlockProg and its operand
// images into shared memory, then per coset the staging tile (loaded, or
// the tile of |0...0> for a circuit's first pass), the blocks, the
// write-back. The two batch tile buffers are the staging tiles. Loads and
// stores go through L2 only (other SMs wrote the state earlier in this
// launch). The dependency is waited for once everything that does not depend
// on it is in place. Returns false when a wait gave up.
// G = 128: two groups of threads take alternate cosets, each with its buffer
// and TMEM columns, as the simulator's pass kernel does: for tasks of two
// cosets and more (17 qubits and up; 192 circuits of 10 to 20 qubits take 6.7
// ms in place of 7.3). G = 256: the whole CTA works on the task's one coset,
// whose latency is what a small circuit waits for.
template <int G>
__device__ __noinline__ bool block_task(float2* st, const BatchProg& BP, const unsigned char* blob, uint32_t slot,
                                        const int* done, unsigned long long wait_ns, int* abort) {
    const BatchTask& K = q_task[slot];
    const uint32_t t = threadIdx.x, grp = t / G;
    const uint32_t c0 = K.c0, c1 = K.c1;
    const bool first = K.first != 0;
    const uint32_t tmem = blk_tmem + grp * blk::TMEM_COLS, sync = blk::smem_u32(&blk_group[grp]);
    uint32_t phase = blk_phase[grp];  // every thread of the group keeps the same copy; its first one stores it back
    unsigned char* raw = batch_smem_raw + 2 * TS * sizeof(float2);
    const uint32_t rawa = blk::smem_u32(raw);
    const uint32_t bbase = (rawa + 1023u) & ~1023u;
    unsigned char* g = raw + (bbase - rawa);
    BlockProg& P = *reinterpret_cast<BlockProg*>(g + BLK_IMG);
    const unsigned char* src = blob + BP.ops_off;
    for (uint32_t i = t; i < sizeof(BlockProg) / 8; i += NT)
        reinterpret_cast<uint64_t*>(&P)[i] = __ldcg(reinterpret_cast<const unsigned long long*>(src) + i);
    __syncthreads();
    // The operand images by the bulk-copy engine (the previous task's
    // products, the last readers of this region, completed before it ended).
    uint32_t phase_img = blk_phase_img;
    const bool img_ok = blk::load_images(P.nblocks, [&](int b) { return src + P.bimg[b]; }, bbase,
                                         blk::smem_u32(&blk_mbar_img), phase_img);
    if (!img_ok) blk_group[0].gave_up = blk_group[1].gave_up = 1;  // before wait_dep's barrier
    blk::Pass<G> X;
    blk::setup(P, X);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (!wait_dep(done, K.need, q_err, wait_ns, abort)) {
        if (t == 0) blk_phase_img = phase_img;
        return false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float2* S = reinterpret_cast<float2*>(batch_smem_raw) + grp * TS;
    const uint32_t sb = blk::smem_u32(batch_smem_raw) + grp * blk::S_BYTES;
    bool ok = true;
    double unused = 0.0;
    for (uint32_t c = c0 + grp; c < c1; c += NT / G) {
        const uint64_t cb = blk::coset_base(P, c);
        const bool take = t == TAKER && c + NT / G >= c1;  // the last group's last coset
        int next = 0;
        if (take) next = take_index();
        if (first) {
            if (cb) {
                if (take) fetch_task(next, slot ^ 1u);
                blk::store_zero<true>(X, st, cb);
                continue;
            }
            blk::zero_tile<G>(S, true);
        } else {
            blk::load_tile<true>(st, cb, sb, X);
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
        }
        if (take) fetch_task(next, slot ^ 1u);
        blk::group_bar<G>();
        ok = blk::apply_blocks(P, X, S, bbase, tmem, sync, phase);
        if (!ok) break;
        blk::store_tile<true, false>(P, X, st, cb, S, unused);
        blk::group_bar<G>();
    }
    if (t % G == 0) blk_phase[grp] = phase;
    if (t == 0) blk_phase_img = phase_img;
    // Whether any group's wait gave up: every thread leaves with the same answer.
    return __syncthreads_and(ok) != 0;
}

// The register-staged program as a call of its own, so that its registers
// are allocated apart from the task loop's. The tile and tables are taken
// from the shared-memory symbol (shared-window addressing).
template <typename C2, bool SM>
__device__ __noinline__ void run_staged(int nops, uint64_t cbase, const DevOp* __restrict__ sops, int sop0,
                                        const double2* __restrict__ pool, uint32_t boff) {
    C2* tile = reinterpret_cast<C2*>(batch_smem_raw + boff);
    const TileTables<C2>& T = *reinterpret_cast<const TileTables<C2>*>(batch_smem_raw + 2 * TS * sizeof(C2));
    const uint32_t tb = (uint32_t)__cvta_generic_to_shared(tile);
    run_program<C2, SM>(T, nops, tb, tile, cbase, sops, sop0, pool, threadIdx.x);
}

// Runs program P (tables already in T) on the tile, for coset base cbase.
template <typename C2>
__device__ __forceinline__ void run_any(const TileTables<C2>& T, const BatchProg& P, const unsigned char* blob,
                                        uint32_t tb, C2* tile, uint64_t cbase, const DevOp* __restrict__ sops,
                                        const double2* __restrict__ pool, uint32_t t) {
    if (P.nstages >= 0) {
        const uint32_t boff = tb - (uint32_t)__cvta_generic_to_shared(batch_smem_raw);
        if (P.flags & BPROG_SMEM) run_staged<C2, true>(P.nops, cbase, sops, P.sop0, pool, boff);
        else run_staged<C2, false>(P.nops, cbase, sops, P.sop0, pool, boff);
    } else {
        const DevOp* gops = reinterpret_cast<const DevOp*>(blob + P.ops_off);
        for (int k = 0; k < P.nops; k++) {
            const DevOp op = gops[k];
            ops::apply_op<C2>(tile, TB, cbase, op, pool, (int)t, NT);
            __syncthreads();
        }
    }
}

// <Z_q> of a resident tile: output q reads tile bit zbit[q].
template <typename C2>
__device__ __noinline__ void small_z(const C2* tile, int nz, const uint8_t* zbit, double* red, double* out) {
    const uint32_t t = threadIdx.x;
    double z[KATE_BATCH_SMALL_MAX];
#pragma unroll
    for (int q = 0; q < KATE_BATCH_SMALL_MAX; q++) z[q] = 0.0;
    for (uint32_t i = t; i < (uint32_t)TS; i += NT) {
        const C2 a = tile[ops::tsw<C2>(i)];
        const double p = (double)a.x * a.x + (double)a.y * a.y;
#pragma unroll
        for (int q = 0; q < KATE_BATCH_SMALL_MAX; q++)
            if (q < nz) z[q] += ((i >> zbit[q]) & 1u) ? -p : p;
    }
    block_sums<KATE_BATCH_SMALL_MAX>(z, nz, red);
    if ((int)t < nz) out[t] = red[KATE_BATCH_SMALL_MAX * (NT / 32) + t];
}

// <Z_q> partial sums of an n-qubit state over 2^16-amplitude chunks
// [ch0, ch1), added to out[q] (q reads physical bit zbit[q]). Thread t takes
// amplitudes chunk * 2^16 + t + 256 k: physical bits 0..7 come from t, 8..15
// from k, the rest from the chunk. With psum, also stores each chunk's
// probability sum at psum[ch] (block-reduced in a fixed order).
template <typename C2>
__device__ __noinline__ void zred(const C2* st, int n, uint32_t ch0, uint32_t ch1, const uint8_t* zbit, double* red,
                                  double* out, double* psum) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    double z[KATE_BATCH_MAX_QUBITS];
#pragma unroll
    for (int q = 0; q < KATE_BATCH_MAX_QUBITS; q++) z[q] = 0.0;
    for (uint32_t ch = ch0; ch < ch1; ch++) {
        double tot = 0.0, kb[8];
#pragma unroll
        for (int b = 0; b < 8; b++) kb[b] = 0.0;
        const uint64_t x0 = (uint64_t)ch << 16;
        for (uint32_t k = 0; k < 256; k++) {
            const uint64_t x = x0 + t + ((uint64_t)k << 8);
            if (x >> n) break;
            const double2 a = ldst(st + x);
            const double p = a.x * a.x + a.y * a.y;
            tot += p;
#pragma unroll
            for (int b = 0; b < 8; b++) kb[b] += ((k >> b) & 1u) ? -p : p;
        }
#pragma unroll
        for (int b = 0; b < KATE_BATCH_MAX_QUBITS; b++) {
            if (b < 8) z[b] += ((t >> b) & 1u) ? -tot : tot;
            else if (b < 16) z[b] += kb[b - 8];
            else z[b] += ((ch >> (b - 16)) & 1u) ? -tot : tot;
        }
        if (psum) {
            double w = tot;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) w += __shfl_down_sync(0xffffffffu, w, o);
            if (lane == 0) red[warp] = w;
            __syncthreads();
            if (t == 0) {
                double sc = 0.0;
                for (int i = 0; i < NT / 32; i++) sc += red[i];
                psum[ch] = sc;
            }
            __syncthreads();
        }
    }
    block_sums<KATE_BATCH_MAX_QUBITS>(z, n, red);
    if ((int)t < n) atomicAdd(out + t, red[KATE_BATCH_MAX_QUBITS * (NT / 32) + zbit[t]]);
}

// Block-wide exclusive scan of one double per thread (fixed order); also
// returns the block total.
__device__ double block_exscan(double v, double* red, double* total) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    double x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) red[warp] = x;
    __syncthreads();
    if (t == 0) {
        double s = 0.0;
        for (int i = 0; i < NT / 32; i++) {
            const double w = red[i];
            red[i] = s;
            s += w;
        }
        red[NT / 32] = s;
    }
    __syncthreads();
    const double r = red[warp] + x - v;
    *total = red[NT / 32];
    __syncthreads();
    return r;
}

// Exclusive prefix of nch chunk sums psum[0..nch) into psum[nch..2 nch),
// the total into psum[2 nch].
__device__ __noinline__ void chunk_prefix(double* psum, uint32_t nch, double* red) {
    const uint32_t t = threadIdx.x;
    const uint32_t per = (nch + NT - 1) / NT, b0 = t * per, b1 = min(nch, b0 + per);
    double loc = 0.0;
    for (uint32_t c = b0; c < b1; c++) loc += psum[c];
    double total;
    double run = block_exscan(loc, red, &total);
    for (uint32_t c = b0; c < b1; c++) {
        psum[nch + c] = run;
        run += psum[c];
    }
    if (t == 0) psum[2 * nch] = total;
}

// Sum of v over the warp's lanes, the same on every lane (a fixed tree).
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Inverse-CDF sampling over chunks [ch0, ch1): shot s (uniforms u ascending)
// targets x = u * total; it falls in chunk ch when pre[ch] <= x < pre[ch] +
// sum[ch] (targets at or past the total go to the last chunk). Inside a
// chunk, the sums of its runs of 256 amplitudes (a warp each) and their
// prefix come first; then every warp takes shots of its own: the prefix names
// the run, whose 256 amplitudes the warp reads at once and walks 32 at a
// time. With a thread owning 256 amplitudes and walking them one load after
// another, 1024 shots of a 16-qubit state took milliseconds, most of a served
// request's time. The tile buffers hold the prefix.
template <typename C2>
__device__ __noinline__ void sample_chunks(const C2* st, int n, uint32_t ch0, uint32_t ch1, const double* psum,
                                           const double* unif, int shots, uint64_t* out, double* red, int* srange) {
    constexpr uint32_t RUN = 256, FULL = 0xffffffffu;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    double* pre = reinterpret_cast<double*>(batch_smem_raw);
    const uint64_t dim = 1ull << n;
    const uint32_t nch = (uint32_t)(dim >> 16 ? dim >> 16 : 1);
    const double total = psum[2 * nch];
    for (uint32_t ch = ch0; ch < ch1; ch++) {
        const double lo_v = psum[nch + ch];
        const double hi_v = lo_v + psum[ch];
        const bool last = ch + 1 == nch;
        if (t == 0) {
            int lo = 0, hi = shots;  // first s with u_s * total >= lo_v
            while (lo < hi) {
                const int m = (lo + hi) >> 1;
                if (unif[m] * total >= lo_v) hi = m;
                else lo = m + 1;
            }
            int e = lo, e1 = shots;  // first s with u_s * total >= hi_v
            if (!last)
                while (e < e1) {
                    const int m = (e + e1) >> 1;
                    if (unif[m] * total >= hi_v) e1 = m;
                    else e = m + 1;
                }
            srange[0] = lo;
            srange[1] = last ? shots : e;
        }
        __syncthreads();
        const int s0 = srange[0], s1 = srange[1];
        __syncthreads();
        if (s0 >= s1) continue;
        const uint64_t x0 = (uint64_t)ch << 16;
        const uint32_t len = (uint32_t)(dim - x0 < (1ull << 16) ? dim - x0 : (1ull << 16));
        const uint32_t nrun = len / RUN;  // states of 12 qubits and more: 16 to 256
        const C2* p = st + x0;
        auto probs = [&](uint32_t run, double (&v)[8]) {
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) {
                const double2 a = ldst(p + run * RUN + 32 * k + lane);
                v[k] = a.x * a.x + a.y * a.y;
            }
        };
        for (uint32_t r = warp; r < nrun; r += NT / 32) {
            double v[8];
            probs(r, v);
            const double w = warp_sum(((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
            if (lane == 0) pre[r] = w;
        }
        __syncthreads();
        double tot;
        const double base = block_exscan(t < nrun ? pre[t] : 0.0, red, &tot);
        if (t < nrun) pre[t] = base;
        __syncthreads();
        for (int s = s0 + (int)warp; s < s1; s += NT / 32) {
            const double y = unif[s] * total - lo_v;
            // Last run whose prefix is at most y: eight runs per lane, then
            // the runs of that lane.
            const uint32_t hi8 = __ballot_sync(FULL, 8 * lane < nrun && pre[8 * lane] <= y);
            const uint32_t g = hi8 ? 8u * (31u - (uint32_t)__clz((int)hi8)) : 0u;
            const uint32_t lo8 = __ballot_sync(FULL, lane < 8 && g + lane < nrun && pre[g + lane] <= y);
            uint32_t r = g + (lo8 ? 31u - (uint32_t)__clz((int)lo8) : 0u);
            uint32_t pick = 0;
            for (bool found = false; !found;) {
                double v[8], acc = pre[r];
                uint32_t lastnz = 0;
                bool any = false;
                probs(r, v);
                double w[8];
#pragma unroll
                for (int k = 0; k < 8; k++) w[k] = warp_sum(v[k]);
#pragma unroll
                for (uint32_t k = 0; k < 8; k++) {
                    if (found) continue;
                    const uint32_t nz = __ballot_sync(FULL, v[k] > 0.0);
                    if (acc + w[k] > y && nz) {
                        double inc = v[k];
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const double u = __shfl_up_sync(FULL, inc, o);
                            if (lane >= (uint32_t)o) inc += u;
                        }
                        // The tree's sum may pass y by a rounding that the
                        // scan does not: then the last nonzero amplitude.
                        const uint32_t hit = __ballot_sync(FULL, v[k] > 0.0 && acc + inc > y);
                        pick = r * RUN + 32 * k + (hit ? (uint32_t)__ffs((int)hit) - 1u : 31u - (uint32_t)__clz((int)nz));
                        found = true;
                    }
                    if (nz) lastnz = r * RUN + 32 * k + 31u - (uint32_t)__clz((int)nz), any = true;
                    acc += w[k];
                }
                // y at or past the run's end (rounding between the sums): the
                // last amplitude of nonzero probability at or before it.
                if (!found && any) pick = lastnz;
                if (found || any || r == 0) break;
                r--;
            }
            if (lane == 0) out[s] = x0 + pick;
        }
        __syncthreads();
    }
}

template <typename C2>
__device__ __forceinline__ void init_basis0(C2* tile, bool one, uint32_t t) {
#pragma unroll 4
    for (uint32_t i = t; i < (uint32_t)TS; i += NT) tile[i] = Amp<C2>::mk(0, 0);
    if (one && t == 0) tile[0] = Amp<C2>::mk(1, 0);  // element 0 sits at offset 0
}

// complex64: two CTAs per SM (128 registers); complex128 programs need more.
// TB (complex64 only): the batch has tensor-core block programs; the kernel
// then holds TMEM and the block region of shared memory. Batches without
// them use the kernel compiled without that code (less shared memory, more
// L1, no spills from it in the task loop).
template <typename C2, bool TB>
__global__ void __launch_bounds__(NT, sizeof(C2) == 8 ? 2 : 1)
    k_batch(C2* __restrict__ arena, const BatchTask* __restrict__ tasks, int ntasks, const BatchCirc* __restrict__ circs,
            const BatchProg* __restrict__ progs, const unsigned char* __restrict__ blob, const DevOp* __restrict__ sops,
            const double2* __restrict__ pool, int* __restrict__ head, int* __restrict__ done,
            double* __restrict__ zout, int* __restrict__ err, double* __restrict__ psum,
            const double* __restrict__ unif, uint64_t* __restrict__ sout, unsigned long long wait_ns) {
    static_assert(!TB || sizeof(C2) == 8, "tensor-core block tasks are complex64");
    // Two tile buffers (a pass task prefetches its next coset into the
    // other one), then the program tables.
    C2* tile = reinterpret_cast<C2*>(batch_smem_raw);
    TileTables<C2>& T = *reinterpret_cast<TileTables<C2>*>(batch_smem_raw + 2 * TS * sizeof(C2));
    __shared__ int s_abort;
    __shared__ uint8_t s_zbit[40];
    __shared__ int s_range[2];
    __shared__ double red[KATE_BATCH_MAX_QUBITS * (NT / 32) + KATE_BATCH_MAX_QUBITS];
    const uint32_t t = threadIdx.x;
    const uint32_t tb = (uint32_t)__cvta_generic_to_shared(tile);
    // Tensor-core block tasks (complex64 only): the CTA's TMEM columns and
    // the products' mbarrier, for the whole launch.
    if constexpr (TB) {
        {
            if (t == 0) {
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(blk::smem_u32(&blk_group[0].mbar)) : "memory");
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(blk::smem_u32(&blk_group[1].mbar)) : "memory");
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(blk::smem_u32(&blk_mbar_img)) : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                blk_group[0].gave_up = blk_group[1].gave_up = 0;
                blk_phase[0] = blk_phase[1] = 0;
                blk_phase_img = 0;
            }
            blk::tmem_alloc(&blk_tmem, 2 * blk::TMEM_COLS);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
    }
    if (t == TAKER) {
        s_abort = 0;
        q_tasks = tasks;
        q_head = head;
        q_err = err;
        q_n = ntasks;
        fetch_task(take_index(), 0);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    for (uint32_t now = 0;; now ^= 1u) {
        if (q_idx[now] >= q_n) break;
        const BatchTask& K = q_task[now];
        if (t == TAKER) q_idx[now ^ 1u] = -1;  // not taken yet
        auto ready = [&] { return wait_dep(done + K.circ, K.need, err, wait_ns, &s_abort); };
        const bool pass = K.kind == BT_PASS;
        bool block_pass = false;
        if constexpr (TB) block_pass = pass && (progs[K.prog].flags & BPROG_BLOCK);
        if (!pass) {
            if (t < 40) s_zbit[t] = circs[K.circ].zbit[t];
            if (!ready()) break;
        }
        if (block_pass) {
            if constexpr (TB) {
                float2* st = arena + circs[K.circ].off;
                const int* dn = done + K.circ;
                if (!(K.c1 - K.c0 >= 2 ? block_task<128>(st, progs[K.prog], blob, now, dn, wait_ns, &s_abort)
                                       : block_task<NT>(st, progs[K.prog], blob, now, dn, wait_ns, &s_abort))) {
                    if (t == 0) atomicExch(err, 1);
                    break;
                }
            }
        } else if (K.kind == BT_SMALL || K.kind == BT_PASS) {
            // SMALL: step s runs program prog + s on the resident tile.
            // PASS: step s runs program prog on coset c0 + s.
            const bool small = K.kind == BT_SMALL;
            const int nsteps = small ? K.nprog : (int)(K.c1 - K.c0);
            C2* st = arena + circs[K.circ].off;
            if (small) {
                init_basis0(tile, true, t);
            } else {
                const ProgView v = view(progs[K.prog], blob);
                setup_program(T, v, t);
                setup_io(T, v, t);
            }
            // The tables are in place: now the dependency.
            if (pass && !ready()) break;
            const bool pre = !small && !K.first;  // pass task that loads: double-buffered
            if (pre) load_async(T, st, K.c0, tb, t);
            for (int s = 0; s < nsteps; s++) {
                const BatchProg& P = progs[small ? K.prog + s : K.prog];
                const uint32_t c = K.c0 + (uint32_t)s;
                const uint32_t cur = pre ? (uint32_t)(s & 1) : 0u;
                const uint32_t tbc = tb + cur * (uint32_t)(TS * sizeof(C2));
                C2* tilec = tile + cur * TS;
                uint64_t cbase = 0;
                __syncthreads();
                if (small) {
                    setup_program(T, view(P, blob), t);
                } else {
                    cbase = coset_base(T, c);
                    if (K.first) {
                        init_basis0(tilec, cbase == 0, t);
                    } else if (s + 1 < nsteps) {
                        load_async(T, st, c + 1, tb + (cur ^ 1u) * (uint32_t)(TS * sizeof(C2)), t);
                        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
                    } else {
                        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                    }
                }
                if (t == TAKER && s + 1 == nsteps) fetch_task(take_index(), now ^ 1u);
                __syncthreads();
                // A first pass's other cosets are zero in and out.
                if (!K.first || cbase == 0) run_any(T, P, blob, tbc, tilec, cbase, sops, pool, t);
                if (!small) {
                    __syncthreads();
                    store_tile<C2, true>(T, st, c, tbc, t);
                }
            }
            __syncthreads();
            if (small) small_z(tile, circs[K.circ].n, s_zbit, red, zout + circs[K.circ].zoff);
        } else {
            const BatchCirc& C = circs[K.circ];
            const int nz = C.n;
            const uint32_t nch = (uint32_t)(((1ull << nz) >> 16) ? ((1ull << nz) >> 16) : 1);
            if (K.kind == BT_ZRED)
                zred(arena + C.off, nz, K.c0, K.c1, s_zbit, red, zout + C.zoff, C.poff >= 0 ? psum + C.poff : nullptr);
            else if (K.kind == BT_PREFIX)
                chunk_prefix(psum + C.poff, nch, red);
            else if (K.kind == BT_SAMPLE)
                sample_chunks(arena + C.off, nz, K.c0, K.c1, psum + C.poff, unif + C.uoff, C.shots, sout + C.soff,
                              red, s_range);
        }
        if (t == TAKER) {
            if (q_idx[now ^ 1u] < 0) fetch_task(take_index(), now ^ 1u);  // a task without steps
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        int* const finished = done + K.circ;  // read before the barrier: K's place is the task's after the next
        __syncthreads();
        if (t == 0) {
            __threadfence();
            atomicAdd(finished, 1);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if constexpr (TB) blk::tmem_free(blk_tmem, 2 * blk::TMEM_COLS);
}

template <typename C2, bool TB>
constexpr size_t batch_smem() {
    // Two tiles, then the tables or (TB) the tensor-core block region,
    // whichever is larger.
    return (size_t)2 * TS * sizeof(C2) +
           (TB && BLK_REGION > sizeof(TileTables<C2>) ? BLK_REGION : sizeof(TileTables<C2>));
}

}  // namespace

int batch_grid(int device, int prec, bool tensor_blocks) {
    static int cached[64][3] = {{0}};
    if (device < 0 || device >= 64) device = 0;
    const int pi = prec == 1 ? (tensor_blocks ? 2 : 1) : 0;
    if (!cached[device][pi]) {
        int sms = 148, occ = 1;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (pi == 2) {
            // About 100 KiB of shared memory per CTA: two CTAs per SM need
            // the largest carveout. The occupancy calculator reports one CTA
            // per SM for this kernel (it holds tcgen05 code), although two fit
            // and run together (measured: 570 against 932 ms per launch of
            // the batching workload with tensor-core block tasks).
            // __launch_bounds__ gives the registers for two; shared memory
            // decides.
            cudaFuncSetAttribute(k_batch<float2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)batch_smem<float2, true>());
            cudaFuncSetAttribute(k_batch<float2, true>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
            cudaFuncAttributes fa{};
            cudaFuncGetAttributes(&fa, k_batch<float2, true>);
            int smem_sm = 0, reserved = 0;
            cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device);
            cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device);
            occ = smem_sm / (int)(batch_smem<float2, true>() + fa.sharedSizeBytes + reserved);
            if (occ > 2) occ = 2;
        } else if (pi == 1) {
            cudaFuncSetAttribute(k_batch<float2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)batch_smem<float2, false>());
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch<float2, false>, NT, batch_smem<float2, false>());
        } else {
            cudaFuncSetAttribute(k_batch<double2, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)batch_smem<double2, false>());
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_batch<double2, false>, NT,
                                                          batch_smem<double2, false>());
        }
        if (occ < 1) occ = 1;
        cached[device][pi] = sms * occ;
    }
    return cached[device][pi];
}

cudaError_t launch_batch(void* arena, int prec, const BatchTask* tasks, int ntasks, const BatchCirc* circs,
                         const BatchProg* progs, const void* blob, const DevOp* sops, const void* pool, int* head,
                         int* done, double* zout, int* err, int grid, cudaStream_t s, double* psum,
                         const double* unif, uint64_t* sout, unsigned long long wait_ns, int tensor_blocks) {
    const unsigned char* b = (const unsigned char*)blob;
    const double2* pl = (const double2*)pool;
    if (prec == 1 && tensor_blocks)
        k_batch<float2, true><<<grid, NT, batch_smem<float2, true>(), s>>>(
            (float2*)arena, tasks, ntasks, circs, progs, b, sops, pl, head, done, zout, err, psum, unif, sout, wait_ns);
    else if (prec == 1)
        k_batch<float2, false><<<grid, NT, batch_smem<float2, false>(), s>>>(
            (float2*)arena, tasks, ntasks, circs, progs, b, sops, pl, head, done, zout, err, psum, unif, sout, wait_ns);
    else
        k_batch<double2, false><<<grid, NT, batch_smem<double2, false>(), s>>>(
            (double2*)arena, tasks, ntasks, circs, progs, b, sops, pl, head, done, zout, err, psum, unif, sout, wait_ns);
    return cudaGetLastError();
}

}  // namespace kate
