// Inverse-CDF sampling of the computational basis on the device, for the
// simulator (kate_sim_sample): nothing but the samples crosses PCIe.
//
// Shot k has the uniform u_k = (the k-th splitmix64 output of the seed >> 11)
// * 2^-53 and takes the first amplitude index i whose cumulative probability
// exceeds y = u_k * total, i.e. cdf(i - 1) <= y < cdf(i); amplitudes of
// probability 0 are never chosen. The cumulative sums are FP64 in a fixed
// order:
//   k_chunk_sums  sum of |a|^2 over each chunk of 2^12 amplitudes, a warp per
//                 chunk (a fixed order per lane, then a fixed tree);
//   k_chunk_scan  exclusive prefix of the chunk sums and their total (one
//                 CTA, a fixed order);
//   k_resolve     one warp per shot: a 32-way search of the prefix finds the
//                 chunk, whose 2^12 amplitudes the warp walks 512 at a time.
// Only the first of them reads the state; it is bound by HBM (8 loads of
// 512 bytes in flight per warp). Chunks of 2^12 keep a shot's walk to 64 KiB
// of contiguous reads and the prefix at 1/2048 of the state's size; with
// chunks of 2^16, in which 256 threads walked runs of 256 amplitudes each
// (4 KiB apart between lanes), finding 1024 shots at 26 qubits took longer
// (212 us) than reading the state.
// Indices are physical (the state's bit layout); the kernel maps them to the
// reference's qubit labels. This is the device counterpart of the
// reference's host-side measurement (HIPcode/simulator.hpp:483-543 copies
// partial sums back); Kate itself has no sampling.
#include "k_common.cuh"
#include "launch.hpp"

namespace kate {

namespace {

constexpr int NTS = 256;
constexpr int CHUNK_BITS = 12;
constexpr uint32_t FULL = 0xffffffffu;

__device__ __forceinline__ double prob(double2 a) { return a.x * a.x + a.y * a.y; }
__device__ __forceinline__ double prob(float2 a) { return (double)a.x * a.x + (double)a.y * a.y; }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}

template <typename C2>
__global__ void __launch_bounds__(NTS) k_chunk_sums(const C2* __restrict__ st, int n, uint32_t nch,
                                                    double* __restrict__ sums) {
    const uint32_t ch = blockIdx.x * (NTS / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (ch >= nch) return;
    const uint32_t len = 1u << (n < CHUNK_BITS ? n : CHUNK_BITS);
    const C2* p = st + ((uint64_t)ch << CHUNK_BITS);
    double acc = 0.0;
    if (len >= 256) {
        for (uint32_t x = lane; x < len; x += 256) {
            C2 a[8];
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) a[k] = __ldcs(p + x + 32 * k);
#pragma unroll
            for (uint32_t k = 0; k < 8; k++) acc += prob(a[k]);
        }
    } else {
        for (uint32_t x = lane; x < len; x += 32) acc += prob(p[x]);
    }
    acc = warp_sum(acc);
    if (lane == 0) sums[ch] = acc;
}

// pre[c] = sum of sums[0..c), pre[nch] = total: one CTA, 4096 sums at a time.
__global__ void __launch_bounds__(1024) k_chunk_scan(const double* __restrict__ sums, uint32_t nch,
                                                     double* __restrict__ pre) {
    __shared__ double wsum[32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    double run = 0.0;
    for (uint32_t c0 = 0; c0 < nch; c0 += 4096) {
        double v[4], loc = 0.0;
        const uint32_t c = c0 + 4 * t;
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            v[k] = c + k < nch ? sums[c + k] : 0.0;
            loc += v[k];
        }
        double inc = loc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(FULL, inc, o);
            if (lane >= (uint32_t)o) inc += y;
        }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        double base = run;
        double tot = 0.0;
        for (uint32_t w = 0; w < 32; w++) {
            if (w < warp) base += wsum[w];
            tot += wsum[w];
        }
        __syncthreads();
        double x = base + (inc - loc);
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            if (c + k < nch) pre[c + k] = x;
            x += v[k];
        }
        run += tot;
    }
    if (t == 0) pre[nch] = run;
}

// Chunk of target y: the first with pre[ch + 1] > y (the last chunk if
// none), by a 32-way search. Every lane returns the same value.
__device__ __forceinline__ uint32_t find_chunk(const double* __restrict__ pre, uint32_t nch, double y) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t lo = 0, hi = nch;  // the answer is in [lo, hi); hi = nch: none yet
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        // Lane i asks whether the answer is at most the end of its part.
        const uint32_t e = min(lo + (lane + 1) * step, hi) - 1;
        const uint32_t hit = __ballot_sync(FULL, e + 1 == hi || pre[e + 1] > y);
        const uint32_t f = (uint32_t)__ffs((int)hit) - 1u;
        const uint32_t nhi = min(lo + (f + 1) * step, hi);
        lo = lo + f * step;
        hi = nhi;
    }
    return lo;
}

template <typename C2>
__global__ void __launch_bounds__(NTS) k_resolve(const C2* __restrict__ st, int n, const double* __restrict__ sums,
                                                 const double* __restrict__ pre, uint32_t nch, uint64_t seed,
                                                 int shots, const SampleLabels L, uint64_t* __restrict__ out) {
    const int s = (int)(blockIdx.x * (NTS / 32) + (threadIdx.x >> 5));
    const uint32_t lane = threadIdx.x & 31u;
    if (s >= shots) return;
    uint64_t z = seed + (uint64_t)(s + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const double u = (double)(z >> 11) * (1.0 / 9007199254740992.0);
    const double y = u * pre[nch];
    uint32_t ch = find_chunk(pre, nch, y);
    // Rounding can name a chunk without any probability: the nearest one
    // before it that has some, else the nearest after it.
    if (sums[ch] == 0.0) {
        uint32_t c = ch;
        while (c > 0 && sums[c] == 0.0) c--;
        if (sums[c] == 0.0)
            for (c = ch; c + 1 < nch && sums[c] == 0.0;) c++;
        ch = c;
    }
    const double yl = y - pre[ch];
    const uint32_t len = 1u << (n < CHUNK_BITS ? n : CHUNK_BITS);
    const uint64_t x0 = (uint64_t)ch << CHUNK_BITS;
    const C2* p = st + x0;
    // 512 amplitudes at a time: the sums of 16 runs of 32 first, then the
    // run that reaches the target, amplitude by amplitude.
    double run = 0.0;
    uint32_t pick = 0, lastnz = 0;
    bool found = false;
    for (uint32_t b = 0; b < len && !found; b += 512) {
        double v[16], w[16];
#pragma unroll
        for (uint32_t k = 0; k < 16; k++) {
            const uint32_t x = b + 32 * k + lane;
            v[k] = x < len ? prob(p[x]) : 0.0;
        }
#pragma unroll
        for (uint32_t k = 0; k < 16; k++) w[k] = warp_sum(v[k]);
#pragma unroll
        for (uint32_t k = 0; k < 16; k++) {
            if (found) continue;
            const uint32_t nz = __ballot_sync(FULL, v[k] > 0.0);
            if (run + w[k] > yl) {
                double inc = v[k];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double t = __shfl_up_sync(FULL, inc, o);
                    if (lane >= (uint32_t)o) inc += t;
                }
                // The run's tree sum may pass the target by a rounding that
                // its scan does not: then its last nonzero amplitude.
                const uint32_t hit = __ballot_sync(FULL, v[k] > 0.0 && run + inc > yl);
                if (hit || nz) {
                    pick = b + 32 * k + (hit ? (uint32_t)__ffs((int)hit) - 1u : 31u - (uint32_t)__clz((int)nz));
                    found = true;
                }
            }
            if (nz) lastnz = b + 32 * k + 31u - (uint32_t)__clz((int)nz);
            run += w[k];
        }
    }
    if (lane == 0) {
        const uint64_t i = x0 + (found ? pick : lastnz);
        uint64_t lab = 0;
        for (int q = 0; q < n; q++) lab |= ((i >> L.phys[q]) & 1ull) << q;
        out[s] = lab;
    }
}

uint32_t chunk_count(int n) { return n > CHUNK_BITS ? 1u << (n - CHUNK_BITS) : 1u; }

template <typename C2>
cudaError_t sample(const C2* st, int n, uint64_t seed, int shots, const SampleLabels& L, double* scratch,
                   uint64_t* out, cudaStream_t s) {
    const uint32_t nch = chunk_count(n);
    double* sums = scratch;
    double* pre = scratch + nch;
    k_chunk_sums<C2><<<(nch + NTS / 32 - 1) / (NTS / 32), NTS, 0, s>>>(st, n, nch, sums);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_chunk_scan<<<1, 1024, 0, s>>>(sums, nch, pre);
    e = cudaGetLastError();
    if (e != cudaSuccess || shots == 0) return e;
    const unsigned grid = ((unsigned)shots + NTS / 32 - 1) / (NTS / 32);
    k_resolve<C2><<<grid, NTS, 0, s>>>(st, n, sums, pre, nch, seed, shots, L, out);
    return cudaGetLastError();
}

}  // namespace

size_t sample_scratch_doubles(int n) { return 2 * (size_t)chunk_count(n) + 1; }

cudaError_t launch_sample(const void* st, int prec, int n, uint64_t seed, int shots, const SampleLabels& L,
                          double* scratch, uint64_t* out, cudaStream_t s) {
    if (n < 1 || shots < 0) return cudaErrorInvalidValue;
    return prec == 1 ? sample((const float2*)st, n, seed, shots, L, scratch, out, s)
                     : sample((const double2*)st, n, seed, shots, L, scratch, out, s);
}

}  // namespace kate
