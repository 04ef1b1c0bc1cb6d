// Measurement reductions over the state, FP64 accumulation.
//
// k_bitsums computes, for every bit b of the amplitude index, the sum over
// amplitudes whose bit b is 0 and the sum over those whose bit b is 1 (kind
// 0: the amplitudes themselves, the reference's proba_state input,
// HIPcode/simulator.hpp:40-61 and 483-543; kind 1: |a|^2, for <Z_q>), in one
// read pass; k_bitsums_finish adds the CTAs' partials on the device, so the
// host receives 2n + 1 sums. Amplitude x is split as
//   x = ((r << g) | cta) << 12 | (12 local bits)
// and every 16-byte load of a thread covers one complex128 amplitude (local
// bits 0..7 = thread, 8..11 = load) or two complex64 ones (bit 0 = within
// the load, 1..8 = thread, 9..11 = load): 16 amplitudes per thread and
// round. Bits held inside a thread are summed by a tree over the 16 values
// (2.75 additions per amplitude where one running sum per bit takes 5),
// thread bits once per CTA, round bits from per-round warp totals kept in
// shared memory, CTA bits by the finishing kernel. Every order is fixed by
// the shape, so results repeat.
//
// Bound by HBM: the state is read once. Loads are issued eight at a time
// into registers before they are added; with one running sum per bit and
// per round bit in registers the amplitude form held 128 registers and read
// 1 GiB in 416 us (2.6 TB/s).
#include "k_common.cuh"
#include "k_norm.cuh"
#include "launch.hpp"

namespace kate {

namespace {

constexpr int NT = 256;
constexpr int MAXR = 8;

template <typename V>
struct Acc;
template <>
struct Acc<double2> {
    __device__ static double2 zero() { return make_double2(0.0, 0.0); }
    __device__ static double2 val(double2 a) { return a; }
    __device__ static double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
    __device__ static double2 shfl(double2 v, int o) {
        return make_double2(__shfl_down_sync(0xffffffffu, v.x, o), __shfl_down_sync(0xffffffffu, v.y, o));
    }
};
template <>
struct Acc<double> {
    __device__ static double zero() { return 0.0; }
    __device__ static double val(double2 a) { return a.x * a.x + a.y * a.y; }
    __device__ static double add(double a, double b) { return a + b; }
    __device__ static double shfl(double v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }
};

__device__ __forceinline__ double2 ld_amp(const double2* p) { return *p; }
__device__ __forceinline__ double2 ld_amp(const float2* p) {
    const float2 v = *p;
    return make_double2(v.x, v.y);
}

// Half a thread's round (8 amplitudes, in-thread bits 0..2 of their index)
// at element x0 of the round: values of element x >= lim are zero. With
// SCALE the amplitudes are first multiplied by f (one rounding) and stored.
template <typename V, bool SCALE>
__device__ __forceinline__ void load_half(const double2* st, uint32_t t, uint32_t h, uint32_t lim, double, V (&v)[8]) {
    static_assert(!SCALE, "complex128 states are not rescaled");
    double2 a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const uint32_t x = t + ((h * 8u + (uint32_t)k) << 8);
        a[k] = x < lim ? __ldcs(st + x) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = Acc<V>::val(a[k]);
}
template <typename V, bool SCALE>
__device__ __forceinline__ void load_half(float2* st, uint32_t t, uint32_t h, uint32_t lim, double f, V (&v)[8]) {
    float4 a[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint32_t x = 2u * t + ((h * 4u + (uint32_t)k) << 9);
        a[k] = x < lim ? __ldcs(reinterpret_cast<const float4*>(st + x)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if constexpr (SCALE) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            a[k].x = (float)((double)a[k].x * f);
            a[k].y = (float)((double)a[k].y * f);
            a[k].z = (float)((double)a[k].z * f);
            a[k].w = (float)((double)a[k].w * f);
            const uint32_t x = 2u * t + ((h * 4u + (uint32_t)k) << 9);
            if (x < lim) __stcs(reinterpret_cast<float4*>(st + x), a[k]);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        v[2 * k] = Acc<V>::val(make_double2(a[k].x, a[k].y));
        v[2 * k + 1] = Acc<V>::val(make_double2(a[k].z, a[k].w));
    }
}

// Partials of CTA c, slot i: part[i * gridDim.x + c]. Slot 0 is the total,
// 1 + 2b / 2 + 2b the sums with bit b 0 / 1, for the local bits b = 0..11,
// then the round bits 12..12+nr-1 (in slot order, not index order). With
// one CTA and no rounds that is k_bitsums_finish's output already.
// SCALE (complex64): every amplitude is also multiplied by scale[1] and
// written back (the renormalisation, whose pass over the state this saves).
template <typename V, typename S, bool SCALE = false>
__global__ void __launch_bounds__(NT, 3) k_bitsums(S* __restrict__ st, int n, int g, int nr, V* __restrict__ part,
                                                   const double* __restrict__ scale, const int* __restrict__ err,
                                                   int* __restrict__ err_out) {
    using A = Acc<V>;
    let_next_start();
    wait_for_previous();
    if (err_out && blockIdx.x == 0 && threadIdx.x == 0) *err_out = *err;
    constexpr bool F = sizeof(S) == 8;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t lim = 1u << (n < 12 ? n : 12);
    const uint32_t rounds = 1u << nr;
    extern __shared__ __align__(16) unsigned char bs_raw[];
    V* rtot = reinterpret_cast<V*>(bs_raw);  // [rounds][8] warp totals (nr > 0)
    __shared__ V st_t[NT];
    __shared__ V sw[NT / 32][8];
    double f = 1.0;
    if constexpr (SCALE) f = scale[1];
    // H[2i] / H[2i + 1]: in-thread bit i is 0 / 1.
    V H[8];
#pragma unroll
    for (int i = 0; i < 8; i++) H[i] = A::zero();
    for (uint32_t r = 0; r < rounds; r++) {
        S* base = st + ((((uint64_t)r << g) | blockIdx.x) << 12);
        V tr = A::zero();
#pragma unroll
        for (uint32_t h = 0; h < 2; h++) {
            V v[8], p[4];
            load_half<V, SCALE>(base, t, h, lim, f, v);
#pragma unroll
            for (int k = 0; k < 4; k++) p[k] = A::add(v[2 * k], v[2 * k + 1]);
            H[0] = A::add(H[0], A::add(A::add(v[0], v[2]), A::add(v[4], v[6])));
            H[1] = A::add(H[1], A::add(A::add(v[1], v[3]), A::add(v[5], v[7])));
            const V q0 = A::add(p[0], p[1]), q1 = A::add(p[2], p[3]);
            H[2] = A::add(H[2], A::add(p[0], p[2]));
            H[3] = A::add(H[3], A::add(p[1], p[3]));
            H[4] = A::add(H[4], q0);
            H[5] = A::add(H[5], q1);
            const V s = A::add(q0, q1);
            H[6 + h] = A::add(H[6 + h], s);
            tr = A::add(tr, s);
        }
        if (nr) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tr = A::add(tr, A::shfl(tr, o));
            if (lane == 0) rtot[r * (NT / 32) + warp] = tr;
        }
    }
    st_t[t] = A::add(H[6], H[7]);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        V w = H[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) w = A::add(w, A::shfl(w, o));
        if (lane == 0) sw[warp][i] = w;
    }
    __syncthreads();
    const uint32_t ncta = gridDim.x, c = blockIdx.x;
    {
        // Thread bits: 16 threads per (bit, value), 8 of the 128 threads'
        // totals each.
        const uint32_t b = t >> 5, one = (t >> 4) & 1u, i = t & 15u;
        V s = A::zero();
#pragma unroll
        for (uint32_t k = 0; k < 8; k++) s = A::add(s, st_t[ins0(i + 16u * k, (int)b) | (one << b)]);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) s = A::add(s, A::shfl(s, o));
        const uint32_t bit = F ? b + 1u : b;
        if (i == 0) part[(size_t)(1 + 2 * bit + one) * ncta + c] = s;
        // The total: the two halves of thread bit 0.
        const V other = A::shfl(s, 16);
        if (t == 0) part[c] = A::add(s, other);
    }
    if (t < 8) {
        V s = A::zero();
#pragma unroll
        for (int w = 0; w < NT / 32; w++) s = A::add(s, sw[w][t]);
        const uint32_t i = t >> 1, bit = F ? (i == 0 ? 0u : 8u + i) : 8u + i;
        part[(size_t)(1 + 2 * bit + (t & 1u)) * ncta + c] = s;
    }
    if (t >= 32 && t < 32 + 2u * (uint32_t)nr) {
        const uint32_t i = (t - 32u) >> 1, one = t & 1u;
        V s = A::zero();
        for (uint32_t r = 0; r < rounds; r++)
            if (((r >> i) & 1u) == one)
                for (int w = 0; w < NT / 32; w++) s = A::add(s, rtot[r * (NT / 32) + w]);
        part[(size_t)(1 + 2 * (12 + i) + one) * ncta + c] = s;
    }
}

// One CTA per output, from output `first`: out[0] = total, out[1 + 2b + v] =
// sum over the amplitudes whose index bit b is v. Partials are added per
// thread in CTA order, then in a fixed tree.
template <typename V>
__global__ void __launch_bounds__(NT) k_bitsums_finish(const V* __restrict__ part, int g, int first,
                                                       V* __restrict__ out) {
    using A = Acc<V>;
    let_next_start();
    wait_for_previous();
    const uint32_t o = blockIdx.x + (uint32_t)first, t = threadIdx.x, ncta = 1u << g;
    const int b = o ? (int)(o - 1) / 2 : 0, one = o ? (int)(o - 1) & 1 : 0;
    const bool cta_bit = o && b >= 12 && b < 12 + g;
    int slot = 0;  // the totals, for o = 0 and for CTA bits
    if (o && b < 12) slot = (int)o;
    else if (o && !cta_bit) slot = 1 + 2 * (b - g) + one;
    const V* p = part + (size_t)slot * ncta;
    V s = A::zero();
    for (uint32_t c = t; c < ncta; c += NT)
        if (!cta_bit || (int)((c >> (b - 12)) & 1u) == one) s = A::add(s, p[c]);
    __shared__ V red[NT / 32];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s = A::add(s, A::shfl(s, d));
    if ((t & 31u) == 0) red[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
        s = red[0];
#pragma unroll
        for (int w = 1; w < NT / 32; w++) s = A::add(s, red[w]);
        out[o] = s;
    }
}

template <typename S>
__global__ void k_probs(const S* __restrict__ st, uint64_t dim, double* __restrict__ out) {
    for (uint64_t x = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; x < dim; x += (uint64_t)gridDim.x * blockDim.x) {
        const double2 a = ld_amp(st + x);
        out[x] = a.x * a.x + a.y * a.y;
    }
}

// ---- renormalisation of complex64 states ----
// ||psi||^2 in FP64: each CTA sums |a|^2 over a grid-stride range (16-byte
// loads, two amplitudes each, in a fixed per-thread order); finish_norm does
// the rest.
__global__ void __launch_bounds__(256) k_norm2_c64(const float4* __restrict__ st, uint64_t npairs, NormScratch N) {
    let_next_start();
    wait_for_previous();
    const uint32_t t = threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * 256;
    double acc = 0.0;
    uint64_t i = (uint64_t)blockIdx.x * 256 + t;
    for (; i + 3 * stride < npairs; i += 4 * stride) {
        float4 v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = __ldcs(st + i + k * stride);
#pragma unroll
        for (int k = 0; k < 4; k++)
            acc += ((double)v[k].x * v[k].x + (double)v[k].y * v[k].y) + ((double)v[k].z * v[k].z + (double)v[k].w * v[k].w);
    }
    for (; i < npairs; i += stride) {
        const float4 v = __ldcs(st + i);
        acc += ((double)v.x * v.x + (double)v.y * v.y) + ((double)v.z * v.z + (double)v.w * v.w);
    }
    finish_norm<256>(acc, N);
}

// Multiplies every amplitude by the scale the norm kernel wrote (read on
// the device: no host round trip between the two launches). The product is
// formed in FP64 and rounded once, so each amplitude carries only its own
// rounding error; a scale rounded to FP32 first would shift the whole norm
// by up to 2^-23.
__global__ void __launch_bounds__(256) k_scale_c64(float4* __restrict__ st, uint64_t npairs,
                                                   const double* __restrict__ out) {
    let_next_start();
    wait_for_previous();
    const double f = out[1];
    const uint64_t stride = (uint64_t)gridDim.x * 256;
    for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < npairs; i += stride) {
        float4 v = __ldcs(st + i);
        v.x = (float)((double)v.x * f);
        v.y = (float)((double)v.y * f);
        v.z = (float)((double)v.z * f);
        v.w = (float)((double)v.w * f);
        __stcs(st + i, v);
    }
}

}  // namespace

size_t renorm_scratch_bytes() { return (RN_GRID + 4) * sizeof(double); }

cudaError_t launch_norm_c64(const void* st, int n, void* scratch, cudaStream_t s) {
    if (n < 1) return cudaErrorInvalidValue;
    const uint64_t npairs = (1ull << n) / 2;
    const unsigned grid = (unsigned)(npairs < (uint64_t)RN_GRID * 256 ? (npairs + 255) / 256 : RN_GRID);
    return launch_after(k_norm2_c64, grid, 256, 0, s, (const float4*)st, npairs, norm_scratch(scratch));
}

cudaError_t launch_renorm_c64(void* st, int n, void* scratch, bool summed, cudaStream_t s) {
    const cudaError_t e = summed ? cudaSuccess : launch_norm_c64(st, n, scratch, s);
    if (e != cudaSuccess) return e;
    const uint64_t npairs = (1ull << n) / 2;
    const unsigned grid = (unsigned)(npairs < (uint64_t)RN_GRID * 256 ? (npairs + 255) / 256 : RN_GRID);
    return launch_after(k_scale_c64, grid, 256, 0, s, (float4*)st, npairs, (const double*)scratch + RN_GRID);
}

BitSumShape bitsum_shape(int n) {
    BitSumShape s{};
    if (n > 12) {
        // One CTA per tile up to 22 qubits (latency: every SM busy), then up
        // to 16 rounds per CTA, which keeps the partials under 1/1000 of the
        // state and leaves thousands of CTAs (2^14 at 30 qubits: 37 waves of
        // 3 per SM, so a last partial wave costs nothing).
        s.nr = n > 30 ? n - 26 : n > 26 ? 4 : n > 22 ? n - 22 : 0;
        if (s.nr > MAXR) s.nr = MAXR;
        s.g = n - 12 - s.nr;
    }
    s.grid = 1 << s.g;
    s.nout = 1 + 2 * (12 + s.nr);
    return s;
}

namespace {

template <typename V, typename S, bool SCALE>
cudaError_t bitsums(S* st, int n, int g, int nr, void* partials, void* out, const double* scale,
                    const int* err, int* err_out, cudaStream_t s, int first = 0) {
    if (nr < 0 || nr > MAXR || g < 0) return cudaErrorInvalidValue;
    if (n >= 12 ? n != 12 + g + nr : g + nr != 0) return cudaErrorInvalidValue;
    const size_t smem = nr ? (sizeof(V) * (NT / 32)) << nr : 0;
    V* dst = (V*)(g + nr ? partials : out);
    const cudaError_t e = launch_after(k_bitsums<V, S, SCALE>, 1u << g, NT, smem, s, st, n, g, nr, dst, scale, err, err_out);
    if (e != cudaSuccess || g + nr == 0) return e;
    return launch_after(k_bitsums_finish<V>, 1 + 2 * n - first, NT, 0, s, (const V*)partials, g, first, (V*)out);
}

}  // namespace

cudaError_t launch_bitsums(const void* st, int prec, int n, int kind, void* partials, void* out, const int* err,
                           int* err_out, cudaStream_t s) {
    const BitSumShape sh = bitsum_shape(n);
    if (prec == 0) {
        double2* p = (double2*)const_cast<void*>(st);
        return kind == 0 ? bitsums<double2, double2, false>(p, n, sh.g, sh.nr, partials, out, nullptr, err, err_out, s)
                         : bitsums<double, double2, false>(p, n, sh.g, sh.nr, partials, out, nullptr, err, err_out, s);
    }
    float2* p = (float2*)const_cast<void*>(st);
    return kind == 0 ? bitsums<double2, float2, false>(p, n, sh.g, sh.nr, partials, out, nullptr, err, err_out, s)
                     : bitsums<double, float2, false>(p, n, sh.g, sh.nr, partials, out, nullptr, err, err_out, s);
}

cudaError_t launch_renorm_bitsums_c64(void* st, int n, void* scratch, bool summed, void* partials, void* out,
                                      const int* err, int* err_out, cudaStream_t s) {
    const cudaError_t e = summed ? cudaSuccess : launch_norm_c64(st, n, scratch, s);
    if (e != cudaSuccess) return e;
    const BitSumShape sh = bitsum_shape(n);
    return bitsums<double2, float2, true>((float2*)st, n, sh.g, sh.nr, partials, out,
                                          (const double*)scratch + RN_GRID, err, err_out, s);
}

cudaError_t launch_bitsums_c128_shape(const void* st, int n, int g, int nr, void* partials, void* out,
                                      cudaStream_t s) {
    return bitsums<double2, double2, false>((double2*)const_cast<void*>(st), n, g, nr, partials, out, nullptr, nullptr, nullptr,
                                           s, 1);
}

cudaError_t launch_probs(const void* st, int prec, uint64_t dim, double* out, cudaStream_t s) {
    uint64_t blocks = (dim + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    if (prec == 0) k_probs<double2><<<(unsigned)blocks, 256, 0, s>>>((const double2*)st, dim, out);
    else k_probs<float2><<<(unsigned)blocks, 256, 0, s>>>((const float2*)st, dim, out);
    return cudaGetLastError();
}

}  // namespace kate
