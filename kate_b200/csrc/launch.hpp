// Host-side launchers of the CUDA kernels (defined in the .cu files).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>

#include "device_types.h"

namespace kate {

// Launches a kernel that may start before the one before it in the stream has
// finished, for kernels that call wait_for_previous (k_common.cuh) before
// they touch any memory that one writes or reads. It hides the launch gap
// between the dependent kernels of a run (about 1.5 us each).
template <typename... KArgs, typename... Args>
cudaError_t launch_after(void (*kernel)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                         Args... args) {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &a;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<KArgs>(args)...);
}

// Product-state initialisation value table: v[b][p] is the factor for
// physical bit p having value b.
struct ProductInit {
    double v[2][KATE_MAX_QUBITS][2];
    int n;
};

// prec: 0 = complex128 (double2 amplitudes), 1 = complex64 (float2).
cudaError_t launch_set_basis0(void* st, uint64_t dim, int prec, cudaStream_t s);
cudaError_t launch_init_product(void* st, int n, const ProductInit& P, int prec, cudaStream_t s);
cudaError_t launch_pass_generic(void* st, int prec, const DevPass& p, const DevOp* ops, const void* pool, int grid,
                                cudaStream_t s);
cudaError_t launch_probs(const void* st, int prec, uint64_t dim, double* out, cudaStream_t s);
// Renormalisation of a complex64 state (n >= 1 qubits): ||psi||^2 reduced in
// FP64 on the device, then every amplitude multiplied by 1 / ||psi||. The
// scratch (renorm_scratch_bytes(), zeroed once) holds the per-CTA partials,
// then ||psi||^2 and 1 / ||psi|| as doubles 0 and 1 after the partials
// (offset renorm_result_offset()), then a counter.
size_t renorm_scratch_bytes();
// Inverse-CDF sampling on the device (k_sample.cu): out[k] receives shot k of
// `seed` as a basis index in program labels, label q read from physical bit
// phys[q]. scratch: sample_scratch_doubles(n) doubles.
struct SampleLabels {
    uint8_t phys[KATE_MAX_QUBITS];
};
size_t sample_scratch_doubles(int n);
cudaError_t launch_sample(const void* st, int prec, int n, uint64_t seed, int shots, const SampleLabels& L,
                          double* scratch, uint64_t* out, cudaStream_t s);
// Device gate merger (k_merge.cu): out[b] is the product of blocks[b] as one
// dense gate on the sorted union of its qubits (at most 10), bit-identical
// to merge_gates (circuit.hpp); all blocks in one launch on `device`, then
// a synchronise of `stream`. Returns "" or an error message.
struct Gate;
std::string merge_gates_device(const std::vector<std::vector<Gate>>& blocks, int device, cudaStream_t stream,
                               std::vector<Gate>* out);
cudaError_t launch_norm_c64(const void* st, int n, void* scratch, cudaStream_t s);  // ||psi||^2 only
constexpr int RN_GRID = 148 * 4;  // CTAs at most
constexpr size_t renorm_result_offset() { return RN_GRID * sizeof(double); }
// summed: the pass before has left ||psi||^2 in the scratch (launch_block_c64).
cudaError_t launch_renorm_c64(void* st, int n, void* scratch, bool summed, cudaStream_t s);

// c128 state (double2 amplitudes)
cudaError_t launch_set_basis0_c128(void* st, uint64_t dim, cudaStream_t s);
cudaError_t launch_init_product_c128(void* st, int n, const ProductInit& P, cudaStream_t s);
// One generic group pass (shared-memory tile, any op mix). Dense ops up to 5 qubits.
cudaError_t launch_pass_generic_c128(void* st, int n, const DevPass& p, const DevOp* ops, const void* pool,
                                     int grid, cudaStream_t s);
int generic_pass_grid(int n, int m, int device);
// Register-staged programs [p0, p1) of a state of fewer than 12 qubits, in
// one CTA (k_small.cu), with 2^reg_bits amplitudes per thread. smem_ops:
// whether any has shared-memory ops. init: 0 the state as it is, 1 |0...0>,
// 2 the product state PI. sums (complex128, nullable): the amplitude bit sums
// of the final state, as launch_bitsums writes them. small_prepare once per
// device first.
cudaError_t small_prepare(int device);
cudaError_t launch_small(void* st, int prec, int n, int reg_bits, const BatchProg* progs, int p0, int p1,
                         const void* blob, const DevOp* sops, const void* pool, bool smem_ops, int init,
                         const ProductInit& PI, void* sums, cudaStream_t s);
// Register-staged tile kernel (12-qubit tiles, 256 threads x 16 amplitudes),
// prec 0: complex128 / FP64, 1: complex64 / FP32. nbuf = 2: one CTA per SM
// with a prefetched second tile; nbuf = 1: two CTAs per SM with one tile each.
cudaError_t launch_tile(void* st, int prec, const PassProg& prog, const DevOp* sops, const void* pool, int grid,
                        int nbuf, cudaStream_t s);
int tile_pass_grid(int n, int device, int nbuf, int prec);
// Warp-specialised complex128 tile kernel (k_tile_ws.cu): one CTA per SM, a
// producer warp streaming tiles with bulk copies into a ring of shared-memory
// buffers. Applies to register-staged programs without shared-memory ops
// whose tile holds physical bits 0..3. err: device int set to 1 if a bounded
// wait gave up.
bool tile_ws_applies(const PassProg& prog);
int tile_ws_grid(int n, int device);
cudaError_t launch_tile_ws(void* st, const PassProg& prog, int* err, int grid, cudaStream_t s);

// Complex64 pass of 5-qubit dense blocks on the tensor cores. from_zero: the
// input is |0...0> and the state is not read. err: device int set to 1 if a
// bounded wait gave up. norm: null, or the renormalisation scratch, which then
// receives ||psi||^2 of the result.
cudaError_t launch_block_c64(void* st, const BlockProg& prog, const void* bimg, bool from_zero, int* err, int grid,
                             void* norm, cudaStream_t s);
int block_c64_grid(int n, int device);

// Persistent batch kernel (k_batch.cu). head, done[circuits], zout (large
// circuits' outputs) must be zero at launch; err is set to 1 when a
// dependency wait gave up after wait_ns (the kernel then stops). psum /
// unif / sout: chunk sums, uniforms and samples of circuits that sample (may
// be null otherwise).
cudaError_t launch_batch(void* arena, int prec, const BatchTask* tasks, int ntasks, const BatchCirc* circs,
                         const BatchProg* progs, const void* blob, const DevOp* sops, const void* pool, int* head,
                         int* done, double* zout, int* err, int grid, cudaStream_t s, double* psum = nullptr,
                         const double* unif = nullptr, uint64_t* sout = nullptr,
                         unsigned long long wait_ns = 5000000000ull, int tensor_blocks = 0);
int batch_grid(int device, int prec, bool tensor_blocks = false);

// Bit sums (k_measure.cu): out[0] = total, out[1 + 2b + v] = the sum over the
// amplitudes whose physical index bit b is v; kind 0 sums amplitudes (double2
// values), kind 1 |a|^2 (double values). `out` holds max(25, 1 + 2n) values,
// `partials` grid * nout of the shape below (CTA partials). *err_out receives
// *err (the error flag of the kernels before; both nullable): out and err_out
// may lie in pinned host memory, so that a caller waits once and copies
// nothing.
struct BitSumShape {
    int grid;   // CTAs (2^g)
    int g;      // coset bits handled by the grid
    int nr;     // round bits handled per CTA
    int nout;   // partial values per CTA
};
BitSumShape bitsum_shape(int n);
cudaError_t launch_bitsums(const void* st, int prec, int n, int kind, void* partials, void* out, const int* err,
                           int* err_out, cudaStream_t s);
// launch_renorm_c64 and the amplitude bit sums (kind 0) of the rescaled
// state, which the rescaling pass adds up as it goes.
cudaError_t launch_renorm_bitsums_c64(void* st, int n, void* scratch, bool summed, void* partials, void* out,
                                      const int* err, int* err_out, cudaStream_t s);
// Amplitude bit sums of a complex128 state with an explicit shape: 2^g CTAs,
// 2^nr rounds each (n = 12 + g + nr when n >= 12, nr <= 8). When g + nr > 0
// the total out[0] is not written.
cudaError_t launch_bitsums_c128_shape(const void* st, int n, int g, int nr, void* partials, void* out,
                                      cudaStream_t s);

}  // namespace kate
