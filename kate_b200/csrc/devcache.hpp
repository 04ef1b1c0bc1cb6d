// Reuse of device buffers (simulator states and workspaces, batch arenas),
// streams and pinned memory.
//
// A caller that loops `Simulator(circuit).execute()` (the reference's usage,
// HIPcode/simulator.hpp:243-300 allocates the state in every constructor and
// frees it in the destructor) would pay cudaMalloc and cudaFree on every
// iteration: hundreds of milliseconds for a state of tens of GB, and for a
// small one most of the iteration (16 qubits: 0.8 of 1.6 ms in cudaMalloc,
// cudaFree and the stream's creation and destruction). The most recently
// released large buffer of each device is kept instead and handed to the next
// request it covers (up to 4x its size); of smaller ones up to
// kSmallBlocks, kSmallTotal bytes in all, are kept per device. They stay
// allocated until a request they do not cover fails or (large) needs memory,
// the creation of a server (which takes its budget in one allocation) or
// kate_release_cached_memory frees them.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace kate {

// Buffers below this size are small.
constexpr size_t kCacheMinBytes = size_t(64) << 20;
constexpr int kSmallBlocks = 16;
constexpr size_t kSmallTotal = size_t(128) << 20;

// Allocates at least `bytes` on the current device (`device`), reusing a
// cached buffer that covers the request.
cudaError_t cached_malloc(void** p, size_t bytes, int device);
// Releases a buffer from cached_malloc (the current device is `device`).
// Waits for the device first unless the caller just has (`idle`), so no
// kernel still uses it when it is reused.
void cached_free(void* p, int device, bool idle = false);
// Waits for the device; clears the error when that fails.
bool device_idle();

// A non-blocking stream of the current device (`device`): one given back
// before (up to kStreams are kept per device), or a new one. stream_give
// takes a stream without work in flight.
constexpr int kStreams = 8;
cudaError_t stream_take(cudaStream_t* s, int device);
void stream_give(cudaStream_t s, int device);
// Frees the cached buffers and streams of `device` (-1: of every device) and,
// for -1, the pinned slab below when none of its slots is out.
void release_cached(int device);

// Pinned host memory for small results (a measurement's sums, samples): slots
// of kPinnedSlotBytes from one slab of kPinnedSlots, allocated at the first
// request and mapped into every device's address space, so that a kernel
// writes its results where the host reads them. pinned_take returns null when
// no slot (or no pinned memory) is left; the caller then copies from device
// memory. A slot belongs to its taker until pinned_give. Thread-safe.
constexpr size_t kPinnedSlotBytes = 16 * 1024;
constexpr int kPinnedSlots = 64;
void* pinned_take();
void pinned_give(void* p);

}  // namespace kate
