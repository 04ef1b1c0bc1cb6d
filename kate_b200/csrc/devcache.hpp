// Reuse of large device buffers (simulator states, batch arenas).
//
// A caller that loops `Simulator(circuit).execute()` (the reference's usage,
// HIPcode/simulator.hpp:243-300 allocates the state in every constructor and
// frees it in the destructor) would pay cudaMalloc and cudaFree of the whole
// state on every iteration: hundreds of milliseconds for tens of GB. The most
// recently released large buffer of each device is kept instead and handed
// to the next request it covers (up to 4x its size). The cached buffer stays
// allocated until a request it does not cover, the creation of a server
// (which takes its budget in one allocation) or kate_release_cached_memory
// frees it.
#pragma once

#include <cstddef>

#include <cuda_runtime.h>

namespace kate {

// Buffers below this size are allocated and freed directly.
constexpr size_t kCacheMinBytes = size_t(64) << 20;

// Allocates at least `bytes` on the current device (`device`), reusing the
// cached buffer when it covers the request.
cudaError_t cached_malloc(void** p, size_t bytes, int device);
// Releases a buffer from cached_malloc (the current device is `device`).
// Waits for the device first, so no kernel still uses it when it is reused.
void cached_free(void* p, int device);
// Frees the cached buffer of `device` (-1: of every device) and, for -1, the
// pinned slab below when none of its slots is out.
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
