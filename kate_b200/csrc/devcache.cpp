// Reuse of device buffers, streams and pinned memory. See devcache.hpp.
#include "devcache.hpp"

#include <algorithm>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace kate {

namespace {

struct Block {
    void* p = nullptr;
    size_t bytes = 0;
};

constexpr int kMaxDevices = 64;
std::mutex g_mu;
Block g_cached[kMaxDevices];                   // one large released buffer per device
std::vector<Block> g_small[kMaxDevices];       // small released buffers
std::vector<cudaStream_t> g_streams[kMaxDevices];
std::unordered_map<void*, size_t> g_live;      // buffers handed out, with their real size
char* g_slab = nullptr;                        // pinned slots
std::vector<char*> g_free_slots;

// Runs f with `device` current.
template <typename F>
void on_device(int device, F&& f) {
    int cur = 0;
    cudaGetDevice(&cur);
    if (cur != device) cudaSetDevice(device);
    f();
    if (cur != device) cudaSetDevice(cur);
}

void free_cached_locked(int device) {
    Block& c = g_cached[device];
    if (!c.p) return;
    on_device(device, [&] { cudaFree(c.p); });
    c = Block{};
}

void free_small_locked(int device) {
    if (g_small[device].empty()) return;
    on_device(device, [&] {
        for (const Block& b : g_small[device]) cudaFree(b.p);
    });
    g_small[device].clear();
}

void free_all_locked(int device) {
    free_cached_locked(device);
    free_small_locked(device);
    if (g_streams[device].empty()) return;
    on_device(device, [&] {
        for (cudaStream_t s : g_streams[device]) cudaStreamDestroy(s);
    });
    g_streams[device].clear();
}

}  // namespace

bool device_idle() {
    if (cudaDeviceSynchronize() == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

cudaError_t cached_malloc(void** p, size_t bytes, int device) {
    *p = nullptr;
    if (device < 0 || device >= kMaxDevices) return cudaMalloc(p, bytes);
    std::lock_guard<std::mutex> lk(g_mu);
    if (bytes < kCacheMinBytes) {
        std::vector<Block>& v = g_small[device];
        bytes = (bytes + 0xffff) & ~size_t(0xffff);
        size_t at = v.size();
        for (size_t i = 0; i < v.size(); i++)
            if (v[i].bytes >= bytes && v[i].bytes <= std::max(4 * bytes, size_t(1) << 20) &&
                (at == v.size() || v[i].bytes < v[at].bytes))
                at = i;
        if (at < v.size()) {
            *p = v[at].p;
            g_live[*p] = v[at].bytes;
            v.erase(v.begin() + (long)at);
            return cudaSuccess;
        }
    } else {
        Block& c = g_cached[device];
        if (c.p && c.bytes >= bytes && c.bytes / 4 <= bytes) {
            *p = c.p;
            g_live[c.p] = c.bytes;
            c = Block{};
            return cudaSuccess;
        }
        free_cached_locked(device);
    }
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        // What is held for reuse may be what is missing.
        cudaGetLastError();
        free_cached_locked(device);
        free_small_locked(device);
        e = cudaMalloc(p, bytes);
    }
    if (e != cudaSuccess) return e;
    g_live[*p] = bytes;
    return cudaSuccess;
}

void cached_free(void* p, int device, bool idle) {
    if (!p) return;
    idle = idle || device_idle();
    std::lock_guard<std::mutex> lk(g_mu);
    auto it = g_live.find(p);
    if (it == g_live.end() || !idle || device < 0 || device >= kMaxDevices) {
        if (it != g_live.end()) g_live.erase(it);
        cudaFree(p);
        return;
    }
    const size_t bytes = it->second;
    g_live.erase(it);
    if (bytes >= kCacheMinBytes) {
        free_cached_locked(device);
        g_cached[device] = Block{p, bytes};
        return;
    }
    // The oldest blocks make room.
    std::vector<Block>& v = g_small[device];
    v.push_back(Block{p, bytes});
    size_t total = 0;
    for (const Block& b : v) total += b.bytes;
    while ((int)v.size() > kSmallBlocks || total > kSmallTotal) {
        total -= v.front().bytes;
        cudaFree(v.front().p);
        v.erase(v.begin());
    }
}

cudaError_t stream_take(cudaStream_t* s, int device) {
    if (device >= 0 && device < kMaxDevices) {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_streams[device].empty()) {
            *s = g_streams[device].back();
            g_streams[device].pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
}

void stream_give(cudaStream_t s, int device) {
    if (!s) return;
    if (device >= 0 && device < kMaxDevices) {
        std::lock_guard<std::mutex> lk(g_mu);
        if ((int)g_streams[device].size() < kStreams) {
            g_streams[device].push_back(s);
            return;
        }
    }
    cudaStreamDestroy(s);
}

void release_cached(int device) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (device >= 0 && device < kMaxDevices) {
        free_all_locked(device);
        return;
    }
    for (int d = 0; d < kMaxDevices; d++) free_all_locked(d);
    if (g_slab && (int)g_free_slots.size() == kPinnedSlots) {
        cudaFreeHost(g_slab);
        g_slab = nullptr;
        g_free_slots.clear();
    }
}

void* pinned_take() {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_slab) {
        void* p = nullptr;
        if (cudaHostAlloc(&p, kPinnedSlotBytes * kPinnedSlots, cudaHostAllocPortable) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        g_slab = static_cast<char*>(p);
        for (int i = kPinnedSlots; i-- > 0;) g_free_slots.push_back(g_slab + (size_t)i * kPinnedSlotBytes);
    }
    if (g_free_slots.empty()) return nullptr;
    void* p = g_free_slots.back();
    g_free_slots.pop_back();
    return p;
}

void pinned_give(void* p) {
    if (!p) return;
    std::lock_guard<std::mutex> lk(g_mu);
    g_free_slots.push_back(static_cast<char*>(p));
}

}  // namespace kate
