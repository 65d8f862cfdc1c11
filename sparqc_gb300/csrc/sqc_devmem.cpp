// Device allocations and kept tables: see sqc_devmem.h.
#include "sqc_devmem.h"

#include <list>
#include <mutex>

namespace sqc {

namespace {

struct Kept {
    const void* owner;
    int device;
    void* base;
    size_t bytes;
};

std::mutex g_mu;
std::list<Kept>& g_kept = *new std::list<Kept>;   // oldest first (never destroyed: states may outlive statics)

int current_device() {
    int d = 0;
    cudaGetDevice(&d);
    return d;
}

template <class F>
bool drop_if(F&& f) {
    bool any = false;
    for (auto it = g_kept.begin(); it != g_kept.end();) {
        if (!f(*it)) {
            ++it;
            continue;
        }
        cudaFree(it->base);
        it = g_kept.erase(it);
        any = true;
    }
    return any;
}

}  // namespace

cudaError_t device_alloc_bytes(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    if (!spare_drop_all()) return e;
    e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) cudaGetLastError();
    return e;
}

void spare_put(const void* owner, void* base, size_t bytes, size_t limit) {
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(g_mu);
    drop_if([&](const Kept& k) { return k.owner == owner; });
    size_t held = bytes;
    for (const Kept& k : g_kept) held += k.device == dev ? k.bytes : 0;
    drop_if([&](const Kept& k) {
        if (k.device != dev || held <= limit) return false;
        held -= k.bytes;
        return true;
    });
    if (held > limit) {
        cudaFree(base);
        return;
    }
    try {
        g_kept.push_back(Kept{owner, dev, base, bytes});
    } catch (...) {
        cudaFree(base);
    }
}

void* spare_take(const void* owner, size_t bytes) {
    std::lock_guard<std::mutex> lock(g_mu);
    for (auto it = g_kept.begin(); it != g_kept.end(); ++it) {
        if (it->owner != owner || it->bytes != bytes) continue;
        void* base = it->base;
        g_kept.erase(it);
        return base;
    }
    return nullptr;
}

size_t spare_bytes(const void* owner) {
    std::lock_guard<std::mutex> lock(g_mu);
    size_t n = 0;
    for (const Kept& k : g_kept) n += k.owner == owner ? k.bytes : 0;
    return n;
}

void spare_drop(const void* owner) {
    std::lock_guard<std::mutex> lock(g_mu);
    drop_if([&](const Kept& k) { return k.owner == owner; });
}

bool spare_drop_all() {
    const int dev = current_device();
    std::lock_guard<std::mutex> lock(g_mu);
    return drop_if([&](const Kept& k) { return k.device == dev; });
}

}  // namespace sqc
