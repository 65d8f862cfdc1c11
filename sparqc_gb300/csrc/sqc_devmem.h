// Device memory of the library's objects, and the tables that states keep for their next rebuild.
//
// A rebuild of a hashed table leaves the old table, and circuits whose keys move are rebuilt several times:
// the next rebuild takes the kept table instead of allocating (a million loaded keys, 60 gates: 8.3 ms, and
// 15.2 with an allocation each time). Kept tables belong to the whole process: at most a quarter of a device
// in all (three such states, 13.6 GB each, run in turns 8.0-9.5 ms, with an eighth 14.5-15.3), the oldest freed first,
// and given back whenever an allocation of any state, batch or server on
// that device fails. A kept table is not in use by any stream (a rebuild ends with a wait).
#pragma once
#include <cstddef>
#include <cuda_runtime_api.h>

namespace sqc {

// cudaMalloc on the current device; when it fails, kept tables are freed and it is tried again. A failure
// is not left in cudaGetLastError.
cudaError_t device_alloc_bytes(void** p, size_t bytes);
template <class T>
cudaError_t device_alloc(T** p, size_t bytes) {
    return device_alloc_bytes(reinterpret_cast<void**>(p), bytes);
}

// Keep a table (one allocation of the current device) of an owner, whose last one is freed, and as many others
// as it takes to hold at most `limit` bytes on the device; the table itself is freed if it is larger.
void spare_put(const void* owner, void* base, size_t bytes, size_t limit);
// The owner's kept table, if it has this size, else null.
void* spare_take(const void* owner, size_t bytes);
size_t spare_bytes(const void* owner);
void spare_drop(const void* owner);
// Free every kept table of the current device; whether there was one.
bool spare_drop_all();

}  // namespace sqc
