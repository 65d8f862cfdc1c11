// Key-ordered readout of mapped tables: see sqc_rank.h.
//
// Three launches: entries per tile of kRankTile ranks, a scan over the tiles, and the copy. Reads
// 16 bytes per header and 16 (FP64) per key, writes 24 per key: bound by HBM (2^25 keys FP64:
// against a list readout, a 64-bit radix sort of key-index pairs and a gather).
#include "sqc_rank.h"
#include "sqc_devmem.h"
#include "sqc_device.cuh"

#include <algorithm>

namespace sqc {
namespace {

constexpr int kRankThreads = 256;
constexpr int kPerThread = kRankTile / kRankThreads;

template <class T> struct AmpOf { using V = double2; };
template <> struct AmpOf<float> { using V = float2; };

__device__ __forceinline__ const RankJob& job_of(const RankJob& one, const RankJob* jobs, uint32_t njobs,
                                                 unsigned long long tile) {
    if (!jobs) return one;
    uint32_t lo = 0, hi = njobs - 1;   // the last job that begins at or before the tile
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) / 2;
        if (jobs[mid].tile0 <= tile) lo = mid;
        else hi = mid - 1;
    }
    return jobs[lo];
}

// Buckets of the tile's ranks and the slots of each that are read, into shared memory (ends with a
// barrier). A rank beyond the table has no slots.
template <class T>
__device__ __forceinline__ void tile_slots(const RankJob& J, unsigned long long tile, bool drop, const PruneBits& pb,
                                           uint32_t* bucket, uint32_t* slots) {
    const unsigned ep = J.ctl->epoch;
    const unsigned long long r0 = (tile - J.tile0) * kRankTile, ranks = 1ULL << J.t.map_n;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
        const unsigned long long r = r0 + threadIdx.x + i * kRankThreads;
        uint32_t b = 0, m = 0;
        if (r < ranks) {
            for (uint32_t k = 0; k < J.t.map_n; ++k) b |= (uint32_t)((r >> k) & 1ULL) << J.bit_of[k];
            b ^= J.bucket_frame;
            if ((b & J.bm) == J.bv) {
                const Header h = load_hdr(J.t.hdr + b);
                if (h.epoch == ep) m = h.aux & J.slots;
            }
        }
        bucket[threadIdx.x + i * kRankThreads] = b;
        slots[threadIdx.x + i * kRankThreads] = m;
    }
    __syncthreads();
    if (!drop) return;
    const int j = threadIdx.x & 15;   // a half-warp per bucket
    for (uint32_t i = threadIdx.x >> 4; i < kRankTile; i += kRankThreads / 16) {
        const uint32_t m = slots[i];
        bool keep = false;
        if ((m >> j) & 1u) {
            const typename AmpOf<T>::V a =
                reinterpret_cast<const typename AmpOf<T>::V*>(J.t.amps)[(size_t)bucket[i] * kSlots + j];
            keep = !negligible(Cx<T>{a.x, a.y}, pb);
        }
        const unsigned bal = __ballot_sync(kFull, keep);
        if (j == 0) slots[i] = (threadIdx.x & 16) ? bal >> 16 : bal & 0xFFFFu;
    }
    __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(kRankThreads)
    rank_count_kernel(const __grid_constant__ RankJob one, const RankJob* jobs, uint32_t njobs, unsigned long long* tiles,
                      int drop, PruneBits pb) {
    __shared__ uint32_t bucket[kRankTile], slots[kRankTile];
    __shared__ unsigned sum;
    if (threadIdx.x == 0) sum = 0;
    const RankJob& J = job_of(one, jobs, njobs, blockIdx.x);
    tile_slots<T>(J, blockIdx.x, drop != 0, pb, bucket, slots);
    unsigned n = 0;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) n += __popc(slots[threadIdx.x + i * kRankThreads]);
    n = __reduce_add_sync(kFull, n);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sum, n);
    __syncthreads();
    if (threadIdx.x == 0) tiles[blockIdx.x] = sum;
}

// Exclusive scan of the tiles' counts in place (one block); the total, and each job's count.
__global__ void __launch_bounds__(1024)
    rank_scan_kernel(const RankJob* jobs, uint32_t njobs, unsigned long long ntiles, unsigned long long* tiles,
                     unsigned long long* total, unsigned long long* counts) {
    __shared__ unsigned long long part[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long carry = 0;
    for (unsigned long long t0 = 0; t0 < ntiles; t0 += blockDim.x) {
        const unsigned long long t = t0 + threadIdx.x;
        const unsigned long long v = t < ntiles ? tiles[t] : 0ULL;
        unsigned long long x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(kFull, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) part[w] = x;
        __syncthreads();
        unsigned long long before = 0, all = 0;
        for (int i = 0; i < 32; ++i) {
            before += i < w ? part[i] : 0ULL;
            all += part[i];
        }
        if (t < ntiles) tiles[t] = carry + before + x - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
    if (counts) {
        for (uint32_t j = threadIdx.x; j < njobs; j += blockDim.x)
            counts[j] = (j + 1 < njobs ? tiles[jobs[j + 1].tile0] : carry) - tiles[jobs[j].tile0];
    }
}

template <class T>
__global__ void __launch_bounds__(kRankThreads)
    rank_copy_kernel(const __grid_constant__ RankJob one, const RankJob* jobs, uint32_t njobs,
                     const unsigned long long* tiles, int drop, PruneBits pb, unsigned long long* __restrict__ okeys,
                     double* __restrict__ ore, double* __restrict__ oim, unsigned long long cap) {
    __shared__ uint32_t bucket[kRankTile], slots[kRankTile], at[kRankTile];
    __shared__ unsigned part[kRankThreads / 32];
    const RankJob& J = job_of(one, jobs, njobs, blockIdx.x);
    tile_slots<T>(J, blockIdx.x, drop != 0, pb, bucket, slots);
    // where each rank's entries begin within the tile
    unsigned mine[kPerThread], n = 0;
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) {
        mine[i] = n;
        n += __popc(slots[threadIdx.x * kPerThread + i]);
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned x = n;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) part[w] = x;
    __syncthreads();
    unsigned before = x - n;
    for (int i = 0; i < w; ++i) before += part[i];
#pragma unroll
    for (int i = 0; i < kPerThread; ++i) at[threadIdx.x * kPerThread + i] = before + mine[i];
    __syncthreads();
    const unsigned long long base = tiles[blockIdx.x];
    const uint32_t fs = (uint32_t)J.frame & 15u;
    const int jj = lane & 15;                     // place in key order within the bucket
    const int j = jj ^ (int)fs;                   // ... and its slot
    for (uint32_t i = threadIdx.x >> 4; i < kRankTile; i += kRankThreads / 16) {
        const uint32_t m = slots[i];
        const bool keep = (m >> j) & 1u;
        const unsigned bal = __ballot_sync(kFull, keep);
        if (!keep) continue;
        const unsigned half = (lane & 16) ? bal >> 16 : bal & 0xFFFFu;
        const unsigned long long to = base + at[i] + __popc(half & ((1u << jj) - 1u));
        if (to >= cap) continue;
        const uint32_t b = bucket[i];
        const size_t s = (size_t)b * kSlots + j;
        const typename AmpOf<T>::V a = reinterpret_cast<const typename AmpOf<T>::V*>(J.t.amps)[s];
        okeys[to] = ((J.t.hdr[b].group << kSlotBits) | (unsigned long long)j) ^ J.frame;
        ore[to] = (double)a.x;
        oim[to] = (double)a.y;
    }
}

}  // namespace

cudaError_t RankScratch::need(size_t ntiles, size_t njobs) {
    if (ntiles > tiles_cap) {
        if (tiles) cudaFree(tiles);
        tiles = nullptr;
        tiles_cap = 0;
        const cudaError_t e = device_alloc(&tiles, ntiles * sizeof(unsigned long long));
        if (e != cudaSuccess) return e;
        tiles_cap = ntiles;
    }
    if (njobs > jobs_cap) {
        if (jobs) cudaFree(jobs);
        if (counts) cudaFree(counts);
        jobs = nullptr;
        counts = nullptr;
        jobs_cap = 0;
        cudaError_t e = device_alloc(&jobs, njobs * sizeof(RankJob));
        if (e == cudaSuccess) e = device_alloc(&counts, (njobs + 1) * sizeof(unsigned long long));
        if (e != cudaSuccess) return e;
        jobs_cap = njobs;
    }
    return cudaSuccess;
}

void RankScratch::release() {
    if (tiles) cudaFree(tiles);
    if (jobs) cudaFree(jobs);
    if (counts) cudaFree(counts);
    *this = RankScratch();
}

RankJob rank_job(const TableDev& t, const Ctl* ctl, unsigned long long frame, unsigned long long smask,
                 unsigned long long sval) {
    RankJob J;
    J.t = t;
    J.ctl = ctl;
    J.frame = frame;
    J.tile0 = 0;
    J.bucket_frame = J.bm = J.bv = 0;
    uint8_t order[kMaxMapBits + 1] = {};
    for (uint32_t i = 0; i < t.map_n; ++i) order[i] = (uint8_t)i;
    std::sort(order, order + t.map_n, [&](uint8_t x, uint8_t y) { return t.map_q[x] < t.map_q[y]; });
    unsigned long long mapped = 15ULL;
    for (uint32_t i = 0; i < t.map_n; ++i) {
        J.bit_of[i] = order[i];
        const uint32_t q = t.map_q[i] + (uint32_t)kSlotBits;
        mapped |= 1ULL << q;
        J.bucket_frame |= (uint32_t)((frame >> q) & 1ULL) << i;
        J.bm |= (uint32_t)((smask >> q) & 1ULL) << i;
        J.bv |= (uint32_t)(((smask & sval) >> q) & 1ULL) << i;
    }
    for (uint32_t i = t.map_n; i <= kMaxMapBits; ++i) J.bit_of[i] = 0;
    J.slots = 0;
    for (uint32_t j = 0; j < (uint32_t)kSlots; ++j)
        if ((j & smask) == (sval & smask & 15ULL)) J.slots |= 1u << j;
    // bits outside the map are stored as 0 in every key; a value outside its mask matches nothing
    if ((sval & ~smask) || (sval & smask & ~mapped)) J.slots = 0;
    return J;
}

cudaError_t launch_ranked(const RankJob& one, const RankJob* jobs, uint32_t njobs, unsigned long long total_tiles,
                          unsigned long long* tiles, bool dbl, unsigned long long* keys, double* re, double* im,
                          unsigned long long cap, bool drop_negl, PruneBits pb, unsigned long long* total,
                          unsigned long long* counts, cudaStream_t st) {
    const unsigned grid = (unsigned)total_tiles;
    const int drop = drop_negl ? 1 : 0;
    if (dbl) rank_count_kernel<double><<<grid, kRankThreads, 0, st>>>(one, jobs, njobs, tiles, drop, pb);
    else rank_count_kernel<float><<<grid, kRankThreads, 0, st>>>(one, jobs, njobs, tiles, drop, pb);
    rank_scan_kernel<<<1, 1024, 0, st>>>(jobs, njobs, total_tiles, tiles, total, counts);
    if (dbl) rank_copy_kernel<double><<<grid, kRankThreads, 0, st>>>(one, jobs, njobs, tiles, drop, pb, keys, re, im, cap);
    else rank_copy_kernel<float><<<grid, kRankThreads, 0, st>>>(one, jobs, njobs, tiles, drop, pb, keys, re, im, cap);
    return cudaGetLastError();
}

}  // namespace sqc
