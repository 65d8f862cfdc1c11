// Key-ordered readout of mapped tables (sqc_rank.cu): host-side launchers.
//
// A mapped table's buckets are addressed by key bits, so its keys in order are its buckets in the
// order of those bits: no sort is needed. Rank r of a table with n mapped bits is the bucket whose
// bits, from the lowest mapped qubit up, are r's (with the key frame applied).
#pragma once
#include <cstdint>
#include <cuda_runtime_api.h>
#include "sqc_types.h"

namespace sqc {

constexpr uint32_t kRankTile = 1024;   // ranks per block

// One table to read: which of its keys, and where its tiles begin among all tables' tiles.
struct RankJob {
    TableDev t;
    const Ctl* ctl;
    unsigned long long frame;    // actual key = stored key ^ frame
    unsigned long long tile0;    // first tile
    uint32_t bucket_frame;       // frame bits on the mapped bits, as bucket bits
    uint32_t bm, bv;             // buckets whose keys may match: (b & bm) == bv ...
    uint32_t slots;              // ... and the slots of theirs that do; 0: nothing matches
    uint8_t bit_of[kMaxMapBits + 1];   // bucket bit of each rank bit
    unsigned long long tiles() const { return ((1ULL << t.map_n) + kRankTile - 1) / kRankTile; }
};

// The keys of table t (mapped) whose stored form has (key & smask) == sval.
RankJob rank_job(const TableDev& t, const Ctl* ctl, unsigned long long frame, unsigned long long smask,
                 unsigned long long sval);

// Whether a ranked readout suits a mapped table of n bits holding nnz keys: it reads every header
// of the span (about 30 us at 2^22), a list readout needs a sort.
inline bool rank_worth(uint32_t n, unsigned long long nnz) {
    return (1ULL << n) <= (1ULL << 22) || (1ULL << n) <= 16 * nnz;
}

// The same for the batch's and the server's tables, whose list readouts are sorted on the host (one circuit of 600
// keys, FP64: 2^18 headers 75 us, 2^20 93, by the list 76).
inline bool rank_worth_unsorted(uint32_t n, unsigned long long nnz) {
    return (1ULL << n) <= (1ULL << 18) || (1ULL << n) <= 256 * nnz;
}

// Device scratch of ranked readouts, grown as needed: a count per tile, and for several jobs the
// jobs, their counts and the total.
struct RankScratch {
    unsigned long long* tiles = nullptr;
    RankJob* jobs = nullptr;
    unsigned long long* counts = nullptr;   // one per job, then the total
    size_t tiles_cap = 0, jobs_cap = 0;
    cudaError_t need(size_t ntiles, size_t njobs);
    void release();
};

// Entries of the jobs in job order, each job's in key order, into (keys, re, im); entries at or
// beyond cap are counted but not written. tiles: device scratch of total_tiles words. *total (device)
// receives the entry count, counts (device, optional) that of each job. With one job, pass it in
// `one` and jobs null; else jobs is a device array.
cudaError_t launch_ranked(const RankJob& one, const RankJob* jobs, uint32_t njobs, unsigned long long total_tiles,
                          unsigned long long* tiles, bool dbl, unsigned long long* keys, double* re, double* im,
                          unsigned long long cap, bool drop_negl, PruneBits pb, unsigned long long* total,
                          unsigned long long* counts, cudaStream_t st);

}  // namespace sqc
