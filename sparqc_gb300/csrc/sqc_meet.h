// The bounded wait of a block at a meeting of a run (run_kernel, sqc_pass.cu), as a function of what it
// reads, so that it can be run on the host.
#pragma once
#include <cstdint>

#include "sqc_types.h"

#if defined(__CUDACC__)
#define SQC_MEET __device__ __forceinline__
#define SQC_NO_UNROLL _Pragma("unroll 1")
#else
#define SQC_NO_UNROLL
#define SQC_MEET inline
#endif

namespace sqc {

enum Meet { MEET_OK, MEET_FAILED, MEET_TIMEOUT };

constexpr unsigned kMaxPolls = 1u << 22;     // a few seconds: far longer than any pass of a run
constexpr unsigned kStatusPolls = 64;        // polls between two looks at the status (about 50 us)

// Poll until met() holds; MEET_TIMEOUT after kMaxPolls polls. With LOOK a state whose status says that it
// failed is not waited for (MEET_FAILED): a block that found that status when it began has returned and never
// comes. Only hashed passes can fail within a run (a claim without room), so mapped runs do not look
// (looking: 1000 gates on 2^19 keys, FP32, 2 to 3% slower).
template <bool LOOK, class Met, class Status>
SQC_MEET Meet wait_meeting(Met&& met, Status&& status) {
    if (!LOOK) {
        unsigned left = kMaxPolls;
        while (!met() && --left) {}
        return left ? MEET_OK : MEET_TIMEOUT;
    }
    for (unsigned left = kMaxPolls / kStatusPolls; left; --left) {
        SQC_NO_UNROLL
        for (unsigned k = kStatusPolls; k; --k)   // tight: the time between the last arrival and its notice
            if (met()) return MEET_OK;
        if (status() != ST_OK) return MEET_FAILED;
    }
    return MEET_TIMEOUT;
}

}  // namespace sqc
