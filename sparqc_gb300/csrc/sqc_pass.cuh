// Kernels of single passes and their launchers, shared by the ordinary passes (sqc_pass.cu) and those with a
// gate whose coefficients are not finite (sqc_odd.cu).
#pragma once
#include "sqc_kernels.h"
#include "sqc_unit.cuh"

#include <algorithm>
#include <type_traits>

namespace sqc {

int launch_odd_unit_pass(const PassArgs& a, bool dbl, int sms, cudaStream_t st);
int launch_odd_hash_pass(const PassArgs& a, unsigned long long list_hint, bool dbl, int sms, cudaStream_t st);

namespace {

// Block-reduce the pass counters; the last block to finish publishes the pass (key count,
// list length, empty buckets, pass counter, amp updates, algorithmic bytes). Nothing is
// published when a pass failed.
__device__ void finish_pass(Ctl* ctl, unsigned long long n, unsigned long long e, unsigned long long u,
                            unsigned long long nnz_in, bool keys_fixed, bool pair, unsigned amp_bytes) {
    __shared__ unsigned long long red[3][32];
    __shared__ bool last;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    n = warp_sum(n); e = warp_sum(e); u = warp_sum(u);
    if (lane == 0) { red[0][w] = n; red[1][w] = e; red[2][w] = u; }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long bn = 0, be = 0, bu = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) { bn += red[0][i]; be += red[1][i]; bu += red[2][i]; }
        if (bn) atomicAdd(&ctl->acc_nnz, bn);
        if (be) atomicAdd(&ctl->acc_empty, be);
        if (bu) atomicAdd(&ctl->acc_upd, bu);
        __threadfence();
        const unsigned prev = atomicAdd(&ctl->done, 1u);
        last = prev == gridDim.x - 1;
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        const unsigned long long tn = atomicExch(&ctl->acc_nnz, 0ULL);
        const unsigned long long te = atomicExch(&ctl->acc_empty, 0ULL);
        const unsigned long long tu = atomicExch(&ctl->acc_upd, 0ULL);
        if (*(volatile unsigned int*)&ctl->status == 0) {
            ctl->nnz = tn;
            ctl->empty_groups = te;
            ctl->list_n = *(volatile unsigned long long*)&ctl->list_tail;
            ctl->amp_updates += tu;
            const unsigned long long ab = keys_fixed ? nnz_in * (8ULL + 2ULL * amp_bytes) : (nnz_in + tn) * (8ULL + amp_bytes);
            ctl->alg_bytes += ab;
            if (pair) ctl->alg_bytes_pair += ab;
            ctl->seq += 1;
        }
        ctl->done = 0;
        __threadfence();
    }
}

// True when a pass could leave more groups than a hashed table takes: a unit has 2^nx groups, and a
// pass makes no more than the state has keys after it.
__device__ __forceinline__ bool could_overflow(unsigned long long n, uint32_t nx, unsigned long long grow_bound,
                                               unsigned long long key_bound, unsigned long long max_groups) {
    return nx > 0 && umin64(umin64(grow_bound, n << nx), n + key_bound) > max_groups;
}

// ---- unit pass (mapped tables) ---------------------------------------------------------------
// Units are dealt out round robin to the warps (they cost the same); a table whose live buckets
// are few among the mapped ones is walked by its list instead, 32 entries per warp at a time.
template <class T, int DIMS> struct UnitOcc {
    static constexpr int kMin = sizeof(T) == 4 ? 4 : DIMS == 2 ? 3 : 2;
};

// ODD: a gate of the pass may be UO_ODD.
template <class T, int DIMS, bool ODD>
__global__ void __launch_bounds__(kThreads, ODD ? 2 : UnitOcc<T, DIMS>::kMin) unit_kernel(const __grid_constant__ PassArgs a) {
    __shared__ UGates<T> sg;
    stage_ugates<T>(sg, a.gates, a.g0, a.g1);   // no kernel writes the gates: staged while the previous pass drains
    wait_prior_grid();
    allow_next_grid();
    Ctl* ctl = a.ctl;
    if (*(volatile unsigned int*)&ctl->status) return;
    if ((1ULL << a.dn) > a.max_groups) {   // the mapped bits outgrow the table: refuse before touching the state
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&ctl->status, 0u, (unsigned)ST_GROW);
        return;
    }
    const unsigned long long n = ctl->list_n;
    const unsigned ep = ctl->epoch;
    const unsigned long long nnz_in = ctl->nnz;
    const int lane = threadIdx.x & 31;
    const UnitPass up = unit_pass<DIMS>(a.dn, a.dim[0], a.dim[1], a.dim[2]);
    // the warp's index as one value for the whole warp: unit addresses and control tests are then
    // uniform, as the heads in the parameter bank are
    const unsigned w = blockIdx.x * (kThreads / 32) + __shfl_sync(kFull, threadIdx.x >> 5, 0);
    const unsigned nw = gridDim.x * (kThreads / 32);
    const uint32_t ng = a.g1 - a.g0;
    const GateDesc* gates = a.gates + a.g0;
    unsigned long long cnt_nnz = 0, cnt_empty = 0, upd = 0;
    using Heads = std::conditional_t<ODD, SharedHeads<T, true>, const UnitHead*>;
    Heads heads;
    if constexpr (ODD) heads.g = sg.g;
    else heads = a.heads;
    if (walk_list(n, a.dn)) {
        const unsigned long long piece = list_piece(n, nw);
        for (unsigned long long e0 = w * piece; e0 < n; e0 += nw * piece)
            walk_entries<T, DIMS>(a.t, a.t.map_q, ctl, ep, up, e0, umin64(e0 + piece, n), heads, sg, gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
    } else {
        walk_all_units<T, DIMS>(a.t, a.t.map_q, ctl, ep, up, w, nw, heads, sg, gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
    }
    finish_pass(ctl, cnt_nnz, cnt_empty, upd, nnz_in, a.keys_fixed != 0, a.nx > 0, a.amp_bytes);
}

// ---- pass over a hashed table -----------------------------------------------------------------------
// resident blocks per SM asked for (FP64 at four: 2% slower; FP32 at three: 4% slower)
template <class T> constexpr int kHashBlocks = sizeof(T) == 8 ? 3 : 4;

template <class T, bool ODD>
__global__ void __launch_bounds__(kThreads, ODD ? 2 : kHashBlocks<T>) hash_kernel(const __grid_constant__ PassArgs a) {
    __shared__ HGates<T> sg;
    __shared__ HashWork wk[kThreads / 32];
    const HashDims dm = hash_dims(a.dim[0], a.dim[1]);
    const uint32_t ng = a.g1 - a.g0;
    const GateDesc* gates = a.gates + a.g0;
    stage_hgates<T>(sg, gates, ng, dm.keys);   // no kernel writes the gates: staged while the previous pass drains
    __syncthreads();
    wait_prior_grid();
    allow_next_grid();
    Ctl* ctl = a.ctl;
    if (*(volatile unsigned int*)&ctl->status) return;
    const unsigned long long n = ctl->list_n;
    if (could_overflow(n, a.nx, a.grow_bound, a.key_bound, a.max_groups)) {   // refuse before touching the state
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&ctl->status, 0u, (unsigned)ST_GROW);
        return;
    }
    const unsigned ep = ctl->epoch;
    const unsigned long long nnz_in = ctl->nnz;
    const int lane = threadIdx.x & 31;
    const unsigned wid = __shfl_sync(kFull, threadIdx.x >> 5, 0);
    unsigned long long cnt_nnz = 0, cnt_empty = 0, upd = 0;
    walk_hashed_all<T, ODD>(a.t, ctl, ep, dm, n, wid * gridDim.x + blockIdx.x, gridDim.x * (kThreads / 32), wk[wid], sg, gates, ng,
                             lane, a.prune, cnt_nnz, cnt_empty, upd);
    finish_pass(ctl, cnt_nnz, cnt_empty, upd, nnz_in, a.keys_fixed != 0, a.nx > 0, a.amp_bytes);
}

// A slot pass (walk_slots; S == kLowForm: walk_low). plain: FP64 products by the FP64 instruction. A few warps are not bound by its pipe
// but by fetching code, and the integer products are 20 times as long.
constexpr int kLowForm = 16;
template <class T, int S, bool ODD>
__global__ void __launch_bounds__(kThreads, ODD ? 2 : kHashBlocks<T>) slot_kernel(const __grid_constant__ PassArgs a) {
    __shared__ HGates<T> sg;
    __shared__ SlotWork wk[S == kLowForm ? 1 : kThreads / 32];
    unsigned long long gm[3];
    for (int i = 0; i < 3; ++i) gm[i] = a.dim[i] < 64u ? 1ULL << (a.dim[i] - kSlotBits) : 0ULL;
    const uint32_t ng = a.g1 - a.g0;
    const GateDesc* gates = a.gates + a.g0;
    stage_hgates<T>(sg, gates, ng, S == kLowForm ? 3ULL : (gm[1] | gm[2]) << kSlotBits);   // no kernel writes the gates: staged while the previous pass drains
    if constexpr (sizeof(T) == 8)
        if (a.plain)
            for (uint32_t i = threadIdx.x; i < ng; i += blockDim.x) sg.g[i].exact = 0;   // (the thread's own)
    __syncthreads();
    wait_prior_grid();
    allow_next_grid();
    Ctl* ctl = a.ctl;
    if (*(volatile unsigned int*)&ctl->status) return;
    const unsigned long long n = ctl->list_n;
    if (could_overflow(n, a.nx, a.grow_bound, a.key_bound, a.max_groups)) {   // refuse before touching the state
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&ctl->status, 0u, (unsigned)ST_GROW);
        return;
    }
    const unsigned ep = ctl->epoch;
    const unsigned long long nnz_in = ctl->nnz;
    const int lane = threadIdx.x & 31;
    const unsigned wid = __shfl_sync(kFull, threadIdx.x >> 5, 0), nw = gridDim.x * (kThreads / 32);
    unsigned long long cnt_nnz = 0, cnt_empty = 0, upd = 0;
    unsigned long long piece = list_piece(n, nw);
    if constexpr (S == kLowForm) {
        piece = 8;
        for (unsigned long long e0 = (wid * gridDim.x + blockIdx.x) * piece; e0 < n; e0 += nw * piece)
            walk_low<T, ODD>(a.t, e0, umin64(e0 + piece, n), sg, gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
    } else {
        if (a.nx == 0) piece += piece & 1;   // (at most 32)
        for (unsigned long long e0 = (wid * gridDim.x + blockIdx.x) * piece; e0 < n; e0 += nw * piece)
            walk_slots<T, S, ODD>(a.t, ctl, ep, gm, a.nx, e0, umin64(e0 + piece, n), wk[wid], sg, gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
    }
    finish_pass(ctl, cnt_nnz, cnt_empty, upd, nnz_in, a.keys_fixed != 0, a.nx > 0, a.amp_bytes);
}

template <class K>
int occupancy(K kernel, int threads) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    return per_sm;
}

// Launch a pass with programmatic stream serialization: its blocks may be scheduled once the
// previous kernel in the stream has let them (allow_next_grid), and they wait for that kernel's
// completion in wait_prior_grid before touching the state.
template <class K>
cudaError_t launch_dep(K kernel, int grid, const PassArgs& a, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)kThreads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

// At most one resident wave; below that a warp per `items` (units of a mapped pass, list entries of a
// hashed one).
int grid_of(unsigned long long items, int threads, int sms, int resident) {
    const unsigned long long wave = (unsigned long long)sms * (unsigned long long)resident, per = (unsigned long long)threads / 32;
    return (int)std::max<unsigned long long>(1, std::min(wave, (items + per - 1) / per));
}

template <class T, int DIMS, bool ODD>
cudaError_t launch_unit(const PassArgs& a, int sms, cudaStream_t st) {
    static int resident = 0;
    if (!resident) resident = occupancy(unit_kernel<T, DIMS, ODD>, kThreads);
    return launch_dep(unit_kernel<T, DIMS, ODD>, grid_of(std::max<unsigned long long>(1, (1ULL << a.dn) >> DIMS), kThreads, sms, resident), a, st);
}

template <class T, bool ODD>
cudaError_t launch_hash(const PassArgs& a, unsigned long long list_hint, int sms, cudaStream_t st) {
    static int resident = 0;
    if (!resident) resident = occupancy(hash_kernel<T, ODD>, kThreads);
    return launch_dep(hash_kernel<T, ODD>, grid_of(list_hint, kThreads, sms, resident), a, st);
}

template <bool ODD>
int launch_unit_kernel(const PassArgs& a, bool dbl, int sms, cudaStream_t st) {
    const cudaError_t e = !dbl ? (a.dims == 3 ? launch_unit<float, 3, ODD>(a, sms, st) : launch_unit<float, 2, ODD>(a, sms, st))
                          : a.dims == 3 ? launch_unit<double, 3, ODD>(a, sms, st) : launch_unit<double, 2, ODD>(a, sms, st);
    return e == cudaSuccess ? 1 : -1;
}

template <class T, int S, bool ODD>
cudaError_t launch_slots(const PassArgs& a, unsigned long long list_hint, int sms, cudaStream_t st) {
    static int resident = 0;
    if (!resident) resident = occupancy(slot_kernel<T, S, ODD>, kThreads);
    // a warp per unit, or per two units of one group
    const unsigned long long items = a.nx ? list_hint : (list_hint + 1) / 2;
    PassArgs b = a;
    b.plain = items <= 4ULL * (unsigned long long)sms;   // at most a warp to a scheduler
    return launch_dep(slot_kernel<T, S, ODD>, grid_of(items, kThreads, sms, resident), b, st);
}

template <class T, bool ODD>
cudaError_t launch_slots(const PassArgs& a, unsigned long long list_hint, int sms, cudaStream_t st) {
    if constexpr (sizeof(T) == 4)
        if (a.slots == 2) return launch_slots<T, kLowForm, ODD>(a, (list_hint + 3) / 4, sms, st);
    return a.nx <= 1 ? launch_slots<T, 1, ODD>(a, list_hint, sms, st)
           : a.nx == 2 ? launch_slots<T, 2, ODD>(a, list_hint, sms, st) : launch_slots<T, 4, ODD>(a, list_hint, sms, st);
}

template <bool ODD>
int launch_hash_kernel(const PassArgs& a, unsigned long long list_hint, bool dbl, int sms, cudaStream_t st) {
    const cudaError_t e = a.slots ? (dbl ? launch_slots<double, ODD>(a, list_hint, sms, st) : launch_slots<float, ODD>(a, list_hint, sms, st))
                          : dbl ? launch_hash<double, ODD>(a, list_hint, sms, st) : launch_hash<float, ODD>(a, list_hint, sms, st);
    return e == cudaSuccess ? 1 : -1;
}

}  // namespace
}  // namespace sqc
