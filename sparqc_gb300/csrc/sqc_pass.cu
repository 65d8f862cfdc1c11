// Gate-pass kernels of the sparse statevector engine (sm_103a).
//
// A gate pass updates the table in place: a run of gates that pair keys across at most two (FP64) or
// three (FP32) cross-group qubits, besides qubits 0..3, whose partners share a bucket. Its units
// (sqc_unit.cuh) are enumerated by address in a mapped table and found through the list of live
// buckets in a hashed one; a group that appears for the first time is claimed and appended to the list
// (such groups are beyond the entries the pass walks). Pruning follows the reference
// (emulator/device/device_data.cuh:108-156): branching gates drop negligible outputs, swap
// and diagonal gates keep every key.
#include "sqc_meet.h"
#include "sqc_pass.cuh"

namespace sqc {

namespace {

// ---- a run of unit passes in one launch ----------------------------------------------------------
// Small and middle states spend most of a pass on its edges: a launch of its own waits for the
// previous pass's last block, publishes the pass through three dependent atomics and reads its
// gates and the control block before the first unit. A run keeps its blocks for all its passes
// (a cooperative launch: every block is resident) and meets at a counter between them, with the
// next pass's gates staged while it waits. All that a pass publishes is linear in its counts, so each thread adds
// its own up and the last block to finish publishes the whole run. Mapped passes never refuse here
// (the host ends a run before one that would); a hashed pass that could overflow the table ends
// the run before it, on every block alike.
struct ParamHeads {   // the heads in the parameter bank from word o on
    const RunArgs& a;
    uint32_t o;
    __device__ __forceinline__ UnitHead operator[](uint32_t i) const { return a.words[o + i]; }
};

__device__ __forceinline__ HashDims run_dims(const RunArgs& a, uint32_t o) {
    return hash_dims(a.words[o].ov & 0xFFu, (a.words[o].ov >> 8) & 0xFFu);
}

template <class T>
__device__ __forceinline__ void stage_run(HGates<T>& sg, const RunArgs& a, uint32_t o) {
    stage_hgates<T>(sg, a.gates + a.words[o].loc, a.words[o].om & 0xFFu, run_dims(a, o).keys);
}

template <class T>
__device__ __forceinline__ void stage_run(UGates<T>& sg, const RunArgs& a, uint32_t o) {
    const uint32_t ng = a.words[o].om & 0xFFu;
    const GateDesc* gates = a.gates + a.words[o].loc;
    for (uint32_t i = threadIdx.x; i < ng; i += blockDim.x) stage_ugate(sg.g + i, gates + i);
    for (uint32_t i = threadIdx.x; i < ng * 32u; i += blockDim.x)
        sg.lw[i >> 5][i & 31u] = short_word(lane_word(a.words[o + 1 + (i >> 5)].loc, i & 31u));
}

template <class T, bool HASHED> struct RunGates { using G = UGates<T>; };
template <class T> struct RunGates<T, true> { using G = HGates<T>; };

template <class T, int DIMS, bool HASHED>
__global__ void __launch_bounds__(kThreads, HASHED ? kHashBlocks<T> : UnitOcc<T, DIMS>::kMin) run_kernel(const __grid_constant__ RunArgs a) {
    __shared__ typename RunGates<T, HASHED>::G sg[2];
    __shared__ HashWork wk[HASHED ? kThreads / 32 : 1];
    __shared__ unsigned long long acc[3][kThreads];   // each thread's own: amp updates, bytes, bytes of pair passes
    __shared__ unsigned long long red[5], n_sh;
    __shared__ int stop, last;
    Ctl* ctl = a.ctl;
    if (*(volatile unsigned int*)&ctl->status) return;
    const unsigned ep = ctl->epoch;
    unsigned long long n = *(volatile unsigned long long*)&ctl->list_n;   // live buckets, at least
    const unsigned long long moved = 8ULL + a.amp_bytes, fixed = 8ULL + 2ULL * a.amp_bytes;
    {
        const uint32_t f = a.words[0].om;
        const unsigned long long in = blockIdx.x == 0 && threadIdx.x == 0 ? *(volatile unsigned long long*)&ctl->nnz : 0;
        acc[0][threadIdx.x] = 0;
        acc[1][threadIdx.x] = in * (f & kRunFixed ? fixed : moved);
        acc[2][threadIdx.x] = f & kRunPair ? in * (f & kRunFixed ? fixed : moved) : 0;
        if (threadIdx.x < 5) red[threadIdx.x] = 0;
        if (threadIdx.x == 0) stop = 0;
    }
    const int lane = threadIdx.x & 31;
    // a pass of fewer units than warps spreads them over the blocks
    const unsigned wid = __shfl_sync(kFull, threadIdx.x >> 5, 0), w = wid * gridDim.x + blockIdx.x;
    const unsigned nw = gridDim.x * (blockDim.x >> 5);
    stage_run<T>(sg[0], a, 0);
    __syncthreads();
    uint32_t o = 0;
    unsigned long long cnt_nnz = 0, cnt_empty = 0;
    uint32_t p = 0;
    bool refused = false;
    for (;; ++p) {
        const UnitHead rec = a.words[o];
        const uint32_t ng = rec.om & 0xFFu;
        const GateDesc* gates = a.gates + rec.loc;
        unsigned long long upd = 0;
        if constexpr (HASHED) {
            const ulonglong2 bound = *reinterpret_cast<const ulonglong2*>(&a.words[o + 1]);
            if (could_overflow(n, rec.om >> 16, bound.x, bound.y, a.max_groups)) {   // before touching the state
                refused = true;
                break;
            }
            cnt_nnz = cnt_empty = 0;
            walk_hashed_all<T>(a.t, ctl, ep, run_dims(a, o), n, w, nw, wk[wid], sg[p & 1], gates, ng, lane, a.prune,
                                     cnt_nnz, cnt_empty, upd);
            o += 2;
        } else {
            const uint32_t dn = rec.om >> 16;
            const UnitPass up = unit_pass<DIMS>(dn, rec.ov & 0xFFu, (rec.ov >> 8) & 0xFFu, (rec.ov >> 16) & 0xFFu);
            const ParamHeads heads{a, o + 1};
            cnt_nnz = cnt_empty = 0;
            if (walk_list(n, dn)) {
                const unsigned long long piece = list_piece(n, nw);
                for (unsigned long long e0 = w * piece; e0 < n; e0 += nw * piece)
                    walk_entries<T, DIMS>(a.t, a.t.map_q, ctl, ep, up, e0, umin64(e0 + piece, n), heads, sg[p & 1], gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
            } else {
                // (FP32 runs have four rounds at most, and no registers to spare for turning the deal)
                if constexpr (sizeof(T) == 4)
                    walk_units<T, DIMS>(a.t, a.t.map_q, ctl, ep, up, w, up.units, nw, heads, sg[p & 1], gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
                else
                    walk_all_units<T, DIMS>(a.t, a.t.map_q, ctl, ep, up, w, nw, heads, sg[p & 1], gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
            }
            o += 1 + ng;
        }
        const bool end = p + 1 == a.np;
        const uint32_t f = rec.om, g = end ? 0u : a.words[o].om;
        const unsigned long long out = f & kRunFixed ? 0 : moved, in = end ? 0 : g & kRunFixed ? fixed : moved;
        acc[0][threadIdx.x] += upd;
        acc[1][threadIdx.x] += cnt_nnz * (out + in);
        acc[2][threadIdx.x] += cnt_nnz * ((f & kRunPair ? out : 0) + (g & kRunPair ? in : 0));
        if (end) break;
        // every block's pass is done before any block's next one; whether the next pass walks the list
        // (and needs its exact length; a hashed one always does) follows from what every block knows
        const bool list = HASHED || walk_list(n, g >> 16);
        const uint32_t tag = p + 1;
        __syncthreads();
        if (gridDim.x == 1) {
            if (threadIdx.x == 0 && list) n_sh = *(volatile unsigned long long*)&ctl->list_tail;
            stage_run<T>(sg[(p + 1) & 1], a, o);
        } else {
            if (threadIdx.x == 0) {
                __threadfence();
                const unsigned prev = atomicAdd(&ctl->bar, 1u);
                if (list && prev + 1 == gridDim.x * (p + 1)) {   // all are here and none goes on: the length is exact
                    __threadfence();
                    const unsigned long long len = *(volatile unsigned long long*)&ctl->list_tail;
                    atomicExch(&ctl->bar_len, ((unsigned long long)tag << 32) | len);
                }
            }
            stage_run<T>(sg[(p + 1) & 1], a, o);
            if (threadIdx.x == 0) {
                auto status = [&] { return *(volatile unsigned int*)&ctl->status; };
                Meet met;
                if (list) {
                    unsigned long long v;
                    met = wait_meeting<HASHED>([&] { return (uint32_t)((v = *(volatile unsigned long long*)&ctl->bar_len) >> 32) == tag; }, status);
                    n_sh = v & 0xFFFFFFFFULL;
                } else {
                    met = wait_meeting<HASHED>([&] { return *(volatile unsigned int*)&ctl->bar >= gridDim.x * (p + 1); }, status);
                }
                if (met == MEET_TIMEOUT) atomicCAS(&ctl->status, 0u, (unsigned)ST_TIMEOUT);
                stop = met != MEET_OK;
                __threadfence();
            }
        }
        __syncthreads();
        if (stop) return;
        if (list) n = n_sh;
    }
    if (refused) {
        // take back what the passes before counted for the refused one's input
        const uint32_t f = a.words[o].om;
        const unsigned long long in = f & kRunFixed ? fixed : moved;
        if (p == 0) {   // nothing ran
            if (blockIdx.x == 0 && threadIdx.x == 0) atomicCAS(&ctl->status, 0u, (unsigned)ST_GROW);
            return;
        }
        acc[1][threadIdx.x] -= cnt_nnz * in;
        if (f & kRunPair) acc[2][threadIdx.x] -= cnt_nnz * in;
    }
    // publish the passes that ran; p blocks' meetings lie behind, and this one is the last
    const uint32_t ran = refused ? p : p + 1;
    const unsigned long long v[5] = {warp_sum(cnt_nnz), warp_sum(cnt_empty), warp_sum(acc[0][threadIdx.x]),
                                     warp_sum(acc[1][threadIdx.x]), warp_sum(acc[2][threadIdx.x])};
    if (lane == 0)
#pragma unroll
        for (int i = 0; i < 5; ++i)
            if (v[i]) atomicAdd(&red[i], v[i]);
    __syncthreads();
    if (threadIdx.x == 0) {
        if (red[0]) atomicAdd(&ctl->acc_nnz, red[0]);
        if (red[1]) atomicAdd(&ctl->acc_empty, red[1]);
        if (red[2]) atomicAdd(&ctl->amp_updates, red[2]);
        if (red[3]) atomicAdd(&ctl->alg_bytes, red[3]);
        if (red[4]) atomicAdd(&ctl->alg_bytes_pair, red[4]);
        __threadfence();
        last = atomicAdd(&ctl->bar, 1u) + 1 == gridDim.x * (gridDim.x == 1 ? 1u : p + 1);
        if (last) {
            __threadfence();
            const unsigned long long tn = atomicExch(&ctl->acc_nnz, 0ULL), te = atomicExch(&ctl->acc_empty, 0ULL);
            if (*(volatile unsigned int*)&ctl->status == 0) {
                ctl->nnz = tn;
                ctl->empty_groups = te;
                ctl->list_n = *(volatile unsigned long long*)&ctl->list_tail;
                ctl->seq += ran;
                if (refused) ctl->status = ST_GROW;
            }
            ctl->bar = 0;
            ctl->bar_len = 0;   // (a recorded run may come again)
            __threadfence();
        }
    }
}

// A run's blocks: a warp per item of its largest pass, at most one resident wave. Few items get blocks
// of four warps, one for each scheduler of an SM, on more SMs.
template <class T, int DIMS, bool HASHED>
cudaError_t launch_run(const RunArgs& a, unsigned long long items, int sms, cudaStream_t st) {
    static int resident = 0;
    if (!resident) resident = occupancy(run_kernel<T, DIMS, HASHED>, kThreads);
    const int threads = items <= 4ULL * (unsigned long long)sms ? 128 : kThreads;
    const int grid = grid_of(items, threads, sms, resident);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = grid > 1 ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, run_kernel<T, DIMS, HASHED>, a);
}

}  // namespace

int launch_unit_pass(const PassArgs& a, bool dbl, int sms, cudaStream_t st) {
    if (a.odd) return launch_odd_unit_pass(a, dbl, sms, st);
    return launch_unit_kernel<false>(a, dbl, sms, st);
}

int launch_hash_pass(const PassArgs& a, unsigned long long list_hint, bool dbl, int sms, cudaStream_t st) {
    if (a.odd) return launch_odd_hash_pass(a, list_hint, dbl, sms, st);
    return launch_hash_kernel<false>(a, list_hint, dbl, sms, st);
}

int launch_run_passes(const RunArgs& a, uint32_t dims, unsigned long long items, bool dbl, int sms, cudaStream_t st) {
    cudaError_t e;
    if (a.t.map_on)
        e = !dbl ? (dims == 3 ? launch_run<float, 3, false>(a, items, sms, st) : launch_run<float, 2, false>(a, items, sms, st))
            : dims == 3 ? launch_run<double, 3, false>(a, items, sms, st) : launch_run<double, 2, false>(a, items, sms, st);
    else
        e = dbl ? launch_run<double, 2, true>(a, items, sms, st) : launch_run<float, 2, true>(a, items, sms, st);
    return e == cudaSuccess ? 1 : -1;
}

}  // namespace sqc
