// Many-circuit batch: one persistent kernel runs the passes of every circuit of a batch.
//
// Every circuit has its own table slice, control block and gate descriptors, planned on the
// host exactly as for a single state; the unit code (sqc_unit.cuh) is the same, so a circuit's
// result is bit-identical to running it alone (its map is known in advance). Scheduling is per
// circuit: pass p is cut into chunks of units, and a block takes chunk i of pass p with one atomicAdd
// on the circuit's scheduling word (pass, chunks, issued). The block that finishes the last
// chunk of a pass publishes the pass (key count, list length, counters) and opens the next
// one. Circuits never wait for each other, so short and long circuits share the GPU without
// lockstep.
//
// This file is compiled with global loads defaulting to L2 (-dlcm=cg): a persistent kernel
// reads, in pass p + 1, buckets that other SMs wrote in pass p, and L1 is not coherent.
// Gate descriptors and the circuit array never change during a launch.
//
// A block that finds no work sleeps briefly and retries; after idle_limit_ns without work it
// records ST_TIMEOUT in the batch control block and returns (the limit is a batch option,
// 2 s by default); every block returns at its next check of that status. Parking: when the batch has a
// deadline, a circuit whose pass ends after the deadline parks instead of opening its next
// pass; a later launch resumes it (used by the serving loop to admit new circuits).
#include "sqc_batch.h"
#include "sqc_unit.cuh"

namespace sqc {
namespace {

constexpr int kBatchThreads = 256;
constexpr int kBatchWarps = kBatchThreads / 32;
constexpr unsigned kBusyChunks = 64;
constexpr unsigned kIdleSleepNs = 1000;                       // back-off of a warp that found no work

__device__ __forceinline__ unsigned long long sched_word(unsigned long long pass, unsigned long long chunks) {
    return (pass << (2 * kSchedFieldBits)) | (chunks << kSchedFieldBits);
}

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

template <int DIMS>
__device__ __forceinline__ UnitPass units_of(const BPass& p) {
    return unit_pass<DIMS>(p.dn, p.dim[0], p.dim[1], p.dim[2]);
}

// Items of a pass: its units, or the list's entries (walk_list).
template <int DIMS>
__device__ __forceinline__ unsigned long long pass_items(const BPass& p, unsigned long long list_n) {
    if (walk_list(list_n, p.dn)) return list_n;
    return units_of<DIMS>(p).units;
}
__device__ __forceinline__ unsigned long long pass_items(const BPass& p, unsigned long long list_n, bool dbl) {
    return dbl ? pass_items<(int)kBatchDims64>(p, list_n) : pass_items<(int)kBatchDims32>(p, list_n);
}

// Chunking of a pass over n items while `running` circuits share the GPU: items per chunk and the
// chunk count. A pass has at most target_chunks chunks shared among the running circuits. A chunk of units gives
// every warp of its block at least min_chunk / 4 of them, and a pass of units up to kBusyChunks chunks, so that a large
// circuit's passes still spread when many run (256 circuits, FP32: 10.7 ms with the smallest chunks
// for all, 7.3 with four times as many entries). A chunk of list entries, whose units follow one another in a
// warp, is at least min_chunk of them and a warp's share at most 32.
__device__ __forceinline__ void chunking(const BatchArgs& a, unsigned long long n, bool list, unsigned running, unsigned* chunk,
                                         unsigned* total) {
    const unsigned share = a.target_chunks / (running ? running : 1u);
    unsigned long long c;
    if (list) {
        c = share ? (n + share - 1) / share : n;
        if (c > 32u * kBatchWarps) c = 32u * kBatchWarps;
        if (c < a.min_chunk) c = a.min_chunk;
    } else {
        const unsigned target = share > kBusyChunks ? share : kBusyChunks;
        c = (n + target - 1) / target;
        const unsigned least = a.min_chunk / 4 * kBatchWarps;
        if (c < least) c = least;
    }
    *chunk = (unsigned)c;
    const unsigned long long t = (n + c - 1) / c;
    *total = (unsigned)(t ? t : 1);
}

// A chunk in hand: circuit, pass, chunk index, chunks of the pass.
struct Claim {
    unsigned c, p, i, total;
};

// One thread, after the last chunk of pass p of circuit c, with the pass's sums: publish the pass
// and open the next one (or finish / park / fail the circuit). True when the next pass is open:
// its chunk 0 is then *next's, without a search.
__device__ __noinline__ bool finish_circuit_pass(const BatchArgs& a, unsigned c, unsigned p, unsigned long long tn,
                                                 unsigned long long te, unsigned long long tu, Claim* next_claim) {
    const BCirc& C = a.circ[c];
    Ctl* ctl = a.ctl + c;
    BSched* s = a.sched + c;
    const unsigned next = p + 1;
    const unsigned npasses = C.npasses;
    const BPass bp = C.passes[p];
    const BPass nxp = C.passes[next < npasses ? next : p];
    const unsigned long long nnz_in = *(volatile unsigned long long*)&ctl->nnz;
    const unsigned long long n = *(volatile unsigned long long*)&ctl->list_tail;
    const unsigned long long dl = *(volatile unsigned long long*)&a.bctl->deadline_ns;
    const unsigned limit = s->limit;
    const bool ok = *(volatile unsigned int*)&ctl->status == 0;
    if (ok) {
        ctl->nnz = tn;
        ctl->empty_groups = te;
        ctl->list_n = n;
        ctl->amp_updates += tu;
        const unsigned long long A = a.amp_bytes;
        const unsigned long long ab = bp.keys_fixed ? nnz_in * (8ULL + 2ULL * A) : (nnz_in + tn) * (8ULL + A);
        ctl->alg_bytes += ab;
        if (bp.nx) ctl->alg_bytes_pair += ab;
        ctl->seq += 1;
    }
    unsigned state = BS_RUN;
    unsigned chunk = 0, total = 0;
    if (!ok) {
        state = BS_FAILED;
    } else if (next >= npasses) {
        state = BS_DONE;
    } else if ((1ULL << nxp.dn) > C.max_groups) {   // the slice could overflow: stop before touching it
        atomicCAS(&ctl->status, 0u, (unsigned)ST_GROW);
        state = BS_FAILED;
    } else {
        chunking(a, pass_items(nxp, n, a.amp_bytes == 16), walk_list(n, nxp.dn), *(volatile unsigned int*)&a.bctl->left, &chunk, &total);
        if (next >= limit || (dl && globaltimer() > dl)) state = BS_PARKED;
    }
    const bool run = state == BS_RUN;
    s->done = 0;
    s->chunk = chunk;
    s->next_total = total;
    s->state = state;
    __threadfence();
    atomicExch(a.words + c, sched_word(next, run ? total : 0) + (run ? 1u : 0u));   // chunk 0 is taken
    if (!run) atomicSub(&a.bctl->left, 1u);
    atomicAdd(&a.bctl->progress, 1ULL);
    *next_claim = Claim{c, next, 0u, total};
    return run;
}

// Warp 0 of a block: find a chunk, starting at circuit c: the lanes read the scheduling words of
// 128 circuits at a time; the first one with a chunk left is tried with an atomicAdd by its lane.
// Waits, with a pause between searches, until there is a chunk (true) or the launch is over.
__device__ bool find_chunk(const BatchArgs& a, unsigned c, int lane, Claim* out) {
    unsigned long long idle_since = 0;
    while (true) {
        const unsigned status = *(volatile unsigned int*)&a.bctl->status, left = *(volatile unsigned int*)&a.bctl->left;
        for (unsigned base = 0; base < a.n; base += 128) {
            unsigned long long w[4];
            unsigned cc[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const unsigned i = base + 32 * k + lane;
                cc[k] = i < a.n ? (c + i) % a.n : 0;
                w[k] = i < a.n ? *(volatile unsigned long long*)(a.words + cc[k]) : 0ULL;   // 0: no chunks
            }
            if (status || !left) return false;   // (read together with the first words)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unsigned mask = __ballot_sync(kFull, (w[k] & kSchedFieldMask) < ((w[k] >> kSchedFieldBits) & kSchedFieldMask));
                while (mask) {
                    const int l = __ffs(mask) - 1;
                    mask &= mask - 1;
                    unsigned long long old = 0;
                    if (lane == l) old = atomicAdd(a.words + cc[k], 1ULL);
                    old = shfl64(old, l);
                    const unsigned total = (unsigned)((old >> kSchedFieldBits) & kSchedFieldMask);
                    const unsigned i = (unsigned)(old & kSchedFieldMask);
                    if (i < total) {
                        *out = Claim{__shfl_sync(kFull, cc[k], l), (unsigned)(old >> (2 * kSchedFieldBits)), i, total};
                        return true;
                    }
                }
            }
        }
        if (status || !left) return false;
        if (lane == 0) {
            const unsigned long long now = globaltimer();
            if (!idle_since) idle_since = now;
            else if (now - idle_since > a.idle_limit_ns) atomicCAS(&a.bctl->status, 0u, (unsigned)ST_TIMEOUT);
        }
        __syncwarp();
        __nanosleep(kIdleSleepNs);
    }
}

// Blocks take chunks: the gates of a pass are staged once per block, its warps run the same code
// (the instruction cache holds one pass's gates, not one per warp), and the bookkeeping of a chunk
// -- claim, fence, completion -- is paid once for eight warps. A block whose chunk ends a pass goes
// on with the next pass's chunk 0, so a circuit that fits one chunk runs like a tiny state, one
// barrier between passes. (A warp per chunk of two units, each with its own staged copy: 128
// circuits FP32 9.6 ms, 256 circuits FP64 35 ms.)
// MINB: blocks per SM the register allocation is sized for; 1: circuits may have UO_ODD gates.
template <class T, int MINB>
__global__ void __launch_bounds__(kBatchThreads, MINB) batch_run_kernel(BatchArgs a) {
    constexpr int DIMS = (int)(sizeof(T) == 8 ? kBatchDims64 : kBatchDims32);
    __shared__ UGates<T> sg;
    __shared__ Claim claim;
    __shared__ bool have;                      // claim holds a chunk taken with the last publication
    __shared__ bool stop;
    __shared__ unsigned long long sums[3];     // keys, empty buckets, amp updates of the chunk
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned last_c = a.n ? blockIdx.x % a.n : 0;
    unsigned staged_c = ~0u, staged_p = 0;     // the pass in sg
    if (threadIdx.x == 0) have = false;
    __syncthreads();
    while (true) {
        if (w == 0 && !have) {
            Claim got{0, 0, 0, 0};
            const bool ok = find_chunk(a, last_c, lane, &got);
            if (lane == 0) {
                claim = got;
                stop = !ok;
            }
        } else if (threadIdx.x == 0) {
            stop = *(volatile unsigned int*)&a.bctl->status != 0;
        }
        if (threadIdx.x == 0) {
            __threadfence();   // acquire: the previous pass of this circuit is visible
            sums[0] = sums[1] = sums[2] = 0;
        }
        __syncthreads();
        if (stop) return;
        const Claim cl = claim;
        last_c = cl.c;
        const BCirc& C = a.circ[cl.c];
        TableDev t;   // all but the map
        t.hdr = C.t.hdr;
        t.keys = C.t.keys;
        t.amps = C.t.amps;
        t.list = C.t.list;
        t.map_n = C.t.map_n;
        const GateDesc* cgates = C.gates;
        Ctl* ctl = a.ctl + cl.c;
        const BPass bp = C.passes[cl.p];
        const unsigned long long n = *(volatile unsigned long long*)&ctl->list_n;
        const unsigned chunk = *(volatile unsigned int*)&a.sched[cl.c].chunk;
        const unsigned ep = *(volatile unsigned int*)&ctl->epoch;
        if (staged_c != cl.c || staged_p != cl.p) {   // (a circuit's descriptors do not change during a launch)
            stage_ugates<T>(sg, cgates, bp.g0, bp.g1);
            staged_c = cl.c;
            staged_p = cl.p;
        }
        const unsigned long long ib = (unsigned long long)cl.i * chunk, ie = umin64(ib + chunk, pass_items<DIMS>(bp, n));
        const UnitPass up = units_of<DIMS>(bp);
        const GateDesc* gates = cgates + bp.g0;
        const uint32_t ng = bp.g1 - bp.g0;
        unsigned long long cnt_nnz = 0, cnt_empty = 0, upd = 0;
        if (walk_list(n, bp.dn)) {
            const unsigned per = (unsigned)(ie - ib + kBatchWarps - 1) / kBatchWarps;   // as many to every warp
            const unsigned long long we = umin64(ib + (w + 1) * per, ie);
            for (unsigned long long e = ib + w * per; e < we; e += 32)
                walk_entries<T, DIMS>(t, C.t.map_q, ctl, ep, up, e, umin64(e + 32, we), SharedHeads<T, MINB == 1>{sg.g}, sg, gates, ng, lane, a.prune, cnt_nnz, cnt_empty, upd);
        } else {
            walk_units<T, DIMS>(t, C.t.map_q, ctl, ep, up, (unsigned)(ib + w), (unsigned)ie, kBatchWarps, SharedHeads<T, MINB == 1>{sg.g}, sg, gates, ng, lane, a.prune, cnt_nnz,
                             cnt_empty, upd);
        }
        cnt_nnz = warp_sum(cnt_nnz);
        cnt_empty = warp_sum(cnt_empty);
        upd = warp_sum(upd);
        if (lane == 0) {
            if (cnt_nnz) atomicAdd(&sums[0], cnt_nnz);
            if (cnt_empty) atomicAdd(&sums[1], cnt_empty);
            if (upd) atomicAdd(&sums[2], upd);
        }
        __syncthreads();   // the block's writes precede thread 0's fence
        if (threadIdx.x == 0) {
            unsigned long long tn = sums[0], te = sums[1], tu = sums[2];
            bool last = cl.total == 1;
            if (!last) {
                if (tn) atomicAdd(&ctl->acc_nnz, tn);
                if (te) atomicAdd(&ctl->acc_empty, te);
                if (tu) atomicAdd(&ctl->acc_upd, tu);
                __threadfence();   // release: this chunk's writes before its completion
                last = atomicAdd(&a.sched[cl.c].done, 1u) == cl.total - 1;
                if (last) {
                    __threadfence();
                    tn = atomicExch(&ctl->acc_nnz, 0ULL);
                    te = atomicExch(&ctl->acc_empty, 0ULL);
                    tu = atomicExch(&ctl->acc_upd, 0ULL);
                }
            }
            have = last && finish_circuit_pass(a, cl.c, cl.p, tn, te, tu, &claim);
        }
        __syncthreads();
    }
}

// Start a launch: one warp per circuit. BC_INIT resets the circuit to |0...0> under a new
// epoch (all its slice's buckets become free) and opens pass 0; BC_RESUME reopens a parked
// circuit's pending pass; BC_KEEP leaves the circuit as it is. The new epoch is taken from
// the batch control block, so a captured launch sequence replays with fresh epochs.
__global__ void batch_begin_kernel(BatchArgs a, unsigned long long deadline_ns) {
    __shared__ unsigned ep_new;
    __shared__ unsigned running;
    __shared__ unsigned any_init;
    if (threadIdx.x == 0) {
        ep_new = a.bctl->epoch + 1;
        if (ep_new == 0) ep_new = 1;   // epoch 0 marks cleared headers: never a live one
        running = 0;
        any_init = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (unsigned c = w; c < a.n; c += nw) {
        const unsigned cmd = a.cmd[c];
        BSched* s = a.sched + c;
        Ctl* ctl = a.ctl + c;
        const BCirc C = a.circ[c];
        if (cmd == BC_INIT) {
            __shared__ long long sb[32];
            if (lane == 0) {
                any_init = 1;
                ctl->epoch = ep_new;
                ctl->status = 0;
                ctl->done = 0;
                ctl->acc_nnz = ctl->acc_empty = ctl->acc_upd = 0;
                ctl->seq = 0;
                ctl->amp_updates = 0;
                ctl->alg_bytes = 0;
                ctl->alg_bytes_pair = 0;
                ctl->out_count = 0;
                bool created;
                sb[w] = claim_group(C.t, ep_new, 0ULL, &ctl->status, &created);
            }
            __syncwarp();
            const long long b = sb[w];
            if (b >= 0 && lane < kSlots) {
                const size_t sl = (size_t)b * kSlots + lane;
                C.t.keys[sl] = lane == 0 ? 0ULL : empty_key(lane);
                if (lane == 0) {
                    C.t.hdr[b].aux = 1u;   // presence mask: slot 0
                    if (a.amp_bytes == 16) reinterpret_cast<double2*>(C.t.amps)[sl] = make_double2(1.0, 0.0);
                    else reinterpret_cast<float2*>(C.t.amps)[sl] = make_float2(1.0f, 0.0f);
                }
            }
            __syncwarp();
            if (lane == 0) {
                C.t.list[0] = (unsigned)(b >= 0 ? b : 0);
                ctl->list_n = ctl->list_tail = b >= 0 ? 1 : 0;
                ctl->nnz = b >= 0 ? 1 : 0;
                ctl->empty_groups = 0;
                const unsigned lim = a.limit[c];
                s->limit = lim;
                s->done = 0;
                unsigned chunk, total;
                chunking(a, C.npasses ? pass_items(C.passes[0], 1, a.amp_bytes == 16) : 1, C.npasses && walk_list(1, C.passes[0].dn), a.n,
                         &chunk, &total);
                s->chunk = chunk;
                s->next_total = total;
                const bool run = b >= 0 && C.npasses > 0 && lim > 0;
                s->state = run ? BS_RUN : (b >= 0 ? (C.npasses == 0 ? BS_DONE : BS_PARKED) : BS_FAILED);
                a.words[c] = sched_word(0, run ? total : 0);
                if (run) atomicAdd(&running, 1u);
            }
        } else if (cmd == BC_RESUME) {
            if (lane == 0) {
                const unsigned long long w0 = a.words[c];
                const unsigned p = (unsigned)(w0 >> (2 * kSchedFieldBits));
                s->limit = a.limit[c];
                if (s->state == BS_PARKED && p < s->limit && ctl->status == 0) {
                    s->state = BS_RUN;
                    s->done = 0;
                    a.words[c] = sched_word(p, s->next_total);
                    atomicAdd(&running, 1u);
                }
            }
        } else if (lane == 0 && s->state == BS_RUN) {
            atomicAdd(&running, 1u);   // kept running circuits still count
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (any_init) a.bctl->epoch = ep_new;
        a.bctl->status = 0;
        a.bctl->left = running;
        a.bctl->deadline_ns = deadline_ns ? globaltimer() + deadline_ns : 0ULL;
        a.bctl->progress = 0;
    }
}

}  // namespace

template <class T, int MINB>
int batch_occupancy() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_run_kernel<T, MINB>, kBatchThreads, 0);
    return n > 0 ? n : 1;
}

template <class T, int MINB>
cudaError_t launch_run(const BatchArgs& a, int grid, cudaStream_t st) {
    batch_run_kernel<T, MINB><<<grid, kBatchThreads, 0, st>>>(a);
    return cudaGetLastError();
}

// Blocks per SM that fit for the variant a launch of `blocks_per_sm` (0: most) would use.
int batch_residency(bool dbl, int blocks_per_sm) {
    static int cache[2][2] = {{0, 0}, {0, 0}};
    const int v = blocks_per_sm == 0 || blocks_per_sm >= 3 ? 1 : 0;
    int& c = cache[dbl ? 1 : 0][v];
    if (!c) c = dbl ? (v ? batch_occupancy<double, 3>() : batch_occupancy<double, 2>())
                    : (v ? batch_occupancy<float, 3>() : batch_occupancy<float, 2>());
    return c;
}

cudaError_t launch_batch(const BatchArgs& a, bool dbl, int grid, int blocks_per_sm, bool odd, unsigned long long deadline_ns,
                         cudaStream_t st) {
    batch_begin_kernel<<<1, 1024, 0, st>>>(a, deadline_ns);
    if (odd) return dbl ? launch_run<double, 1>(a, grid, st) : launch_run<float, 1>(a, grid, st);
    const bool v3 = blocks_per_sm == 0 || blocks_per_sm >= 3;
    if (dbl) return v3 ? launch_run<double, 3>(a, grid, st) : launch_run<double, 2>(a, grid, st);
    return v3 ? launch_run<float, 3>(a, grid, st) : launch_run<float, 2>(a, grid, st);
}

}  // namespace sqc
