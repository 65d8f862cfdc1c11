// Bookkeeping kernels of the sparse statevector engine (sm_103a): reset, loading a state,
// counting, readout, norm, state comparison and table rebuild. All walk the list of live
// buckets. The gate passes are in sqc_pass.cu.
#include "sqc_kernels.h"
#include "sqc_exact.cuh"

#include <algorithm>

namespace sqc {

namespace {

template <class T> struct AmpT;
template <> struct AmpT<double> { using V = double2; };
template <> struct AmpT<float> { using V = float2; };

template <class T>
__device__ __forceinline__ Cx<T> load_amp(const void* amps, size_t s) {
    const typename AmpT<T>::V v = reinterpret_cast<const typename AmpT<T>::V*>(amps)[s];
    return Cx<T>{v.x, v.y};
}
__device__ __forceinline__ Cx<double> load_amp_any(const void* amps, size_t s, bool dbl) {
    if (dbl) { const double2 v = reinterpret_cast<const double2*>(amps)[s]; return Cx<double>{v.x, v.y}; }
    const float2 v = reinterpret_cast<const float2*>(amps)[s];
    return Cx<double>{(double)v.x, (double)v.y};
}

__device__ __forceinline__ bool slot_present(unsigned long long key, int j) { return (int)(key & 15ULL) == j; }

// |0...0>: new epoch (every bucket becomes free), claim group 0, store key 0 with amplitude 1.
__global__ void set_zero_kernel(TableDev t, Ctl* ctl, int dbl) {
    const int lane = threadIdx.x;
    __shared__ long long sb;
    if (lane == 0) {
        ctl->epoch += 1;
        ctl->status = 0;
        ctl->done = 0;
        ctl->bar = 0;
        ctl->bar_len = 0;
        ctl->acc_nnz = ctl->acc_empty = ctl->acc_upd = 0;
        ctl->seq = 0;
        ctl->amp_updates = 0;
        ctl->alg_bytes = 0;
        ctl->alg_bytes_pair = 0;
        bool created;
        sb = claim_group(t, ctl->epoch, 0ULL, &ctl->status, &created);
    }
    __syncwarp();
    const long long b = sb;
    if (b >= 0 && lane < kSlots) {
        const size_t s = (size_t)b * kSlots + lane;
        t.keys[s] = lane == 0 ? 0ULL : empty_key(lane);
        if (lane == 0) {
            t.hdr[b].aux = 1u;   // presence mask: slot 0
            if (dbl) reinterpret_cast<double2*>(t.amps)[s] = make_double2(1.0, 0.0);
            else reinterpret_cast<float2*>(t.amps)[s] = make_float2(1.0f, 0.0f);
        }
    }
    __syncwarp();
    if (lane == 0) {
        t.list[0] = (unsigned)(b >= 0 ? b : 0);
        ctl->list_n = ctl->list_tail = b >= 0 ? 1 : 0;
        ctl->nnz = b >= 0 ? 1 : 0;
        ctl->empty_groups = 0;
    }
}

// set_state step 0: new epoch, counters reset (one thread).
__global__ void set_state_begin_kernel(Ctl* ctl) {
    ctl->epoch += 1;
    ctl->status = 0;
    ctl->done = 0;
    ctl->bar = 0;
    ctl->bar_len = 0;
    ctl->acc_nnz = ctl->acc_empty = ctl->acc_upd = 0;
    ctl->seq = 0;
    ctl->amp_updates = 0;
    ctl->alg_bytes = 0;
    ctl->alg_bytes_pair = 0;
    ctl->out_count = 0;
    ctl->list_n = ctl->list_tail = 0;
    ctl->nnz = 0;
    ctl->empty_groups = 0;
}

// set_state step 1: claim the bucket of every entry's group; the claimer appends it to the list.
__global__ void set_state_claim_kernel(const unsigned long long* __restrict__ keys, unsigned long long n,
                                       unsigned long long frame, TableDev t, Ctl* ctl) {
    const unsigned ep = ctl->epoch;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        bool created;
        const long long b = claim_group(t, ep, (keys[i] ^ frame) >> kSlotBits, &ctl->status, &created);
        if (created) t.list[atomicAdd(&ctl->list_tail, 1ULL)] = (unsigned)b;
    }
}

// set_state step 2: mark every slot of every listed bucket empty.
__global__ void set_state_clear_kernel(TableDev t, Ctl* ctl) {
    const unsigned long long n = ctl->list_tail;
    for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < n * kSlots;
         s += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned b = t.list[s >> kSlotBits];
        t.keys[(size_t)b * kSlots + (s & 15)] = empty_key((int)(s & 15));
    }
}

// set_state step 3: store every entry in its slot and mark it present; a slot marked twice is a duplicate
// key.
__global__ void set_state_fill_kernel(const unsigned long long* __restrict__ keys, const double* __restrict__ re,
                                      const double* __restrict__ im, unsigned long long n,
                                      unsigned long long frame, TableDev t, Ctl* ctl, int dbl) {
    const unsigned ep = ctl->epoch;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i] ^ frame;
        const long long b = lookup_group(t, ep, k >> kSlotBits);
        if (b < 0) { atomicCAS(&ctl->status, 0u, (unsigned)ST_TABLE_FULL); continue; }
        const int j = (int)(k & 15ULL);
        const size_t s = (size_t)b * kSlots + j;
        if ((atomicOr(&t.hdr[b].aux, 1u << j) >> j) & 1u) { atomicCAS(&ctl->status, 0u, (unsigned)ST_DUPLICATE); continue; }
        t.keys[s] = k;
        if (dbl) reinterpret_cast<double2*>(t.amps)[s] = make_double2(re[i], im[i]);
        else reinterpret_cast<float2*>(t.amps)[s] = make_float2((float)re[i], (float)im[i]);
    }
}

// set_state step 4 (one thread): commit the list.
__global__ void set_state_end_kernel(Ctl* ctl, unsigned long long n) {
    ctl->list_n = ctl->list_tail;
    ctl->nnz = n;
}

// Presence masks of a table's listed buckets, from their keys (a half-warp per bucket).
__global__ void refresh_masks_kernel(TableDev t, Ctl* ctl) {
    const unsigned long long n = ctl->list_tail;
    const int lane = threadIdx.x & 31, j = lane & 15;
    const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    for (unsigned long long e0 = warp * 2; e0 < n; e0 += nwarps * 2) {
        const unsigned long long e = e0 + (lane >> 4);
        const unsigned b = e < n ? t.list[e] : 0u;
        const bool p = e < n && slot_present(t.keys[(size_t)b * kSlots + j], j);
        const unsigned bal = __ballot_sync(kFull, p);
        if (e < n && j == 0) t.hdr[b].aux = lane >= 16 ? bal >> 16 : bal & 0xFFFFu;
    }
}

// Compact the present entries whose stored key matches (key & smask) == sval into
// (keys ^ frame, re, im). A lane takes a list entry and reads its presence mask; the warp's present
// slots are then dealt to its lanes, 32 at a time, so that thin buckets cost no more than their
// keys. Entries beyond cap are counted but not written. (608 keys: 33 -> 3 us, a million 274 -> 146; before,
// half-warps read every bucket's keys twice.)
template <class T>
__global__ void readout_kernel(TableDev t, Ctl* ctl, unsigned long long frame, unsigned long long* okeys,
                               double* ore, double* oim, unsigned long long cap, int drop_negl, PruneBits pb,
                               unsigned long long smask, unsigned long long sval) {
    __shared__ unsigned short slots[kThreads / 32][32 * kSlots];
    const unsigned long long n = ctl->list_n;
    const int lane = threadIdx.x & 31;
    unsigned short* mine = slots[threadIdx.x >> 5];
    unsigned low = 0;   // slots that match in the low bits
    for (unsigned j = 0; j < (unsigned)kSlots; ++j) low |= (j & (unsigned)smask & 15u) == ((unsigned)sval & 15u) ? 1u << j : 0u;
    const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    for (unsigned long long e0 = warp * 32; e0 < n; e0 += nwarps * 32) {
        unsigned b = 0, m = 0;
        unsigned long long G = 0;
        if (e0 + lane < n) {
            b = t.list[e0 + lane];
            const Header h = load_hdr(t.hdr + b);
            G = h.group;
            if ((G & (smask >> kSlotBits)) == (sval >> kSlotBits)) m = h.aux & low;
        }
        unsigned upto = __popc(m);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(kFull, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned total = __shfl_sync(kFull, upto, 31);
        if (!total) continue;
        unsigned at = upto - __popc(m);
        for (unsigned c = m; c; c &= c - 1) mine[at++] = (unsigned short)((lane << 4) | (__ffs(c) - 1));
        __syncwarp();
        unsigned long long base = 0;
        if (lane == 0 && !drop_negl) base = atomicAdd(&ctl->out_count, (unsigned long long)total);
        for (unsigned c0 = 0; c0 < total; c0 += 32) {
            const bool on = c0 + lane < total;
            const unsigned id = on ? mine[c0 + lane] : 0u;
            const unsigned bk = __shfl_sync(kFull, b, (int)(id >> 4));
            const unsigned long long key = (shfl64(G, (int)(id >> 4)) << kSlotBits) | (id & 15u);
            Cx<T> v{T(0), T(0)};
            if (on) v = load_amp<T>(t.amps, (size_t)bk * kSlots + (id & 15u));
            const unsigned keep = __ballot_sync(kFull, on && !(drop_negl && negligible(v, pb)));
            if (lane == 0 && drop_negl && keep) base = atomicAdd(&ctl->out_count, (unsigned long long)__popc(keep));
            const unsigned long long to = shfl64(base, 0) + (drop_negl ? 0u : c0) + __popc(keep & ((1u << lane) - 1u));
            if (((keep >> lane) & 1u) && to < cap) {
                okeys[to] = key ^ frame;
                ore[to] = (double)v.r;
                oim[to] = (double)v.i;
            }
        }
        __syncwarp();
    }
}

// Sum of |a|^2 over the state, exactly (sqc_exact.cuh), into sums->c[SUM_NORM].
template <class T>
__global__ void norm_kernel(TableDev t, Ctl* ctl, ExactSums* sums) {
    const unsigned long long n = ctl->list_n;
    unsigned long long acc[kSumChunks] = {};
    for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < n * kSlots;
         s += (unsigned long long)gridDim.x * blockDim.x) {
        const size_t slot = (size_t)t.list[s >> kSlotBits] * kSlots + (s & 15);
        if (!slot_present(t.keys[slot], (int)(s & 15))) continue;
        const Cx<T> v = load_amp<T>(t.amps, slot);
        const double r = (double)v.r, i = (double)v.i;
        exact_add_prod(acc, r, r);
        exact_add_prod(acc, i, i);
    }
    exact_flush(acc, sums->c[SUM_NORM]);
}

__device__ __forceinline__ void atomic_max_nonneg(unsigned long long* p, double v) {
    atomicMax(p, (unsigned long long)__double_as_longlong(v));
}

// Amplitude of the key stored as sb in state B, if present.
__device__ __forceinline__ bool find_other(const TableDev& tb, unsigned ep_b, unsigned long long sb, bool dbl_b,
                                           Cx<double>* out) {
    const long long bb = lookup_group(tb, ep_b, sb >> kSlotBits);
    if (bb < 0) return false;
    const int j = (int)(sb & 15ULL);
    const size_t s = (size_t)bb * kSlots + j;
    if (!slot_present(tb.keys[s], j)) return false;
    *out = load_amp_any(tb.amps, s, dbl_b);
    return true;
}

// Over the keys of a, exactly (sqc_exact.cuh): PART 0 sums conj(b)*a (real part into
// SUM_ORE, imaginary into SUM_OIM), PART 1 sums |a|^2 (SUM_NA) and |b|^2 (SUM_NB) and takes the
// max |a-b| (a max does not depend on the order). Two accumulators per launch keep the
// registers in check. d = frame_a ^ frame_b translates a stored key of a into b's frame.
template <int PART>
__global__ void compare_a_kernel(TableDev ta, const Ctl* ca, int dbl_a, TableDev tb, const Ctl* cb, int dbl_b,
                                 unsigned long long d, Ctl* out, ExactSums* sums) {
    const unsigned long long n = ca->list_n;
    const unsigned ep_b = cb->epoch;
    unsigned long long s0[kSumChunks] = {}, s1[kSumChunks] = {};
    double mx = 0;
    for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < n * kSlots;
         s += (unsigned long long)gridDim.x * blockDim.x) {
        const size_t slot = (size_t)ta.list[s >> kSlotBits] * kSlots + (s & 15);
        const unsigned long long key = ta.keys[slot];
        if (!slot_present(key, (int)(s & 15))) continue;
        const Cx<double> va = load_amp_any(ta.amps, slot, dbl_a);
        Cx<double> vb{0.0, 0.0};
        find_other(tb, ep_b, key ^ d, dbl_b, &vb);
        if (PART == 0) {
            exact_add_prod(s0, vb.r, va.r);
            exact_add_prod(s0, vb.i, va.i);
            exact_add_prod(s1, vb.r, va.i);
            exact_add_prod(s1, -vb.i, va.r);
        } else {
            exact_add_prod(s0, va.r, va.r);
            exact_add_prod(s0, va.i, va.i);
            exact_add_prod(s1, vb.r, vb.r);
            exact_add_prod(s1, vb.i, vb.i);
            const double dr = va.r - vb.r, di = va.i - vb.i;
            mx = fmax(mx, sqrt(dr * dr + di * di));
        }
    }
    exact_flush(s0, sums->c[PART == 0 ? SUM_ORE : SUM_NA]);
    exact_flush(s1, sums->c[PART == 0 ? SUM_OIM : SUM_NB]);
    if (PART == 1) {
        for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_down_sync(kFull, mx, o));
        if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&out->acc_max, mx);
    }
}

// Keys of b absent from a: SUM_NB_ONLY += |b|^2 (exactly), max |b|.
__global__ void compare_b_kernel(TableDev ta, const Ctl* ca, TableDev tb, const Ctl* cb, int dbl_b,
                                 unsigned long long d, Ctl* out, ExactSums* sums) {
    const unsigned long long n = cb->list_n;
    const unsigned ep_a = ca->epoch;
    unsigned long long s0[kSumChunks] = {};
    double mx = 0;
    for (unsigned long long s = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; s < n * kSlots;
         s += (unsigned long long)gridDim.x * blockDim.x) {
        const size_t slot = (size_t)tb.list[s >> kSlotBits] * kSlots + (s & 15);
        const unsigned long long key = tb.keys[slot];
        if (!slot_present(key, (int)(s & 15))) continue;
        Cx<double> dummy;
        if (find_other(ta, ep_a, key ^ d, true, &dummy)) continue;
        const Cx<double> vb = load_amp_any(tb.amps, slot, dbl_b);
        exact_add_prod(s0, vb.r, vb.r);
        exact_add_prod(s0, vb.i, vb.i);
        mx = fmax(mx, sqrt(vb.r * vb.r + vb.i * vb.i));
    }
    exact_flush(s0, sums->c[SUM_NB_ONLY]);
    for (int o = 16; o; o >>= 1) mx = fmax(mx, __shfl_down_sync(kFull, mx, o));
    if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&out->acc_max, mx);
}

// Copy the live, non-empty buckets of the old table into a new one (fresh headers, epoch
// ep_new), rebuilding the list. Each group appears once, so each new bucket has one writer.
__global__ void rehash_kernel(TableDev told, unsigned long long n_old, TableDev tnew, unsigned ep_new,
                              int amp_bytes, Ctl* ctl) {
    const int lane = threadIdx.x & 31, j = lane & 15, half = lane >> 4;
    const unsigned long long warp = ((unsigned long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned long long nwarps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    // a lane claims for its entry, all claims of the warp together; the buckets are then copied by
    // half-warps (a half-warp that claimed for its own bucket waited for each claim alone: a million
    // keys 1.2 ms, now 0.48)
    for (unsigned long long e0 = warp * 32; e0 < n_old; e0 += nwarps * 32) {
        unsigned b = 0;
        Header h;
        h.group = 0;
        h.aux = 0;
        if (e0 + lane < n_old) {
            b = told.list[e0 + lane];
            h = load_hdr(told.hdr + b);
        }
        unsigned to = kNoBucket;
        if (h.aux != 0) {
            bool created;
            const long long nb = claim_group(tnew, ep_new, h.group, &ctl->status, &created);
            if (nb >= 0) {
                to = (unsigned)nb;
                tnew.hdr[to].aux = h.aux;
            }
        }
        const unsigned fm = __ballot_sync(kFull, to != kNoBucket);
        if (!fm) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&ctl->list_tail, (unsigned long long)__popc(fm));
        base = shfl64(base, 0);
        if (to != kNoBucket) tnew.list[base + __popc(fm & ((1u << lane) - 1u))] = to;
#pragma unroll 4
        for (int i = 0; i < 32; i += 2) {
            const int l = i + half;
            const unsigned from = __shfl_sync(kFull, b, l), d = __shfl_sync(kFull, to, l), mine = __shfl_sync(kFull, h.aux, l);
            const unsigned long long G = shfl64(h.group, l);
            if (d == kNoBucket) continue;
            const bool p = (mine >> j) & 1u;
            const size_t src = (size_t)from * kSlots + j, dst = (size_t)d * kSlots + j;
            tnew.keys[dst] = p ? (G << kSlotBits) | (unsigned)j : empty_key(j);
            if (!p) continue;
            if (amp_bytes == 16) reinterpret_cast<double2*>(tnew.amps)[dst] = reinterpret_cast<const double2*>(told.amps)[src];
            else reinterpret_cast<float2*>(tnew.amps)[dst] = reinterpret_cast<const float2*>(told.amps)[src];
        }
    }
}

int grid_for(unsigned long long work_items, int per_block, int sms) {
    unsigned long long g = (work_items + per_block - 1) / per_block;
    const unsigned long long cap = (unsigned long long)sms * 4;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

cudaError_t launch_set_zero(const TableDev& t, Ctl* ctl, bool dbl, cudaStream_t st) {
    set_zero_kernel<<<1, 32, 0, st>>>(t, ctl, dbl ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_set_state(const unsigned long long* keys, const double* re, const double* im,
                             unsigned long long n, unsigned long long frame, const TableDev& t, Ctl* ctl, bool dbl,
                             int sms, cudaStream_t st) {
    set_state_begin_kernel<<<1, 1, 0, st>>>(ctl);
    const int ge = grid_for(n, kThreads, sms);
    if (n) {
        set_state_claim_kernel<<<ge, kThreads, 0, st>>>(keys, n, frame, t, ctl);
        set_state_clear_kernel<<<grid_for(n * kSlots, kThreads, sms), kThreads, 0, st>>>(t, ctl);
        set_state_fill_kernel<<<ge, kThreads, 0, st>>>(keys, re, im, n, frame, t, ctl, dbl ? 1 : 0);
    }
    set_state_end_kernel<<<1, 1, 0, st>>>(ctl, n);
    return cudaGetLastError();
}

cudaError_t launch_refresh_masks(const TableDev& t, Ctl* ctl, unsigned long long list_hint, int sms, cudaStream_t st) {
    refresh_masks_kernel<<<grid_for(list_hint, kThreads / 16, sms), kThreads, 0, st>>>(t, ctl);
    return cudaGetLastError();
}

cudaError_t launch_readout(const TableDev& t, Ctl* ctl, unsigned long long list_hint, unsigned long long frame,
                           bool dbl, unsigned long long* okeys, double* ore, double* oim, unsigned long long cap,
                           bool drop_negl, PruneBits pb, int sms, cudaStream_t st, unsigned long long smask,
                           unsigned long long sval) {
    const int grid = grid_for(list_hint / 32 + 1, kThreads / 32, sms);
    if (dbl)
        readout_kernel<double><<<grid, kThreads, 0, st>>>(t, ctl, frame, okeys, ore, oim, cap, drop_negl, pb,
                                                           smask, sval);
    else
        readout_kernel<float><<<grid, kThreads, 0, st>>>(t, ctl, frame, okeys, ore, oim, cap, drop_negl, pb,
                                                          smask, sval);
    return cudaGetLastError();
}

cudaError_t launch_norm(const TableDev& t, Ctl* ctl, unsigned long long list_hint, bool dbl, ExactSums* sums, int sms,
                        cudaStream_t st) {
    const int grid = grid_for(list_hint * kSlots + 1, kThreads, sms);
    if (dbl) norm_kernel<double><<<grid, kThreads, 0, st>>>(t, ctl, sums);
    else norm_kernel<float><<<grid, kThreads, 0, st>>>(t, ctl, sums);
    return cudaGetLastError();
}

cudaError_t launch_compare(const TableDev& ta, const Ctl* ca, unsigned long long hint_a, bool dbl_a,
                           const TableDev& tb, const Ctl* cb, unsigned long long hint_b, bool dbl_b,
                           unsigned long long d, Ctl* out, ExactSums* sums, int sms, cudaStream_t st) {
    const int ga = grid_for(hint_a * kSlots + 1, kThreads, sms);
    compare_a_kernel<0><<<ga, kThreads, 0, st>>>(ta, ca, dbl_a, tb, cb, dbl_b, d, out, sums);
    compare_a_kernel<1><<<ga, kThreads, 0, st>>>(ta, ca, dbl_a, tb, cb, dbl_b, d, out, sums);
    compare_b_kernel<<<grid_for(hint_b * kSlots + 1, kThreads, sms), kThreads, 0, st>>>(ta, ca, tb, cb, dbl_b, d, out,
                                                                                        sums);
    return cudaGetLastError();
}

// Throughput probe of the FP64 pipe: every thread runs eight independent chains of dependent
// fused multiply-adds (x = x * a + b), so the pipe, not latency, bounds it. The result is kept
// alive by a store no input can trigger.
__global__ void fp64_rate_kernel(double* sink, double a, double b, int iters) {
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = 1.0 + 1e-3 * (threadIdx.x + k);
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = __fma_rn(x[k], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x[k];
    if (s == -1.0) sink[0] = s;
}

cudaError_t measure_fp64_rate(int sms, double* fma_per_s) {
    const int blocks = sms * 8, threads = 256, iters = 4096;
    double* sink = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t e = cudaMalloc(&sink, sizeof(double));
    if (e == cudaSuccess) e = cudaEventCreate(&e0);
    if (e == cudaSuccess) e = cudaEventCreate(&e1);
    float best = 0.f;
    for (int rep = 0; rep < 3 && e == cudaSuccess; ++rep) {   // the first launch warms up
        cudaEventRecord(e0);
        fp64_rate_kernel<<<blocks, threads>>>(sink, 0.9999999, 1e-7, iters);
        cudaEventRecord(e1);
        e = cudaEventSynchronize(e1);
        float ms = 0.f;
        if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0 && (best == 0.f || ms < best)) best = ms;
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (sink) cudaFree(sink);
    *fma_per_s = (e == cudaSuccess && best > 0.f) ? (double)blocks * threads * iters * 8 / (best * 1e-3) : 0.0;
    return e;
}

cudaError_t launch_rehash(const TableDev& told, unsigned long long n_old, const TableDev& tnew, unsigned ep_new,
                          int amp_bytes, Ctl* ctl, int sms, cudaStream_t st) {
    const int grid = grid_for(n_old / 32 + 1, kThreads / 32, sms);
    rehash_kernel<<<grid, kThreads, 0, st>>>(told, n_old, tnew, ep_new, amp_bytes, ctl);
    return cudaGetLastError();
}

}  // namespace sqc
