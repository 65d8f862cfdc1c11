// Device-side layout and arithmetic of the sparse statevector table.
//
// Table layout (one table per state, updated in place by every pass):
//   hdr [nb]          16-byte bucket headers {group, epoch, presence mask}
//   keys[nb * 16]     64-bit stored keys, 16 per bucket (128 bytes)
//   amps[nb * 16]     amplitudes, double2 (FP64) or float2 (FP32), same slot order
//   list[nb]          indices of the live buckets, in claim order
// A bucket holds the keys of one group G = key >> 4 at slot key & 15. Buckets are found by
// their mapped bits, or in hashed tables by linear probing from mix64(G) & (nb - 1) (sqc_types.h,
// TableDev). A bucket is live iff hdr.epoch equals the state's
// epoch, so a reset only bumps the epoch. A slot is occupied iff the low 4 bits of its
// stored key equal the slot index; empty slots hold EMPTY(j) = 0xFFFF...F0 | (15 - j).
// Live buckets are never freed between resets: a group whose keys are all pruned stays as an
// empty live bucket, so probe chains never break.
//
// The reference keeps one dense slot per basis state (identity hash, 2^nq slots,
// emulator/device/table_manager.cuh:114-119, emulator/include/sim_parameters_types.h:153-158);
// here the table is sized by load factor and holds only present keys, so 64-qubit keys work.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "sqc_types.h"

namespace sqc {

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 30; x *= 0xbf58476d1ce4e5b9ULL;
    x ^= x >> 27; x *= 0x94d049bb133111ebULL;
    x ^= x >> 31; return x;
}

__device__ __forceinline__ unsigned long long empty_key(int j) {
    return 0xFFFFFFFFFFFFFFF0ULL | (unsigned long long)(15 - j);
}

__device__ __forceinline__ unsigned long long shfl64(unsigned long long v, int src) {
    unsigned lo = __shfl_sync(kFull, (unsigned)v, src);
    unsigned hi = __shfl_sync(kFull, (unsigned)(v >> 32), src);
    return ((unsigned long long)hi << 32) | lo;
}

__device__ __forceinline__ Header load_hdr(const Header* p) {
    ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    Header h;
    h.group = v.x;
    h.epoch = (unsigned)v.y;
    h.aux = (unsigned)(v.y >> 32);
    return h;
}

__device__ __forceinline__ Header load_hdr_cg(const Header* p) {
    ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
    Header h;
    h.group = v.x;
    h.epoch = (unsigned)v.y;
    h.aux = (unsigned)(v.y >> 32);
    return h;
}

// 128-bit compare-and-swap on a bucket header. Returns the previous content.
__device__ __forceinline__ Header cas_hdr(Header* p, const Header& expect, const Header& desired) {
    unsigned long long e0 = expect.group, e1 = (unsigned long long)expect.epoch | ((unsigned long long)expect.aux << 32);
    unsigned long long d0 = desired.group, d1 = (unsigned long long)desired.epoch | ((unsigned long long)desired.aux << 32);
    unsigned long long o0, o1;
    asm volatile(
        "{\n\t.reg .b128 d, c, s;\n\t"
        "mov.b128 c, {%2, %3};\n\t"
        "mov.b128 s, {%4, %5};\n\t"
        "atom.global.cas.b128 d, [%6], c, s;\n\t"
        "mov.b128 {%0, %1}, d;\n\t}"
        : "=l"(o0), "=l"(o1)
        : "l"(e0), "l"(e1), "l"(d0), "l"(d1), "l"(p)
        : "memory");
    Header o;
    o.group = o0;
    o.epoch = (unsigned)o1;
    o.aux = (unsigned)(o1 >> 32);
    return o;
}

// Bucket where group G lives (mapped table) or where its probe chain starts (hashed table).
__device__ __forceinline__ unsigned long long home_bucket(const TableDev& t, unsigned long long G) {
    if (!t.map_on) return mix64(G) & t.mask;
    unsigned b = 0;
    for (uint32_t i = 0; i < t.map_n; ++i) b |= (unsigned)((G >> t.map_q[i]) & 1ULL) << i;
    return b;
}

// Group of bucket b of a mapped table (map_n bits, mq its map_q).
__device__ __forceinline__ unsigned long long group_of_bucket(uint32_t map_n, const uint8_t* mq, unsigned b) {
    unsigned long long G = 0;
    for (uint32_t i = 0; i < map_n; ++i) G |= (unsigned long long)((b >> i) & 1u) << mq[i];
    return G;
}

// Find the live bucket of group G, or -1. Correct while other threads claim buckets: a
// claim only turns a non-live bucket live, and G's probe chain has no non-live bucket.
__device__ __forceinline__ long long lookup_group(const TableDev& t, unsigned ep, unsigned long long G) {
    unsigned long long b = home_bucket(t, G);
    for (uint32_t i = 0; i < kMaxProbe; ++i) {
        const Header h = load_hdr_cg(t.hdr + b);
        if (h.epoch != ep) return -1;
        if (h.group == G) return (long long)b;
        if (t.map_on) return -1;   // the address is exact: a group with a bit outside the map is nowhere else
        b = (b + 1) & t.mask;
    }
    return -1;
}

// Claim (or find) the bucket of group G: linear probing with a 128-bit CAS per attempt,
// bounded. *created tells whether this call turned the bucket live. -1 and ST_TABLE_FULL
// when no bucket within kMaxProbe of the home bucket is free.
__device__ __forceinline__ long long claim_group(const TableDev& t, unsigned ep, unsigned long long G,
                                                 unsigned int* status, bool* created) {
    *created = false;
    unsigned long long b = home_bucket(t, G);
    Header cur = load_hdr_cg(t.hdr + b);
    uint32_t probes = 0, attempts = 0;
    while (probes < kMaxProbe && attempts < 4 * kMaxProbe) {
        ++attempts;
        if (cur.epoch == ep) {
            if (cur.group == G) return (long long)b;
            b = (b + 1) & t.mask;
            ++probes;
            cur = load_hdr_cg(t.hdr + b);
            continue;
        }
        Header want;
        want.group = G; want.epoch = ep; want.aux = 0;
        const Header old = cas_hdr(t.hdr + b, cur, want);
        if (old.group == cur.group && old.epoch == cur.epoch && old.aux == cur.aux) {
            *created = true;
            return (long long)b;
        }
        cur = old;   // re-examine this bucket with its actual content
    }
    atomicCAS(status, 0u, (unsigned)ST_TABLE_FULL);
    return -1;
}

// ---- arithmetic --------------------------------------------------------------------------
// Explicit round-to-nearest operations: nothing is contracted, so every product and sum
// rounds exactly as in the reference's source formulas (emulator/device/device_data.cuh:159-319).
template <class T> struct Arith;
template <> struct Arith<double> {
    __device__ static __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    __device__ static __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    __device__ static __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
};
template <> struct Arith<float> {
    __device__ static __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    __device__ static __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ static __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    __device__ static __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
};

template <class T> struct Cx { T r, i; };

// Sign flips and magnitude tests as integer operations: on this GPU every FP64 instruction,
// compares and negations included, issues on the slow FP64 pipe. Both forms are exact. The
// flip is an opaque integer xor on the high word, so the compiler cannot turn it back into
// a floating-point negation (which it may lower to an FP64 add).
__device__ __forceinline__ double neg(double x) {
    int hi = __double2hiint(x);
    const int lo = __double2loint(x);
    asm("xor.b32 %0, %0, 0x80000000;" : "+r"(hi));
    return __hiloint2double(hi, lo);
}
__device__ __forceinline__ float neg(float x) {
    int v = __float_as_int(x);
    asm("xor.b32 %0, %0, 0x80000000;" : "+r"(v));
    return __int_as_float(v);
}

// Programmatic dependent launch. Single passes are launched with programmatic stream
// serialization, so the next pass's blocks may be placed on the SMs while the running pass
// drains. Such a kernel first waits until the previous grid in the stream has completed and
// its writes are visible (a no-op without that launch attribute), and then lets the next pass
// be scheduled: its blocks only wait in turn, and all of this grid's blocks are already
// resident by then, so nothing waits on a block that cannot be placed.
__device__ __forceinline__ void wait_prior_grid() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void allow_next_grid() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Swap update for gate kind K: the amplitude arriving from the partner (reference: x_core,
// y_core).
template <class T, uint32_t K>
__device__ __forceinline__ Cx<T> swap_update(bool bit, Cx<T> b) {
    if constexpr (K == KX) return b;
    else return bit ? Cx<T>{neg(b.i), b.r} : Cx<T>{b.i, neg(b.r)};   // Y
}

__host__ __device__ constexpr bool branch_kind(uint32_t k) { return k == KH || k == KRX || k == KRY || k == KU; }

// Prune rule of the reference (emulator/include/data_t.h:50-60): |re| < thr && |im| < thr,
// decided in FP64. For doubles |x| < thr is compared on the bit patterns (non-negative
// doubles order like their bits; NaN compares false as in the FP64 test). For floats the
// host passes the largest float f with (double)f < thr, so |x| <= f is the same FP64 test.
__device__ __forceinline__ bool negligible(Cx<double> v, const PruneBits& t) {
    const unsigned long long m = 0x7FFFFFFFFFFFFFFFULL;
    return ((unsigned long long)__double_as_longlong(v.r) & m) < t.d &&
           ((unsigned long long)__double_as_longlong(v.i) & m) < t.d;
}
// FP32 compares issue on the wide FP32 pipes and take |x| as an operand modifier: one compare
// per component (NaN compares false, as its bit pattern does above t.f).
__device__ __forceinline__ bool negligible(Cx<float> v, const PruneBits& t) {
    const float f = __int_as_float((int)t.f);
    return fabsf(v.r) <= f && fabsf(v.i) <= f;
}

}  // namespace sqc
