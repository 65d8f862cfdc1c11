// Unit passes over mapped tables (sqc_types.h, TableDev), shared by the single-state kernels and
// the persistent batch kernel.
//
// A mapped table addresses groups directly, so a pass needs no list walk, no lookups and no
// ownership: a unit of DIMS dimensions (2: four buckets, 3: eight) is the set of buckets that
// differ in DIMS bucket bits, unit u of a table of dn mapped bits has its base bucket at u with
// zeros inserted at those bits, and one warp holds the whole unit: half h of the warp the buckets
// with dimension 1 equal h, lane j of a half the slots j of S = 2^(DIMS-1) buckets (slot bit 0 is
// dimension 0, slot bit 1 is dimension 2). Dimensions no gate of the pass pairs across are filled
// with low bucket bits, so every pass has the same shape.
//
// Everything a gate tests is then known by place instead of by key: controls outside the unit are
// one comparison per warp (a gate they exclude costs a few instructions for the whole unit),
// controls inside it one per lane, and slot controls are uniform. Presence is one bit per slot,
// kept per bucket in Header.aux, so passes move amplitudes and headers and touch keys only where
// presence changes: FP32 16.5 bytes per key and pass instead of 32.
#pragma once
#include "sqc_dmul.cuh"
#include "sqc_device.cuh"

namespace sqc {
namespace {

template <class T> struct AmpT;
template <> struct AmpT<double> { using V = double2; };
template <> struct AmpT<float> { using V = float2; };

template <class T> __device__ __forceinline__ Cx<T> czero() { return Cx<T>{T(0), T(0)}; }

__device__ __forceinline__ unsigned long long umin64(unsigned long long a, unsigned long long b) { return a < b ? a : b; }

template <class T>
__device__ __forceinline__ void store_amp(void* amps, size_t s, Cx<T> a) {
    typename AmpT<T>::V v;
    v.x = a.r;
    v.y = a.i;
    reinterpret_cast<typename AmpT<T>::V*>(amps)[s] = v;
}

template <class T>
__device__ __forceinline__ Cx<T> pick(bool c, Cx<T> x, Cx<T> y) {
    return Cx<T>{c ? x.r : y.r, c ? x.i : y.i};
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
    for (int o = 16; o; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    return v;
}

// A pass's gate in shared memory: the first 16 bytes say where it acts, then the coefficients.
template <class T> struct UGate;
template <> struct alignas(16) UGate<float> {
    uint32_t om, ov, loc, weight;        // weight: amp updates a present key counts (1 + credit)
    float c, s, pad[2];
    float m[8];                          // U
};
template <> struct alignas(16) UGate<double> {
    uint32_t om, ov, loc, weight;
    double c, s;
    uint32_t ch, cl, ce, min_exp;        // DCoef of c; the larger min_exp of the two
    uint32_t sh, sl, se, exact;          // DCoef of s; integer products allowed for both
};

__device__ __forceinline__ void stage_ugate_head(uint32_t& om, uint32_t& ov, uint32_t& loc, uint32_t& weight,
                                                 const GateDesc* g) {
    om = __ldg(&g->om);
    ov = __ldg(&g->ov);
    loc = __ldg(&g->loc);
    weight = __ldg(&g->pad) + 1u;
}

__device__ __forceinline__ void stage_ugate(UGate<float>* d, const GateDesc* g) {
    UGate<float> x;
    stage_ugate_head(x.om, x.ov, x.loc, x.weight, g);
    x.c = __ldg(&g->cf);
    x.s = __ldg(&g->sf);
    x.pad[0] = x.pad[1] = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) x.m[i] = __ldg(&g->mf[i]);
    *d = x;
}

__device__ __forceinline__ void stage_ugate(UGate<double>* d, const GateDesc* g) {
    UGate<double> x;
    stage_ugate_head(x.om, x.ov, x.loc, x.weight, g);
    x.c = __ldg(&g->c);
    x.s = __ldg(&g->s);
    const DCoef c = dcoef((uint64_t)__double_as_longlong(x.c));
    const uint32_t op = x.loc >> kLocOp;
    const uint32_t form = op >= UO_ALL3 ? (op - UO_ALL3) & ~1u : op >= UO_ALL ? op - UO_ALL : op;
    const bool two = form >= UO_RX_PAIR;   // H has one coefficient
    const DCoef s = dcoef((uint64_t)__double_as_longlong(two ? x.s : x.c));
    x.exact = c.ok && s.ok;
    x.ch = c.hi; x.cl = c.lo; x.ce = c.exp;
    x.sh = s.hi; x.sl = s.lo; x.se = s.exp;
    x.min_exp = c.min_exp > s.min_exp ? c.min_exp : s.min_exp;
    *d = x;
}

// What a gate does on one lane, decoded once per pass: bits 0..3 the slots it acts on (its controls
// on lane and slot bits hold), bits 4..7 the slots among them with logical target bit 1 (diagonal
// gates; as if the target's bit of the unit's base were 0), bit 31 the logical target bit of the
// lane (shuffles) or of the first slot of a pair. Kept as 16 bits, the top one sign-extended.
__device__ __forceinline__ uint32_t lane_word(uint32_t loc, uint32_t lane) {
    const bool on = (((loc >> kLocLaneVal) ^ lane) & loc & 31u) == 0;
    const uint32_t tb = (loc >> kLocBit) & 31u;
    const bool at = (loc & kLocLane) && ((lane >> tb) & 1u), flip = (loc & kLocFlip) != 0;
    const uint32_t act = on ? (loc >> kLocSlots) & 15u : 0u;
    const uint32_t e = (((loc >> kLocSlotBit) & 15u) ^ (at ? 15u : 0u)) & act;
    return act | (e << 4) | (at != flip ? 0x80000000u : 0u);
}

__device__ __forceinline__ int16_t short_word(uint32_t w) { return (int16_t)((w & 0xFFu) | ((w >> 16) & 0x8000u)); }

// A pass's heads read from its gates in shared memory. ODD: some may be UO_ODD gates.
template <class T, bool ODD = false> struct SharedHeads {
    const UGate<T>* g;
    __device__ __forceinline__ UnitHead operator[](uint32_t i) const {
        const uint4 h = *reinterpret_cast<const uint4*>(g + i);   // om, ov, loc, weight
        return UnitHead{h.x, h.y, h.z, h.w};
    }
};

template <class Heads> constexpr bool kOddHeads = false;
template <class T> constexpr bool kOddHeads<SharedHeads<T, true>> = true;

// The gates of a pass in shared memory: the gates, and their lane words.
template <class T> struct UGates {
    UGate<T> g[kMaxRun];
    int16_t lw[kMaxRun][32];
};

// Copy gates [g0, g1) (at most kMaxRun) into shared memory; every thread of the block calls it, and it
// ends with a barrier.
template <class T>
__device__ __forceinline__ void stage_ugates(UGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t g0, uint32_t g1) {
    for (uint32_t i = threadIdx.x; g0 + i < g1; i += blockDim.x) stage_ugate(sg.g + i, gates + g0 + i);
    for (uint32_t i = threadIdx.x; i < (g1 - g0) * 32u; i += blockDim.x)
        sg.lw[i >> 5][i & 31u] = short_word(lane_word(__ldg(&gates[g0 + (i >> 5)].loc), i & 31u));
    __syncthreads();
}

// ---- arithmetic of one slot -----------------------------------------------------------------------
// Products of one amplitude by the gate's coefficients: C = c * x and, with TWO, P = s * x. FP64
// forms them on the integer pipes where the operands allow it (sqc_dmul.cuh).
__device__ __forceinline__ double dmul_exact(const DUnpacked& u, uint32_t h, uint32_t l, uint32_t e, double c) {
    uint32_t oh, ol;
    dproduct(u, h, l, e, (uint32_t)__double2hiint(c), &oh, &ol);
    return __hiloint2double((int)oh, (int)ol);
}
template <bool TWO>
__device__ __forceinline__ void products(const UGate<double>& g, Cx<double> x, Cx<double>& C, Cx<double>& P) {
    const DUnpacked r = dunpack((uint32_t)__double2hiint(x.r), (uint32_t)__double2loint(x.r), g.min_exp);
    const DUnpacked i = dunpack((uint32_t)__double2hiint(x.i), (uint32_t)__double2loint(x.i), g.min_exp);
    if (g.exact && !r.slow && !i.slow) {
        C.r = dmul_exact(r, g.ch, g.cl, g.ce, g.c);
        C.i = dmul_exact(i, g.ch, g.cl, g.ce, g.c);
        if (TWO) {
            P.r = dmul_exact(r, g.sh, g.sl, g.se, g.s);
            P.i = dmul_exact(i, g.sh, g.sl, g.se, g.s);
        }
    } else {
        C.r = __dmul_rn(g.c, x.r);
        C.i = __dmul_rn(g.c, x.i);
        if (TWO) {
            P.r = __dmul_rn(g.s, x.r);
            P.i = __dmul_rn(g.s, x.i);
        }
    }
}
// FP32 arithmetic on an amplitude's two components at once (one instruction each; every component is
// rounded as by the scalar instruction).
__device__ __forceinline__ unsigned long long pack2(float r, float i) {
    unsigned long long p;
    asm("mov.b64 %0, {%1, %2};" : "=l"(p) : "f"(r), "f"(i));
    return p;
}
__device__ __forceinline__ unsigned long long pack2(Cx<float> v) { return pack2(v.r, v.i); }
__device__ __forceinline__ Cx<float> unpack2(unsigned long long p) {
    Cx<float> v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.r), "=f"(v.i) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// Sums of two products go through scalar additions: the assembler fuses a packed product into a
// packed sum (found by comparing with the oracle), which rounds once instead of twice.
__device__ __forceinline__ Cx<float> add_parts(unsigned long long a, unsigned long long b) {
    const Cx<float> x = unpack2(a), y = unpack2(b);
    return Cx<float>{__fadd_rn(x.r, y.r), __fadd_rn(x.i, y.i)};
}

// x with its sign flipped where m has bit 31 set. The xor is opaque: written in C++ the compiler
// turned it into FP64 negations (Rz 8.7 -> 6.5 us per gate on 2^20 keys without them).
__device__ __forceinline__ double flip_sign(double x, uint32_t m) {
    int hi = __double2hiint(x);
    asm("lop3.b32 %0, %0, %1, 0x80000000, 0x78;" : "+r"(hi) : "r"(m));   // hi ^ (m & sign)
    return __hiloint2double(hi, __double2loint(x));
}
__device__ __forceinline__ float flip_sign(float x, uint32_t m) {
    return __int_as_float(__float_as_int(x) ^ (int)(m & 0x80000000u));
}

template <class T>
__device__ __forceinline__ Cx<T> shfl_cx(Cx<T> a, int off) {
    return Cx<T>{__shfl_xor_sync(kFull, a.r, off), __shfl_xor_sync(kFull, a.i, off)};
}

// ---- one gate on the slots a lane holds ---------------------------------------------------------
// Every result rounds as the reference's pair formula for that member (emulator/device/device_data.cuh:159-319):
//   H : bit 0 -> f*(v0 + v1),             bit 1 -> f*(v0 - v1)
//   Rx: c*own + s*(i-rotated partner)      (symmetric in the two members)
//   Ry: bit 0 -> c*v0 - s*v1,             bit 1 -> c*v1 + s*v0
//   U : self term first, then partner term, fused multiply-add chain (no reference form).
// An Rx, Ry, Rz or Phase result is C + P', C = c * own, P' the s-product of the own or the partner
// amplitude with its sign flipped and its components exchanged as the kind asks (a - b and a + (-b),
// (-s) * x and -(s * x), and (-1) * a + b and b - a, round alike).
template <class T, int S> struct Slots {
    Cx<T> v[S];
    unsigned pm;   // presence bits
    unsigned n;    // their number
};

// Both results of a branching gate on a lane-local pair: a the slot whose logical target bit is w's
// bit 31, b its partner.
template <uint32_t K>
__device__ __forceinline__ void pair_results(const UGate<float>& g, const GateDesc*, uint32_t w, Cx<float>& a, Cx<float>& b) {
    const unsigned long long pa = pack2(a), pb = pack2(b);
    if constexpr (K == KH) {   // logical bit 0: v0 + v1, bit 1: v0 - v1
        const float one = __int_as_float(0x3F800000 | (int)(w & 0x80000000u));   // -1 where a has bit 1
        const unsigned long long f = pack2(g.c, g.c);
        a = unpack2(mul2(f, fma2(pa, pack2(one, one), pb)));
        b = unpack2(mul2(f, fma2(pb, pack2(-one, -one), pa)));
    } else if constexpr (K == KRX) {
        const unsigned long long c = pack2(g.c, g.c), s = pack2(g.s, g.s);
        const Cx<float> ca = unpack2(mul2(c, pa)), cb = unpack2(mul2(c, pb));
        const Cx<float> sa = unpack2(mul2(s, pa)), sb = unpack2(mul2(s, pb));
        a = Cx<float>{__fadd_rn(ca.r, sb.i), __fsub_rn(ca.i, sb.r)};
        b = Cx<float>{__fadd_rn(cb.r, sa.i), __fsub_rn(cb.i, sa.r)};
    } else if constexpr (K == KRY) {   // bit 0: c*own - s*partner, bit 1: c*own + s*partner
        const float sa = flip_sign(g.s, ~w);
        const unsigned long long c = pack2(g.c, g.c);
        a = add_parts(mul2(c, pa), mul2(pack2(sa, sa), pb));
        b = add_parts(mul2(c, pb), mul2(pack2(-sa, -sa), pa));
    } else {   // U: fused multiply-add chains, the self terms first
        const bool bit = (w >> 31) != 0;
        const unsigned long long xa = pack2(a.i, a.r), xb = pack2(b.i, b.r);
        const int own = bit ? 6 : 0, mix = bit ? 4 : 2;   // a's row; b's row is the other one
        const float ar = g.m[own], ai = g.m[own + 1], br = g.m[6 - own], bi = g.m[7 - own];
        const float amr = g.m[mix], ami = g.m[mix + 1], bmr = g.m[6 - mix], bmi = g.m[7 - mix];
        unsigned long long oa = mul2(pack2(ar, ar), pa), ob = mul2(pack2(br, br), pb);
        oa = fma2(pack2(-ai, ai), xa, oa);
        ob = fma2(pack2(-bi, bi), xb, ob);
        oa = fma2(pack2(amr, amr), pb, oa);
        ob = fma2(pack2(bmr, bmr), pa, ob);
        a = unpack2(fma2(pack2(-ami, ami), xb, oa));
        b = unpack2(fma2(pack2(-bmi, bmi), xa, ob));
    }
}

// Whether x is finite and its high word not 0: adding +-0 to it then changes nothing (no FP64 compare).
__device__ __forceinline__ bool plain(double x) { return ((uint32_t)__double2hiint(x) & 0x7FFFFFFFu) - 1u < 0x7FEFFFFFu; }
// U's chain for one member. `uniform`: its logical bit is the whole warp's; the bit-0 row's own
// coefficient is real, and its imaginary terms are 0 * a part of a: they add +-0, and two of the chain's
// eight FP64 instructions are spared, unless a part is infinite or NaN (the sum so far, a part
// times a coefficient of at most 1, then is too) or the sum so far is 0.
__device__ __forceinline__ Cx<double> u_update(const GateDesc* gd, bool bit, bool uniform, Cx<double> a, Cx<double> b) {
    auto m = [&](int i) { return __ldg(&gd->m[i]); };
    const double msr = bit ? m(6) : m(0), mor = bit ? m(4) : m(2), moi = bit ? m(5) : m(3);
    double r = __dmul_rn(msr, a.r), i = __dmul_rn(msr, a.i);
    if (!uniform || bit || !plain(r) || !plain(i)) {
        const double msi = bit ? m(7) : m(1);
        r = __fma_rn(neg(msi), a.i, r);
        i = __fma_rn(msi, a.r, i);
    }
    return Cx<double>{__fma_rn(neg(moi), b.i, __fma_rn(mor, b.r, r)), __fma_rn(moi, b.r, __fma_rn(mor, b.i, i))};
}
template <uint32_t K>
__device__ __forceinline__ void pair_results(const UGate<double>& g, const GateDesc* gd, uint32_t w, Cx<double>& a,
                                             Cx<double>& b) {
    using A = Arith<double>;
    if constexpr (K == KH) {
        const Cx<double> y0{A::add(b.r, flip_sign(a.r, w)), A::add(b.i, flip_sign(a.i, w))};
        const Cx<double> y1{A::add(a.r, flip_sign(b.r, ~w)), A::add(a.i, flip_sign(b.i, ~w))};
        Cx<double> none;
        products<false>(g, y0, a, none);
        products<false>(g, y1, b, none);
    } else if constexpr (K == KU) {
        const Cx<double> o = u_update(gd, (w >> 31) != 0, true, a, b);
        b = u_update(gd, (w >> 31) == 0, true, b, a);
        a = o;
    } else {
        Cx<double> C0, C1, P0, P1;
        products<true>(g, a, C0, P0);
        products<true>(g, b, C1, P1);
        if constexpr (K == KRX) {
            a = Cx<double>{A::add(C0.r, P1.i), A::sub(C0.i, P1.r)};
            b = Cx<double>{A::add(C1.r, P0.i), A::sub(C1.i, P0.r)};
        } else {
            a = Cx<double>{A::add(C0.r, flip_sign(P1.r, ~w)), A::add(C0.i, flip_sign(P1.i, ~w))};
            b = Cx<double>{A::add(C1.r, flip_sign(P0.r, w)), A::add(C1.i, flip_sign(P0.i, w))};
        }
    }
}

// A branching gate's result for a slot whose partner is in lane ^ off; every lane calls it.
template <uint32_t K>
__device__ __forceinline__ Cx<float> shfl_result(const UGate<float>& g, const GateDesc*, uint32_t w, int off, Cx<float> a) {
    const unsigned long long pa = pack2(a);
    if constexpr (K == KH) {
        const float one = __int_as_float(0x3F800000 | (int)(w & 0x80000000u));
        return unpack2(mul2(pack2(g.c, g.c), fma2(pa, pack2(one, one), pack2(shfl_cx(a, off)))));
    } else if constexpr (K == KRX) {
        const Cx<float> b = shfl_cx(a, off);
        const Cx<float> c = unpack2(mul2(pack2(g.c, g.c), pa)), s = unpack2(mul2(pack2(g.s, g.s), pack2(b)));
        return Cx<float>{__fadd_rn(c.r, s.i), __fsub_rn(c.i, s.r)};
    } else if constexpr (K == KRY) {
        const float s = flip_sign(g.s, ~w);
        return add_parts(mul2(pack2(g.c, g.c), pa), mul2(pack2(s, s), pack2(shfl_cx(a, off))));
    } else {
        const Cx<float> b = shfl_cx(a, off);
        const bool bit = (w >> 31) != 0;
        const float sr = bit ? g.m[6] : g.m[0], si = bit ? g.m[7] : g.m[1];
        const float mr = bit ? g.m[4] : g.m[2], mi = bit ? g.m[5] : g.m[3];
        unsigned long long o = mul2(pack2(sr, sr), pa);
        o = fma2(pack2(-si, si), pack2(a.i, a.r), o);
        o = fma2(pack2(mr, mr), pack2(b), o);
        return unpack2(fma2(pack2(-mi, mi), pack2(b.i, b.r), o));
    }
}
template <uint32_t K>
__device__ __forceinline__ Cx<double> shfl_result(const UGate<double>& g, const GateDesc* gd, uint32_t w, int off,
                                                  Cx<double> a) {
    using A = Arith<double>;
    Cx<double> o, P;
    if constexpr (K == KH) {
        const Cx<double> b = shfl_cx(a, off);
        const Cx<double> y{A::add(b.r, flip_sign(a.r, w)), A::add(b.i, flip_sign(a.i, w))};
        products<false>(g, y, o, P);
        return o;
    } else if constexpr (K == KU) {
        return u_update(gd, (w >> 31) != 0, false, a, shfl_cx(a, off));
    } else {
        products<true>(g, a, o, P);   // the partner lane needs this lane's s-product
        P = shfl_cx(P, off);
        if constexpr (K == KRX) return Cx<double>{A::add(o.r, P.i), A::sub(o.i, P.r)};
        else return Cx<double>{A::add(o.r, flip_sign(P.r, ~w)), A::add(o.i, flip_sign(P.i, ~w))};
    }
}

// After a branching gate on the slots of `act`: they are present, but for results below the prune
// threshold, which are rare in slots that hold keys: one test over all slots, and a branch that
// looks at each.
template <int S>
__device__ __forceinline__ bool may_prune(const Slots<float, S>& x, const PruneBits& pb) {
    float m = fmaxf(fabsf(x.v[0].r), fabsf(x.v[0].i));
#pragma unroll
    for (int s = 1; s < S; ++s) m = fminf(m, fmaxf(fabsf(x.v[s].r), fabsf(x.v[s].i)));
    return !(m > __int_as_float((int)pb.f));
}
template <int S>
__device__ __forceinline__ bool may_prune(const Slots<double, S>& x, const PruneBits& pb) {
    uint32_t m = ~0u;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const uint32_t r = (uint32_t)__double2hiint(x.v[s].r) & 0x7FFFFFFFu, i = (uint32_t)__double2hiint(x.v[s].i) & 0x7FFFFFFFu;
        m = min(m, max(r, i));
    }
    return m <= (uint32_t)(pb.d >> 32);
}
template <class T, int S>
__device__ __forceinline__ void settle(Slots<T, S>& x, uint32_t act, const PruneBits& pb) {
    x.pm |= act;
    if (!may_prune<S>(x, pb)) {
        x.n = __popc(x.pm);
        return;
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if ((act & (1u << s)) && negligible(x.v[s], pb)) {
            x.v[s] = czero<T>();
            x.pm &= ~(1u << s);
        }
    }
    x.n = __popc(x.pm);
}

// The first slot of pair p of stride ST: (0, 1), (2, 3) or (0, 2), (1, 3).
template <int ST> __device__ constexpr int pair_slot(int p) { return ST == 1 ? 2 * p : p; }

template <class T, uint32_t K, int S, int ST, bool ALL>
__device__ __forceinline__ void branch_pair(const UGate<T>& g, const GateDesc* gd, uint32_t w, Slots<T, S>& x,
                                            const PruneBits& pb) {
#pragma unroll
    for (int p = 0; p < S / 2; ++p) {
        constexpr int kStep = S == 2 ? 1 : ST;
        const int s = S == 2 ? 0 : pair_slot<ST>(p);
        if (ALL || (w & (1u << s))) pair_results<K>(g, gd, w, x.v[s], x.v[s + kStep]);
    }
    settle<T, S>(x, ALL ? (1u << S) - 1u : w & ((1u << S) - 1u), pb);
}

template <class T, uint32_t K, int S, bool ALL>
__device__ __forceinline__ void branch_shfl(const UGate<T>& g, const GateDesc* gd, uint32_t loc, uint32_t w, Slots<T, S>& x,
                                            const PruneBits& pb) {
    const int off = 1 << ((loc >> kLocBit) & 31u);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (!ALL && !(loc & (1u << (kLocSlots + s)))) continue;
        const Cx<T> o = shfl_result<K>(g, gd, w, off, x.v[s]);
        if (ALL || (w & (1u << s))) x.v[s] = o;
    }
    settle<T, S>(x, ALL ? (1u << S) - 1u : w & ((1u << S) - 1u), pb);
}

template <class T, uint32_t K, int S, int ST, bool ALL>
__device__ __forceinline__ void swap_pair(uint32_t w, Slots<T, S>& x) {
    const bool flip = (w >> 31) != 0;
#pragma unroll
    for (int p = 0; p < S / 2; ++p) {
        constexpr int kStep = S == 2 ? 1 : ST;
        const int s = S == 2 ? 0 : pair_slot<ST>(p);
        if (!ALL && !(w & (1u << s))) continue;
        const Cx<T> a = x.v[s], b = x.v[s + kStep];
        x.v[s] = swap_update<T, K>(flip, b);
        x.v[s + kStep] = swap_update<T, K>(!flip, a);
        const unsigned lo = 1u << s, hi = lo << kStep;
        x.pm = (x.pm & ~(lo | hi)) | ((x.pm >> kStep) & lo) | ((x.pm << kStep) & hi);
    }
}

template <class T, uint32_t K, int S, bool ALL>
__device__ __forceinline__ void swap_shfl(uint32_t loc, uint32_t w, Slots<T, S>& x) {
    const int off = 1 << ((loc >> kLocBit) & 31u);
    const unsigned pp = __shfl_xor_sync(kFull, x.pm, off);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (!ALL && !(loc & (1u << (kLocSlots + s)))) continue;
        const Cx<T> b = shfl_cx(x.v[s], off);
        if (ALL || (w & (1u << s))) x.v[s] = swap_update<T, K>((w >> 31) != 0, b);
    }
    x.pm = ALL ? pp : (x.pm & ~(w & 15u)) | (pp & w & 15u);
    x.n = __popc(x.pm);   // (a lane's, not the unit's, changes)
}

// Rz (every bit; minus: bit 31 set where the logical bit is 1) and Phase (bit 1 only) on one slot.
template <bool RZ>
__device__ __forceinline__ Cx<float> turn(const UGate<float>& g, uint32_t minus, Cx<float> v) {
    const float sg = RZ ? flip_sign(g.s, ~minus) : g.s;   // bit 0 turns the other way
    const Cx<float> C = unpack2(mul2(pack2(g.c, g.c), pack2(v))), P = unpack2(mul2(pack2(sg, sg), pack2(v)));
    return Cx<float>{__fsub_rn(C.r, P.i), __fadd_rn(C.i, P.r)};
}
template <bool RZ>
__device__ __forceinline__ Cx<double> turn(const UGate<double>& g, uint32_t minus, Cx<double> v) {
    using A = Arith<double>;
    Cx<double> C, P;
    products<true>(g, v, C, P);
    if constexpr (RZ) return Cx<double>{A::add(C.r, flip_sign(P.i, minus)), A::add(C.i, flip_sign(P.r, ~minus))};
    else return Cx<double>{A::sub(C.r, P.i), A::add(C.i, P.r)};
}

// Diagonal gates: e has bit s set where the gate acts on slot s and its logical target bit is 1.
template <class T, uint32_t K, int S>
__device__ __forceinline__ void diag(const UGate<T>& g, unsigned e, unsigned act, Slots<T, S>& x) {
    if (K != KZ && !(K == KYPH || K == KRZ ? act : e)) return;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        Cx<T>& v = x.v[s];
        const uint32_t m = e << (31 - s);   // bit 31: logical target bit 1
        if constexpr (K == KZ) {
            v = Cx<T>{flip_sign(v.r, m), flip_sign(v.i, m)};
        } else if constexpr (K == KS || K == KSDG) {   // S: i * v, Sdg: -i * v
            if (e & (1u << s)) v = K == KSDG ? Cx<T>{v.i, neg(v.r)} : Cx<T>{neg(v.i), v.r};
        } else if constexpr (K == KYPH) {              // bit 1: i * v, bit 0: -i * v
            if (act & (1u << s)) v = Cx<T>{flip_sign(v.i, m), flip_sign(v.r, ~m)};
        } else if (K == KRZ ? (act & (1u << s)) : (e & (1u << s))) {
            v = turn<K == KRZ>(g, m, v);
        }
    }
}

// A gate with a coefficient that is not finite (an infinite or NaN angle). The forms above run absent
// slots along, as products of 0 are 0; here they would become NaN, and pairs without keys would get some. So
// presence is looked at: every pair with a key follows the formula, all others stay absent and 0.
// Only U can have finite rows beside others; every other result of such a gate is NaN. Passes with such
// a gate go to kernels of their own: as one more case in the ordinary ones, it cost FP32 passes 8 to 20% in
// spilled registers, though it never ran.
template <class T> __device__ __forceinline__ T u_coef(const GateDesc* gd, int i);
template <> __device__ __forceinline__ double u_coef<double>(const GateDesc* gd, int i) { return __ldg(&gd->m[i]); }
template <> __device__ __forceinline__ float u_coef<float>(const GateDesc* gd, int i) { return __ldg(&gd->mf[i]); }
template <class T, int S>
__device__ __forceinline__ Slots<T, S> odd_gate(const GateDesc* gd, uint32_t loc, uint32_t w, unsigned ones, Slots<T, S> x, PruneBits pb) {
    using A = Arith<T>;
    const uint32_t kind = __ldg(&gd->kind), form = (loc >> kLocOp) - UO_ODD;
    const T nan = (T)__int_as_float(0x7FC00000);
    const unsigned act = w & ((1u << S) - 1u);
    if (!branch_kind(kind)) {   // Rz, Phase
        const unsigned on = (kind == KRZ ? act : ones) & x.pm;
#pragma unroll
        for (int s = 0; s < S; ++s)
            if ((on >> s) & 1u) x.v[s] = Cx<T>{nan, nan};
        return x;
    }
    Cx<T> b[S];   // the partners
    unsigned pp;
    if (form == 1) {
        const int off = 1 << ((loc >> kLocBit) & 31u);
        pp = __shfl_xor_sync(kFull, x.pm, off);
#pragma unroll
        for (int s = 0; s < S; ++s) b[s] = shfl_cx(x.v[s], off);
    } else {
        const bool far = S == 4 && form == 2;
        pp = far ? (x.pm << 2) | (x.pm >> 2) : ((x.pm & 5u) << 1) | ((x.pm >> 1) & 5u);
#pragma unroll
        for (int s = 0; s < S; ++s) b[s] = S == 1 ? x.v[0] : pick(far, x.v[s ^ (S == 4 ? 2 : S - 1 & 1)], x.v[s ^ (S > 1)]);
    }
    const unsigned any = (x.pm | pp) & act;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (!((any >> s) & 1u)) continue;
        Cx<T> o{nan, nan};
        if (kind == KU) {
            const bool bit = ((w >> 31) != 0) != (form != 1 && (s & (form == 2 ? 2 : 1)));
            const int own = bit ? 6 : 0, mix = bit ? 4 : 2;
            const T sr = u_coef<T>(gd, own), si = u_coef<T>(gd, own + 1), mr = u_coef<T>(gd, mix), mi = u_coef<T>(gd, mix + 1);
            const Cx<T> a = x.v[s], c = b[s];
            o.r = A::fma(neg(mi), c.i, A::fma(mr, c.r, A::fma(neg(si), a.i, A::mul(sr, a.r))));
            o.i = A::fma(mi, c.r, A::fma(mr, c.i, A::fma(si, a.r, A::mul(sr, a.i))));
        }
        const bool keep = !negligible(o, pb);
        x.v[s] = pick(keep, o, czero<T>());
        x.pm = (x.pm & ~(1u << s)) | ((unsigned)keep << s);
    }
    x.n = __popc(x.pm);
    return x;
}

// The gates of a pass on the unit a warp holds; uid is the unit's base index. Absent slots hold
// +-0, and the prune threshold is positive: no gate makes a slot present out of absent ones.
// `heads` says where each gate acts (UnitHead): the gates' own in shared memory, or the kernel's
// parameters, where the whole warp reads them as one.
template <class T, int S, class Heads>
__device__ __forceinline__ void run_unit(const Heads& heads, const UGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t ng,
                                         uint32_t uid, int lane, Slots<T, S>& x, bool& touched,
                                         const PruneBits& pb, unsigned long long& upd) {
#pragma unroll 1
    for (uint32_t gi = 0; gi < ng; ++gi) {
        const UGate<T>& g = sg.g[gi];
        const UnitHead head = heads[gi];
        upd += (unsigned long long)x.n * head.weight;
        if ((uid & head.om) != head.ov) continue;   // a control outside the unit excludes all of it
        const uint32_t w = (uint32_t)(int)sg.lw[gi][lane];
        const uint32_t loc = head.loc;
        const GateDesc* gd = gates + gi;
        touched = true;
        const unsigned act = w & 15u;
        // diagonal gates: slots with logical target bit 1, the target's bit of the unit's base applied
        auto ones = [&]() {
            return ((w >> 4) & 15u) ^ (((uid >> ((loc >> kLocBit) & 31u)) & 1u) && !(loc & kLocLane) ? act : 0u);
        };
        switch (loc >> kLocOp) {
        case UO_X_PAIR: swap_pair<T, KX, S, 1, false>(w, x); break;
        case UO_X_SHFL: swap_shfl<T, KX, S, false>(loc, w, x); break;
        case UO_ALL + UO_X_PAIR: swap_pair<T, KX, S, 1, true>(w, x); break;
        case UO_ALL + UO_X_SHFL: swap_shfl<T, KX, S, true>(loc, w, x); break;
        case UO_PAIR3 + UO_X_PAIR:
            if constexpr (S == 4) swap_pair<T, KX, S, 2, false>(w, x);
            break;
        case UO_ALL3 + UO_X_PAIR:
            if constexpr (S == 4) swap_pair<T, KX, S, 2, true>(w, x);
            break;
        case UO_Y_PAIR: swap_pair<T, KY, S, 1, false>(w, x); break;
        case UO_Y_SHFL: swap_shfl<T, KY, S, false>(loc, w, x); break;
        case UO_ALL + UO_Y_PAIR: swap_pair<T, KY, S, 1, true>(w, x); break;
        case UO_ALL + UO_Y_SHFL: swap_shfl<T, KY, S, true>(loc, w, x); break;
        case UO_PAIR3 + UO_Y_PAIR:
            if constexpr (S == 4) swap_pair<T, KY, S, 2, false>(w, x);
            break;
        case UO_ALL3 + UO_Y_PAIR:
            if constexpr (S == 4) swap_pair<T, KY, S, 2, true>(w, x);
            break;
        case UO_H_PAIR: branch_pair<T, KH, S, 1, false>(g, gd, w, x, pb); break;
        case UO_H_SHFL: branch_shfl<T, KH, S, false>(g, gd, loc, w, x, pb); break;
        case UO_ALL + UO_H_PAIR: branch_pair<T, KH, S, 1, true>(g, gd, w, x, pb); break;
        case UO_ALL + UO_H_SHFL: branch_shfl<T, KH, S, true>(g, gd, loc, w, x, pb); break;
        case UO_PAIR3 + UO_H_PAIR:
            if constexpr (S == 4) branch_pair<T, KH, S, 2, false>(g, gd, w, x, pb);
            break;
        case UO_ALL3 + UO_H_PAIR:
            if constexpr (S == 4) branch_pair<T, KH, S, 2, true>(g, gd, w, x, pb);
            break;
        case UO_RX_PAIR: branch_pair<T, KRX, S, 1, false>(g, gd, w, x, pb); break;
        case UO_RX_SHFL: branch_shfl<T, KRX, S, false>(g, gd, loc, w, x, pb); break;
        case UO_ALL + UO_RX_PAIR: branch_pair<T, KRX, S, 1, true>(g, gd, w, x, pb); break;
        case UO_ALL + UO_RX_SHFL: branch_shfl<T, KRX, S, true>(g, gd, loc, w, x, pb); break;
        case UO_PAIR3 + UO_RX_PAIR:
            if constexpr (S == 4) branch_pair<T, KRX, S, 2, false>(g, gd, w, x, pb);
            break;
        case UO_ALL3 + UO_RX_PAIR:
            if constexpr (S == 4) branch_pair<T, KRX, S, 2, true>(g, gd, w, x, pb);
            break;
        case UO_RY_PAIR: branch_pair<T, KRY, S, 1, false>(g, gd, w, x, pb); break;
        case UO_RY_SHFL: branch_shfl<T, KRY, S, false>(g, gd, loc, w, x, pb); break;
        case UO_ALL + UO_RY_PAIR: branch_pair<T, KRY, S, 1, true>(g, gd, w, x, pb); break;
        case UO_ALL + UO_RY_SHFL: branch_shfl<T, KRY, S, true>(g, gd, loc, w, x, pb); break;
        case UO_PAIR3 + UO_RY_PAIR:
            if constexpr (S == 4) branch_pair<T, KRY, S, 2, false>(g, gd, w, x, pb);
            break;
        case UO_ALL3 + UO_RY_PAIR:
            if constexpr (S == 4) branch_pair<T, KRY, S, 2, true>(g, gd, w, x, pb);
            break;
        case UO_U_PAIR: branch_pair<T, KU, S, 1, false>(g, gd, w, x, pb); break;
        case UO_U_SHFL: branch_shfl<T, KU, S, false>(g, gd, loc, w, x, pb); break;
        case UO_ALL + UO_U_PAIR: branch_pair<T, KU, S, 1, true>(g, gd, w, x, pb); break;
        case UO_ALL + UO_U_SHFL: branch_shfl<T, KU, S, true>(g, gd, loc, w, x, pb); break;
        case UO_PAIR3 + UO_U_PAIR:
            if constexpr (S == 4) branch_pair<T, KU, S, 2, false>(g, gd, w, x, pb);
            break;
        case UO_ALL3 + UO_U_PAIR:
            if constexpr (S == 4) branch_pair<T, KU, S, 2, true>(g, gd, w, x, pb);
            break;
        case UO_Z: diag<T, KZ, S>(g, ones(), act, x); break;
        case UO_S: diag<T, KS, S>(g, ones(), act, x); break;
        case UO_SDG: diag<T, KSDG, S>(g, ones(), act, x); break;
        case UO_YPH: diag<T, KYPH, S>(g, ones(), act, x); break;
        case UO_RZ: diag<T, KRZ, S>(g, ones(), act, x); break;
        case UO_PHASE: diag<T, KPHASE, S>(g, ones(), act, x); break;
        default:
            if constexpr (kOddHeads<Heads>) x = odd_gate<T, S>(gd, loc, w, ones(), x, pb);
            else __builtin_unreachable();
        }
    }
}

// Base bucket of unit u: zeros inserted at the (ascending) bits lo[0..DIMS-1].
template <int DIMS>
__device__ __forceinline__ unsigned unit_base(unsigned u, const uint32_t (&lo)[3]) {
#pragma unroll
    for (int d = 0; d < DIMS; ++d) u = ((u >> lo[d]) << (lo[d] + 1)) | (u & ((1u << lo[d]) - 1u));
    return u;
}

// What a pass over units needs besides its gates.
struct UnitPass {
    uint32_t dim[3];    // bucket bit of each dimension
    uint32_t lo[3];     // the same, ascending
    uint32_t units;     // units that enumerate the table's 2^dn buckets
};

template <int DIMS>
__device__ __forceinline__ UnitPass unit_pass(uint32_t dn, uint32_t d0, uint32_t d1, uint32_t d2) {
    UnitPass p;
    p.dim[0] = d0; p.dim[1] = d1; p.dim[2] = DIMS == 3 ? d2 : 31u;
    uint32_t a = d0 < d1 ? d0 : d1, b = d0 < d1 ? d1 : d0, c = p.dim[2];
    if (c < b) { const uint32_t x = b; b = c; c = x; }
    if (b < a) { const uint32_t x = a; a = b; b = x; }
    p.lo[0] = a; p.lo[1] = b; p.lo[2] = c;
    uint32_t in = (d0 < dn) + (d1 < dn) + (DIMS == 3 && d2 < dn);   // dimensions within the mapped bits
    p.units = 1u << (dn - in);
    return p;
}

// (t's map is read through mq: a pass over many circuits leaves it in memory.)
// One unit: load, apply the gates, write back. Absent buckets are created (header, keys, list
// entry) when a key of theirs becomes present; the unit is this warp's alone, so plain stores do.
template <class T, int DIMS, class Heads>
__device__ __forceinline__ void do_unit(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up, unsigned base,
                                        const Heads& heads, const UGates<T>& sg, const GateDesc* gates, uint32_t ng, int lane,
                                        const PruneBits& pb, unsigned long long& cnt_nnz, unsigned long long& cnt_empty,
                                        unsigned long long& upd) {
    constexpr int S = 1 << (DIMS - 1);
    const int j = lane & 15;
    const unsigned b0 = base | ((unsigned)(lane >> 4) << up.dim[1]);
    unsigned bk[S];
    Slots<T, S> x;
    // lane k < 2^DIMS reads member k's header; a unit whose buckets are all live and full (every unit,
    // in a state that fills its span) needs nothing more of them
    constexpr unsigned kMembers = 1u << DIMS;
    uint2 hk = make_uint2(ep, 0xFFFFu);
    if (lane < (int)kMembers) {
        unsigned b = base;
#pragma unroll
        for (int d = 0; d < DIMS; ++d) b |= (((unsigned)lane >> d) & 1u) << up.dim[d];
        hk = __ldcg(reinterpret_cast<const uint2*>(&t.hdr[b].epoch));
    }
#pragma unroll
    for (int s = 0; s < S; ++s) {
        bk[s] = b0 | ((s & 1) ? 1u << up.dim[0] : 0u) | ((s & 2) ? 1u << up.dim[2] : 0u);
        const typename AmpT<T>::V a =
            __ldcg(reinterpret_cast<const typename AmpT<T>::V*>(t.amps) + (size_t)bk[s] * kSlots + j);
        x.v[s] = Cx<T>{a.x, a.y};
    }
    uint2 h[S];
    const bool full = __all_sync(kFull, hk.x == ep && hk.y == 0xFFFFu);
    x.pm = (1u << S) - 1u;
    if (!full) {
        x.pm = 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const int m = (s & 1) | ((lane >> 4) << 1) | ((s & 2) << 1);
            h[s] = make_uint2(__shfl_sync(kFull, hk.x, m), __shfl_sync(kFull, hk.y, m));
            const bool p = h[s].x == ep && ((h[s].y >> j) & 1u);
            x.pm |= (unsigned)p << s;
            x.v[s] = pick(p, x.v[s], czero<T>());
        }
    } else {
#pragma unroll
        for (int s = 0; s < S; ++s) h[s] = make_uint2(ep, 0xFFFFu);
    }
    bool touched = false;
    const unsigned pm0 = x.pm;
    x.n = __popc(pm0);
    if (full || __any_sync(kFull, pm0 != 0)) run_unit<T, S>(heads, sg, gates, ng, base, lane, x, touched, pb, upd);
    const unsigned pm = x.pm;
    cnt_nnz += __popc(pm);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const bool p = (pm >> s) & 1u;
        if (touched && p)
            store_amp<T>(t.amps, (size_t)bk[s] * kSlots + j, x.v[s]);
    }
    if (__any_sync(kFull, pm != pm0)) {
        // presence changed somewhere in the unit: headers, keys, the list
        unsigned mk[S], fresh = 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned bal = __ballot_sync(kFull, (pm >> s) & 1u);
            mk[s] = lane >= 16 ? bal >> 16 : bal & 0xFFFFu;
            const bool live = h[s].x == ep, make = !live && mk[s] != 0;
            if (live ? mk[s] != h[s].y : make) {
                const unsigned long long G = group_of_bucket(t.map_n, mq, bk[s]);
                const bool p = (pm >> s) & 1u;
                if (make || p != (((pm0 >> s) & 1u) != 0))
                    t.keys[(size_t)bk[s] * kSlots + j] = p ? (G << kSlotBits) | (unsigned)j : empty_key(j);
                if (j == 0) {
                    ulonglong2 w;
                    w.x = G;
                    w.y = (unsigned long long)ep | ((unsigned long long)mk[s] << 32);
                    *reinterpret_cast<ulonglong2*>(t.hdr + bk[s]) = w;
                    if (make) fresh |= 1u << s;
                }
            }
            if (j == 0 && mk[s] == 0 && live) cnt_empty += 1;
        }
        if (__any_sync(kFull, fresh != 0)) {
            const unsigned m = __popc(fresh);
            const unsigned hi = __shfl_sync(kFull, m, 16), lo = __shfl_sync(kFull, m, 0);
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(&ctl->list_tail, (unsigned long long)(lo + hi));
            at = shfl64(at, 0) + (lane >= 16 ? lo : 0u);
#pragma unroll
            for (int s = 0; s < S; ++s)
                if ((fresh >> s) & 1u) t.list[at++] = bk[s];
        }
    } else if (!full) {
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (j == 0 && h[s].x == ep && h[s].y == 0) cnt_empty += 1;
    }
}

// A warp's share of a pass over all `units` units, dealt in rounds of one to each of nw warps. The deal
// turns by an odd number of places every round: in place, a warp would meet the same low bits of
// the unit index in every round (nw has many factors of two), and a gate controlled there would leave
// some warps without work and others with all of it. (500 gates on 2^24 keys, FP64: 21.2 -> 19.7 ms; 1000
// on 2^22, FP32, scheduled: 2.49 -> 2.23 ms.)
template <class T, int DIMS, class Heads>
__device__ __forceinline__ void walk_all_units(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up,
                                               unsigned w, unsigned nw, const Heads& heads, const UGates<T>& sg, const GateDesc* gates, uint32_t ng, int lane,
                                               const PruneBits& pb, unsigned long long& cnt_nnz,
                                               unsigned long long& cnt_empty, unsigned long long& upd) {
    const unsigned turn = ((nw * 79u) >> 7) | 1u;   // (no overflow: nw is at most a few thousand; nw = 1 turns by a whole round)
    unsigned at = w;
    for (unsigned r = 0; r < up.units; r += nw) {   // (at most 2^29 units: no wrap)
        if (r + at < up.units)
            do_unit<T, DIMS>(t, mq, ctl, ep, up, unit_base<DIMS>(r + at, up.lo), heads, sg, gates, ng, lane, pb, cnt_nnz, cnt_empty, upd);
        at += turn;
        if (at >= nw) at -= nw;
    }
}

// Units [u0, u1) step `stride` of a table whose live buckets fill it.
template <class T, int DIMS, class Heads>
__device__ __forceinline__ void walk_units(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up,
                                           unsigned u0, unsigned u1, unsigned stride, const Heads& heads, const UGates<T>& sg, const GateDesc* gates, uint32_t ng, int lane,
                                           const PruneBits& pb, unsigned long long& cnt_nnz,
                                           unsigned long long& cnt_empty, unsigned long long& upd) {
    for (unsigned u = u0; u < u1; u += stride)   // (at most 2^29 units: no wrap)
        do_unit<T, DIMS>(t, mq, ctl, ep, up, unit_base<DIMS>(u, up.lo), heads, sg, gates, ng, lane, pb, cnt_nnz, cnt_empty,
                         upd);
}

// List entries a warp takes at a time, for n entries and nw warps: up to 32, as many pieces to every warp.
// Few entries make small pieces: the units of a piece run one after another in a mapped pass (2^11
// keys, FP32: 27 -> 5 us a pass), and a piece is a chain of dependent loads in any.
__device__ __forceinline__ unsigned long long list_piece(unsigned long long n, unsigned nw) {
    const unsigned long long rounds = (n + nw * 32ULL - 1) / (nw * 32ULL);
    return rounds ? (n + nw * rounds - 1) / (nw * rounds) : 1;
}

// The units of list entries [e0, e1) (at most 32), for tables whose live buckets are few among
// the mapped ones: lane l takes entry e0 + l; the unit belongs to its live member of smallest index
// (members a pass creates are made by the unit's owner, after its own check), found by reading
// the headers of the smaller members.
template <class T, int DIMS, class Heads>
__device__ __forceinline__ void walk_entries(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up,
                                             unsigned long long e0, unsigned long long e1, const Heads& heads, const UGates<T>& sg,
                                             const GateDesc* gates, uint32_t ng, int lane, const PruneBits& pb,
                                             unsigned long long& cnt_nnz, unsigned long long& cnt_empty,
                                             unsigned long long& upd) {
    constexpr int K = 1 << DIMS;
    unsigned base = 0;
    bool own = false;
    if (e0 + lane < e1) {
        const unsigned b = __ldcg(t.list + e0 + lane);   // (an earlier pass of the same launch may have written it)
        int idx = 0;
        base = b;
#pragma unroll
        for (int d = 0; d < DIMS; ++d) {
            idx |= (int)((b >> up.dim[d]) & 1u) << d;
            base &= ~(1u << up.dim[d]);
        }
        own = true;
        for (int k = 0; k < K && k < idx && own; ++k) {
            unsigned m = base;
#pragma unroll
            for (int d = 0; d < DIMS; ++d) m |= (unsigned)((k >> d) & 1) << up.dim[d];
            own = __ldcg(&t.hdr[m].epoch) != ep;
        }
    }
    unsigned todo = __ballot_sync(kFull, own);
    while (todo) {
        const int l = __ffs(todo) - 1;
        todo &= todo - 1;
        do_unit<T, DIMS>(t, mq, ctl, ep, up, __shfl_sync(kFull, base, l), heads, sg, gates, ng, lane, pb, cnt_nnz, cnt_empty, upd);
    }
}

// Whether a pass walks the list (live buckets below an eighth of the mapped ones) or every unit:
// a unit without keys costs its headers and amplitudes (about an eighth of a unit of a ten-gate
// pass), a list entry its ownership check.
__device__ __forceinline__ bool walk_list(unsigned long long list_n, uint32_t dn) {
    return dn >= 6 && list_n < (1ULL << (dn - 3));
}

// ---- hashed tables -------------------------------------------------------------------------------
// Keys too thin for a map: most groups hold one key among their 16 slots, and a warp per unit would
// run every gate on lanes without one. A pass here pairs keys across at most two qubits, the low four
// included, and splits its units into columns: the four keys that differ in those qubits, all in
// one lane, so gates need no exchange between lanes and 32 columns of any units run together. A warp takes
// a piece of the live list. Each lane looks up the members of one entry's unit and settles
// whether the entry owns it; the presence masks (Header.aux) come with the lookups. The columns of the
// owned units that hold a key are then dealt to the lanes, 32 at a time; only amplitudes of
// present keys are read. Controls and diagonal targets outside the column are tested per lane.
// 2^17 keys in FP64, one or two to a group: 285 us a pass with a warp per unit (and 335 us by pairs of
// slots with their keys), see hash_kernel for this form.
constexpr int kColumn = 4;   // keys of a column

// A pass's gate in shared memory.
template <class T> struct HGates {
    UGate<T> g[kMaxRun];
    unsigned long long om[kMaxRun], ov[kMaxRun];   // controls outside the column
};

// Where a pass's two qubits lie: group masks, or slot masks of the low four (both 0: no such qubit).
struct HashDims {
    unsigned long long gm[2], keys;   // keys: both as key bits
    unsigned lm[2];
    unsigned groups, valid;           // column bits that change the group, that exist
};
__device__ __forceinline__ HashDims hash_dims(uint32_t d0, uint32_t d1) {
    HashDims r;
    const uint32_t d[2] = {d0, d1};
    r.keys = 0;
    r.groups = r.valid = 0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        r.gm[i] = d[i] >= (uint32_t)kSlotBits && d[i] < 64u ? 1ULL << (d[i] - kSlotBits) : 0ULL;
        r.lm[i] = d[i] < (uint32_t)kSlotBits ? 1u << d[i] : 0u;
        if (d[i] < 64u) r.keys |= 1ULL << d[i];
        if (r.gm[i]) r.groups |= 1u << i;
        if (d[i] < 64u) r.valid |= 1u << i;
    }
    return r;
}

// Copy ng gates into shared memory for a pass with pairing qubits dk (key bits); no barrier.
template <class T>
__device__ __forceinline__ void stage_hgates(HGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t ng, unsigned long long dk) {
    for (uint32_t i = threadIdx.x; i < ng; i += blockDim.x) {
        const GateDesc* g = gates + i;
        stage_ugate(sg.g + i, g);
        const unsigned long long om = __ldg(&g->ctrl) & ~dk;
        sg.om[i] = om;
        sg.ov[i] = __ldg(&g->cval) & om;
    }
}

// A warp's piece of a pass: per list entry the members of its unit (bucket, kNoBucket when absent, and
// presence mask before the pass), their masks now, and the columns that hold keys (entry << 4 | slot).
struct HashWork {
    uint2 m[32][4];
    unsigned now[32][4];
    unsigned short cols[512];
};

// The gates of a pass on one column a lane; kb is the column's key with the pass's qubits 0. ODD: some may be
// UO_ODD gates.
template <class T, bool ODD>
__device__ __forceinline__ void run_columns(const HGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t ng, unsigned long long kb,
                                            bool on, Slots<T, kColumn>& x, bool& touched, const PruneBits& pb,
                                            unsigned long long& upd) {
#pragma unroll 1
    for (uint32_t gi = 0; gi < ng; ++gi) {
        const UGate<T>& g = sg.g[gi];
        upd += (unsigned long long)x.n * g.weight;
        const uint32_t loc = g.loc;
        const bool acts = on && (kb & sg.om[gi]) == sg.ov[gi];
        if (!__any_sync(kFull, acts)) continue;
        touched = touched || acts;
        const GateDesc* gd = gates + gi;
        const unsigned act = acts ? (loc >> kLocSlots) & 15u : 0u;
        const uint32_t w = act | (loc & kLocFlip ? 0x80000000u : 0u);   // pairing gates: slots, logical bit of the first
        auto ones = [&]() {   // diagonal gates: slots with logical target bit 1
            const uint32_t word = loc & kLocHigh ? (uint32_t)(kb >> 32) : (uint32_t)kb;
            const bool at = !(loc & kLocLane) && ((word >> ((loc >> kLocBit) & 31u)) & 1u);
            return (((loc >> kLocSlotBit) & 15u) ^ (at ? 15u : 0u)) & act;
        };
        switch (loc >> kLocOp) {
        case UO_X_PAIR: swap_pair<T, KX, kColumn, 1, false>(w, x); break;
        case UO_PAIR3 + UO_X_PAIR: swap_pair<T, KX, kColumn, 2, false>(w, x); break;
        case UO_Y_PAIR: swap_pair<T, KY, kColumn, 1, false>(w, x); break;
        case UO_PAIR3 + UO_Y_PAIR: swap_pair<T, KY, kColumn, 2, false>(w, x); break;
        case UO_H_PAIR: branch_pair<T, KH, kColumn, 1, false>(g, gd, w, x, pb); break;
        case UO_PAIR3 + UO_H_PAIR: branch_pair<T, KH, kColumn, 2, false>(g, gd, w, x, pb); break;
        case UO_RX_PAIR: branch_pair<T, KRX, kColumn, 1, false>(g, gd, w, x, pb); break;
        case UO_PAIR3 + UO_RX_PAIR: branch_pair<T, KRX, kColumn, 2, false>(g, gd, w, x, pb); break;
        case UO_RY_PAIR: branch_pair<T, KRY, kColumn, 1, false>(g, gd, w, x, pb); break;
        case UO_PAIR3 + UO_RY_PAIR: branch_pair<T, KRY, kColumn, 2, false>(g, gd, w, x, pb); break;
        case UO_U_PAIR: branch_pair<T, KU, kColumn, 1, false>(g, gd, w, x, pb); break;
        case UO_PAIR3 + UO_U_PAIR: branch_pair<T, KU, kColumn, 2, false>(g, gd, w, x, pb); break;
        case UO_Z: diag<T, KZ, kColumn>(g, ones(), act, x); break;
        case UO_S: diag<T, KS, kColumn>(g, ones(), act, x); break;
        case UO_SDG: diag<T, KSDG, kColumn>(g, ones(), act, x); break;
        case UO_YPH: diag<T, KYPH, kColumn>(g, ones(), act, x); break;
        case UO_RZ: diag<T, KRZ, kColumn>(g, ones(), act, x); break;
        case UO_PHASE: diag<T, KPHASE, kColumn>(g, ones(), act, x); break;
        default:
            if constexpr (ODD) x = odd_gate<T, kColumn>(gd, loc, w, ones(), x, pb);
            else __builtin_unreachable();
        }
    }
}

// The units of list entries [e0, e1) (at most 32). An entry owns its unit when it is the live member of
// smallest index (the reference's pair rule, emulator/device/device_table_FC.cuh:62-110, lifted to
// groups; members a pass creates are made by the unit's owner, after its own check).
template <class T, bool ODD>
__device__ __forceinline__ void walk_hashed(const TableDev& t, Ctl* ctl, unsigned ep, const HashDims& dm, unsigned long long e0,
                                            unsigned long long e1, HashWork& wk, const HGates<T>& sg, const GateDesc* gates,
                                            uint32_t ng, int lane, const PruneBits& pb, unsigned long long& cnt_nnz,
                                            unsigned long long& cnt_empty, unsigned long long& upd) {
    unsigned long long base = 0;
    bool owns = false;
    unsigned cols = 0;
    auto member = [&](unsigned long long G0, int k) { return G0 | ((k & 1) ? dm.gm[0] : 0ULL) | ((k & 2) ? dm.gm[1] : 0ULL); };
    if (e0 + lane < e1) {
        const unsigned b = __ldcg(t.list + e0 + lane);   // (an earlier pass of the same launch may have written it)
        const Header own = load_hdr_cg(t.hdr + b);
        const int idx = ((own.group & dm.gm[0]) ? 1 : 0) | ((own.group & dm.gm[1]) ? 2 : 0);
        base = own.group & ~(dm.gm[0] | dm.gm[1]);
        Header h[4];
        unsigned at[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {   // the first probes of all members together
            h[k].epoch = ep + 1;
            at[k] = b;
            if (k != idx && (k & ~dm.groups) == 0) {
                at[k] = (unsigned)(mix64(member(base, k)) & t.mask);
                h[k] = load_hdr_cg(t.hdr + at[k]);
            }
        }
        owns = true;
        unsigned any = own.aux;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint2 m = make_uint2(kNoBucket, 0u);
            if (k == idx) {
                m = make_uint2(b, own.aux);
            } else if (h[k].epoch == ep) {
                const unsigned long long G = member(base, k);
                Header c = h[k];
                unsigned long long p = at[k];
                for (uint32_t i = 1; i < kMaxProbe && c.epoch == ep && c.group != G; ++i) {
                    p = (p + 1) & t.mask;
                    c = load_hdr_cg(t.hdr + p);
                }
                if (c.epoch == ep && c.group == G) {
                    m = make_uint2((unsigned)p, c.aux);
                    if (k < idx) owns = false;
                    any |= c.aux;
                }
            }
            wk.m[lane][k] = m;
            wk.now[lane][k] = m.y;
        }
        if (owns) {   // its columns: slots with the pass's low qubits 0
            cols = any;
#pragma unroll
            for (int d = 0; d < 2; ++d) {
                const unsigned q = dm.lm[d];
                if (q) cols = (cols | (cols >> q)) & (q == 1 ? 0x5555u : q == 2 ? 0x3333u : q == 4 ? 0x0F0Fu : 0x00FFu);
            }
        }
    }
    unsigned upto = __popc(cols);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned v = __shfl_up_sync(kFull, upto, o);
        if (lane >= o) upto += v;
    }
    const unsigned total = __shfl_sync(kFull, upto, 31);
    {
        unsigned at = upto - __popc(cols);
        for (unsigned c = cols; c; c &= c - 1) wk.cols[at++] = (unsigned short)((lane << 4) | (__ffs(c) - 1));
    }
    __syncwarp();
    unsigned fresh = 0;   // members of this lane's entry that the pass has made
    for (unsigned c0 = 0; c0 < total; c0 += 32) {
        const bool on = c0 + lane < total;
        const unsigned id = on ? wk.cols[c0 + lane] : 0u;
        const int l = (int)(id >> 4);
        const unsigned j0 = id & 15u;
        const unsigned long long G0 = shfl64(base, l);
        Slots<T, kColumn> x;
        x.pm = 0;
#pragma unroll
        for (int s = 0; s < kColumn; ++s) {
            const unsigned j = j0 | ((s & 1) ? dm.lm[0] : 0u) | ((s & 2) ? dm.lm[1] : 0u);
            const uint2 m = wk.m[l][s & dm.groups];
            const bool p = on && (s & ~dm.valid) == 0 && ((m.y >> j) & 1u);
            x.pm |= (unsigned)p << s;
            x.v[s] = czero<T>();
            if (p) {
                const typename AmpT<T>::V a = __ldcg(reinterpret_cast<const typename AmpT<T>::V*>(t.amps) + (size_t)m.x * kSlots + j);
                x.v[s] = Cx<T>{a.x, a.y};
            }
        }
        bool touched = false;
        const unsigned pm0 = x.pm;
        x.n = __popc(pm0);
        run_columns<T, ODD>(sg, gates, ng, (G0 << kSlotBits) | j0, on, x, touched, pb, upd);
        const unsigned pm = x.pm;
        cnt_nnz += __popc(pm);
        bool absent = false;
#pragma unroll
        for (int s = 0; s < kColumn; ++s) {
            if (!(((pm ^ pm0) >> s) & 1u)) continue;
            const unsigned j = j0 | ((s & 1) ? dm.lm[0] : 0u) | ((s & 2) ? dm.lm[1] : 0u);
            if ((pm >> s) & 1u) {
                atomicOr(&wk.now[l][s & dm.groups], 1u << j);
                absent = absent || wk.m[l][s & dm.groups].x == kNoBucket;
            } else {
                atomicAnd(&wk.now[l][s & dm.groups], ~(1u << j));
            }
        }
        if (__any_sync(kFull, absent)) {   // groups that appear: claimed by the lane of their unit's entry
            __syncwarp();
            if (owns) {
#pragma unroll 1
                for (int k = 0; k < 4; ++k) {
                    if (wk.m[lane][k].x != kNoBucket || wk.now[lane][k] == 0) continue;
                    bool created;
                    const long long nb = claim_group(t, ep, member(base, k), &ctl->status, &created);
                    if (nb < 0) continue;
                    wk.m[lane][k].x = (unsigned)nb;
                    fresh |= 1u << k;
                    ulonglong2* keys = reinterpret_cast<ulonglong2*>(t.keys + (size_t)nb * kSlots);
#pragma unroll
                    for (int j = 0; j < kSlots; j += 2) keys[j / 2] = make_ulonglong2(empty_key(j), empty_key(j + 1));
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int s = 0; s < kColumn; ++s) {
            const bool p = (pm >> s) & 1u, moved = ((pm ^ pm0) >> s) & 1u;
            if (!moved && !(p && touched)) continue;
            const unsigned j = j0 | ((s & 1) ? dm.lm[0] : 0u) | ((s & 2) ? dm.lm[1] : 0u);
            const unsigned b = wk.m[l][s & dm.groups].x;
            if (b == kNoBucket) continue;   // (the table is full: the pass has failed)
            if (p) store_amp<T>(t.amps, (size_t)b * kSlots + j, x.v[s]);
            if (moved) t.keys[(size_t)b * kSlots + j] = p ? (member(G0, s & (int)dm.groups) << kSlotBits) | j : empty_key((int)j);
        }
    }
    __syncwarp();
    // masks that changed, and the buckets made: those go to the list together, with one addition to its
    // length (every warp adds to it)
    if (owns) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint2 m = wk.m[lane][k];
            if (m.x == kNoBucket) continue;
            const unsigned now = wk.now[lane][k];
            if (now != m.y) t.hdr[m.x].aux = now;
            if (now == 0) cnt_empty += 1;
        }
    }
    if (__any_sync(kFull, fresh != 0)) {
        const unsigned made = __popc(fresh);
        unsigned sum = made;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(kFull, sum, o);
            if (lane >= o) sum += v;
        }
        unsigned long long at = 0;
        if (lane == 31) at = atomicAdd(&ctl->list_tail, (unsigned long long)sum);
        at = shfl64(at, 31) + (sum - made);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((fresh >> k) & 1u) t.list[at++] = wk.m[lane][k].x;
    }
    __syncwarp();
}

// A hashed pass's share of a warp.
template <class T, bool ODD = false>
__device__ __forceinline__ void walk_hashed_all(const TableDev& t, Ctl* ctl, unsigned ep, const HashDims& dm, unsigned long long n,
                                                unsigned w, unsigned nw, HashWork& wk, const HGates<T>& sg,
                                                const GateDesc* gates, uint32_t ng, int lane, const PruneBits& pb,
                                                unsigned long long& cnt_nnz, unsigned long long& cnt_empty, unsigned long long& upd) {
    const unsigned long long piece = list_piece(n, nw);
    for (unsigned long long e0 = w * piece; e0 < n; e0 += nw * piece)
        walk_hashed<T, ODD>(t, ctl, ep, dm, e0, umin64(e0 + piece, n), wk, sg, gates, ng, lane, pb, cnt_nnz, cnt_empty, upd);
}

// ---- slot passes over hashed tables ---------------------------------------------------------------
// A column pass pairs across two qubits. Gates that go back and forth between more of them, the four low ones
// above all, would take a pass for every few gates; a slot pass takes any number on qubits 0..3 and on up to three
// cross-group ones. Its units are whole: the 16 slots of each of the 2^nx groups that differ in the cross-group
// qubits, a lane per slot. The first cross-group qubit is lane bit 4 (without one, a warp holds two units), the
// next two pair the S = 1, 2 or 4 slots of a lane. Absent slots are run along: the host takes this form
// where it spares column passes, or where a state is so small that lanes are idle anyway (plan_hashed).
constexpr int kSlotMembers = 8;   // groups of a unit at most
struct SlotWork {
    uint2 m[32][kSlotMembers];    // as HashWork::m
};

// Op codes that pair the slots of a lane.
constexpr unsigned long long kSlotLocal = (1ULL << UO_X_PAIR) | (1ULL << UO_Y_PAIR) | (1ULL << UO_H_PAIR) | (1ULL << UO_RX_PAIR) |
                                          (1ULL << UO_RY_PAIR) | (1ULL << UO_U_PAIR) |
                                          (1ULL << (UO_PAIR3 + UO_X_PAIR)) | (1ULL << (UO_PAIR3 + UO_Y_PAIR)) |
                                          (1ULL << (UO_PAIR3 + UO_H_PAIR)) | (1ULL << (UO_PAIR3 + UO_RX_PAIR)) |
                                          (1ULL << (UO_PAIR3 + UO_RY_PAIR)) | (1ULL << (UO_PAIR3 + UO_U_PAIR)) | (7ULL << UO_ODD);

// The gates of a slot pass on the S slots of a lane; kb is the key of the lane's first slot.
template <class T, int S, bool ODD>
__device__ __forceinline__ void run_slots(const HGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t ng, unsigned long long kb,
                                          int lane, bool on, Slots<T, S>& x, bool& touched, const PruneBits& pb,
                                          unsigned long long& upd) {
#pragma unroll 1
    for (uint32_t gi = 0; gi < ng; ++gi) {
        const UGate<T>& g = sg.g[gi];
        upd += (unsigned long long)x.n * g.weight;
        const bool acts = on && (kb & sg.om[gi]) == sg.ov[gi];
        // a slot that no acting lane has a key in stays absent, but for gates that pair the slots of a lane
        unsigned live = 0;
        if constexpr (S == 1) live = __any_sync(kFull, acts && x.pm) ? 1u : 0u;
        else live = __reduce_or_sync(kFull, acts ? x.pm : 0u);
        if (!live) continue;
        uint32_t loc = g.loc;
        if (S > 1 && !(kSlotLocal >> (loc >> kLocOp) & 1ULL)) loc &= ~((~live & 15u) << kLocSlots);
        touched = touched || acts;
        const GateDesc* gd = gates + gi;
        const unsigned act = acts ? (loc >> kLocSlots) & 15u : 0u;
        const uint32_t w = act | (loc & kLocFlip ? 0x80000000u : 0u);            // pairs of slots: the logical bit of the first
        const uint32_t wl = w ^ (((uint32_t)lane >> ((loc >> kLocBit) & 31u)) << 31);   // pairs of lanes: that of the lane
        auto ones = [&]() {   // diagonal gates: slots with logical target bit 1
            const uint32_t word = loc & kLocHigh ? (uint32_t)(kb >> 32) : (uint32_t)kb;
            const bool at = !(loc & kLocLane) && ((word >> ((loc >> kLocBit) & 31u)) & 1u);
            return (((loc >> kLocSlotBit) & 15u) ^ (at ? 15u : 0u)) & act;
        };
        switch (loc >> kLocOp) {
        case UO_X_SHFL: swap_shfl<T, KX, S, false>(loc, wl, x); break;
        case UO_Y_SHFL: swap_shfl<T, KY, S, false>(loc, wl, x); break;
        case UO_H_SHFL: branch_shfl<T, KH, S, false>(g, gd, loc, wl, x, pb); break;
        case UO_RX_SHFL: branch_shfl<T, KRX, S, false>(g, gd, loc, wl, x, pb); break;
        case UO_RY_SHFL: branch_shfl<T, KRY, S, false>(g, gd, loc, wl, x, pb); break;
        case UO_U_SHFL: branch_shfl<T, KU, S, false>(g, gd, loc, wl, x, pb); break;
        case UO_Z: diag<T, KZ, S>(g, ones(), act, x); break;
        case UO_S: diag<T, KS, S>(g, ones(), act, x); break;
        case UO_SDG: diag<T, KSDG, S>(g, ones(), act, x); break;
        case UO_YPH: diag<T, KYPH, S>(g, ones(), act, x); break;
        case UO_RZ: diag<T, KRZ, S>(g, ones(), act, x); break;
        case UO_PHASE: diag<T, KPHASE, S>(g, ones(), act, x); break;
        default:
            if constexpr (ODD)
                if (loc >> kLocOp >= UO_ODD) {
                    x = odd_gate<T, S>(gd, loc, loc >> kLocOp == UO_ODD + 1 ? wl : w, ones(), x, pb);
                    break;
                }
            if constexpr (S > 1) {
                switch (loc >> kLocOp) {
                case UO_X_PAIR: swap_pair<T, KX, S, 1, false>(w, x); break;
                case UO_Y_PAIR: swap_pair<T, KY, S, 1, false>(w, x); break;
                case UO_H_PAIR: branch_pair<T, KH, S, 1, false>(g, gd, w, x, pb); break;
                case UO_RX_PAIR: branch_pair<T, KRX, S, 1, false>(g, gd, w, x, pb); break;
                case UO_RY_PAIR: branch_pair<T, KRY, S, 1, false>(g, gd, w, x, pb); break;
                case UO_U_PAIR: branch_pair<T, KU, S, 1, false>(g, gd, w, x, pb); break;
                default:
                    if constexpr (S == 4) {
                        switch (loc >> kLocOp) {
                        case UO_PAIR3 + UO_X_PAIR: swap_pair<T, KX, S, 2, false>(w, x); break;
                        case UO_PAIR3 + UO_Y_PAIR: swap_pair<T, KY, S, 2, false>(w, x); break;
                        case UO_PAIR3 + UO_H_PAIR: branch_pair<T, KH, S, 2, false>(g, gd, w, x, pb); break;
                        case UO_PAIR3 + UO_RX_PAIR: branch_pair<T, KRX, S, 2, false>(g, gd, w, x, pb); break;
                        case UO_PAIR3 + UO_RY_PAIR: branch_pair<T, KRY, S, 2, false>(g, gd, w, x, pb); break;
                        case UO_PAIR3 + UO_U_PAIR: branch_pair<T, KU, S, 2, false>(g, gd, w, x, pb); break;
                        default: __builtin_unreachable();
                        }
                    } else {
                        __builtin_unreachable();
                    }
                }
            } else {
                __builtin_unreachable();
            }
        }
    }
}

// The units of list entries [e0, e1) (at most 32) of a pass with cross-group bits gm (nx of them, S = 1 for
// nx <= 1, else 2^(nx - 1)).
template <class T, int S, bool ODD>
__device__ __forceinline__ void walk_slots(const TableDev& t, Ctl* ctl, unsigned ep, const unsigned long long (&gm)[3], uint32_t nx,
                                           unsigned long long e0, unsigned long long e1, SlotWork& wk, const HGates<T>& sg,
                                           const GateDesc* gates, uint32_t ng, int lane, const PruneBits& pb,
                                           unsigned long long& cnt_nnz, unsigned long long& cnt_empty, unsigned long long& upd) {
    auto member = [&](unsigned long long G0, int k) {
        return G0 | ((k & 1) ? gm[0] : 0ULL) | ((k & 2) ? gm[1] : 0ULL) | ((k & 4) ? gm[2] : 0ULL);
    };
    // a lane per entry: its unit's members, and whether it owns the unit (as in walk_hashed)
    unsigned long long base = 0;
    bool owns = false;
    if (e0 + lane < e1) {
        const unsigned b = __ldcg(t.list + e0 + lane);   // (an earlier pass of the same launch may have written it)
        const Header own = load_hdr_cg(t.hdr + b);
        const int idx = ((own.group & gm[0]) ? 1 : 0) | ((own.group & gm[1]) ? 2 : 0) | ((own.group & gm[2]) ? 4 : 0);
        base = own.group & ~(gm[0] | gm[1] | gm[2]);
        owns = true;
        constexpr int kMost = S == 1 ? 2 : 2 * S;
        Header h[kMost];
        unsigned at[kMost];
#pragma unroll
        for (int k = 0; k < kMost; ++k) {   // the first probes of all members together
            h[k].epoch = ep + 1;
            at[k] = b;
            if (k != idx && k < (1 << nx)) {
                at[k] = (unsigned)(mix64(member(base, k)) & t.mask);
                h[k] = load_hdr_cg(t.hdr + at[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < kMost; ++k) {
            uint2 m = make_uint2(kNoBucket, 0u);
            if (k == idx) {
                m = make_uint2(b, own.aux);
            } else if (h[k].epoch == ep) {
                const unsigned long long G = member(base, k);
                Header c = h[k];
                unsigned long long p = at[k];
                for (uint32_t i = 1; i < kMaxProbe && c.epoch == ep && c.group != G; ++i) {
                    p = (p + 1) & t.mask;
                    c = load_hdr_cg(t.hdr + p);
                }
                if (c.epoch == ep && c.group == G) {
                    m = make_uint2((unsigned)p, c.aux);
                    if (k < idx) owns = false;
                }
            }
            wk.m[lane][k] = m;
        }
    }
    unsigned todo = __ballot_sync(kFull, owns);
    __syncwarp();
    const int half = lane >> 4, j = lane & 15;
    while (todo) {
        int l = __ffs(todo) - 1;   // the unit of the lane's half, or of the warp
        todo &= todo - 1;
        bool on = true;
        if (S == 1 && nx == 0) {
            const int second = todo ? __ffs(todo) - 1 : -1;
            todo &= todo - 1;
            on = half == 0 || second >= 0;
            if (half && on) l = second;
        }
        const unsigned long long G0 = member(shfl64(base, l), S == 1 && nx == 0 ? 0 : half);
        uint2 m[S];
        Slots<T, S> x;
        x.pm = 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            m[s] = on ? wk.m[l][(S == 1 && nx == 0 ? 0 : half) | (s << 1)] : make_uint2(kNoBucket, 0u);
            const bool p = (m[s].y >> j) & 1u;
            x.pm |= (unsigned)p << s;
            x.v[s] = czero<T>();
            if (p) {
                const typename AmpT<T>::V a = __ldcg(reinterpret_cast<const typename AmpT<T>::V*>(t.amps) + (size_t)m[s].x * kSlots + j);
                x.v[s] = Cx<T>{a.x, a.y};
            }
        }
        bool touched = false;
        const unsigned pm0 = x.pm;
        x.n = __popc(pm0);
        run_slots<T, S, ODD>(sg, gates, ng, (G0 << kSlotBits) | (unsigned)j, lane, on, x, touched, pb, upd);
        const unsigned pm = x.pm;
        cnt_nnz += __popc(pm);
        // groups that appear, all claimed together: member s of a half by its lane s
        unsigned now[S];
        bool make = false;
        unsigned long long mine = 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned bal = __ballot_sync(kFull, (pm >> s) & 1u);
            now[s] = half ? bal >> 16 : bal & 0xFFFFu;
            if (j == s) {
                make = on && m[s].x == kNoBucket && now[s] != 0;
                mine = member(G0, s << 1);
            }
        }
        unsigned nb = kNoBucket;
        if (__any_sync(kFull, make)) {
            bool created = false;
            if (make) {
                const long long c = claim_group(t, ep, mine, &ctl->status, &created);
                if (c >= 0) nb = (unsigned)c;
            }
            __syncwarp();
            const unsigned got = __ballot_sync(kFull, created);
            unsigned long long at = 0;
            if (lane == 0 && got) at = atomicAdd(&ctl->list_tail, (unsigned long long)__popc(got));
            at = shfl64(at, 0) + __popc(got & ((1u << lane) - 1u));
            if (created) t.list[at] = nb;
        }
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const unsigned made = __shfl_sync(kFull, nb, (lane & 16) | s);
            const bool fresh = m[s].x == kNoBucket;
            const unsigned b = fresh ? made : m[s].x;
            if (b == kNoBucket) continue;   // absent, or the table is full: the pass has failed
            const bool p = (pm >> s) & 1u, moved = ((pm ^ pm0) >> s) & 1u;
            const size_t at = (size_t)b * kSlots + j;
            if (p && (touched || moved)) store_amp<T>(t.amps, at, x.v[s]);
            if (fresh || moved) t.keys[at] = p ? (member(G0, s << 1) << kSlotBits) | (unsigned)j : empty_key(j);
            if (j == 0 && (fresh || now[s] != m[s].y)) t.hdr[b].aux = now[s];
            if (j == 0 && now[s] == 0) cnt_empty += 1;
        }
    }
    __syncwarp();
}

// The list entries [e0, e1) of a slot pass without cross-group qubits, four slots to a lane: qubits 0 and 1 in a
// lane, 2 and 3 lane bits 0 and 1, eight groups to a warp. Decoding a gate then serves four slots. FP32 passes
// over many groups are bound by that (2^16 groups of 16 keys, 24 gates: 108 us with a slot to a lane); FP64 ones
// by the products, and small ones by the chain of a lane's slots.
template <class T, bool ODD>
__device__ __forceinline__ void walk_low(const TableDev& t, unsigned long long e0, unsigned long long e1, const HGates<T>& sg,
                                         const GateDesc* gates, uint32_t ng, int lane, const PruneBits& pb,
                                         unsigned long long& cnt_nnz, unsigned long long& cnt_empty, unsigned long long& upd) {
    const int quarter = (lane & 3) * 4;
    for (unsigned long long e = e0 + (lane >> 2); __any_sync(kFull, e < e1); e += 8) {
        const bool on = e < e1;
        unsigned b = 0;
        Header h;
        h.group = 0;
        h.aux = 0;
        if (on) {
            b = __ldcg(t.list + e);   // (an earlier pass of the same launch may have written it)
            h = load_hdr_cg(t.hdr + b);
        }
        const size_t at = (size_t)b * kSlots + quarter;
        Slots<T, 4> x;
        x.pm = (h.aux >> quarter) & 15u;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            x.v[s] = czero<T>();
            if ((x.pm >> s) & 1u) {
                const typename AmpT<T>::V a = __ldcg(reinterpret_cast<const typename AmpT<T>::V*>(t.amps) + at + s);
                x.v[s] = Cx<T>{a.x, a.y};
            }
        }
        bool touched = false;
        const unsigned pm0 = x.pm;
        x.n = __popc(pm0);
        run_slots<T, 4, ODD>(sg, gates, ng, (h.group << kSlotBits) | (unsigned)quarter, lane, on, x, touched, pb, upd);
        const unsigned pm = x.pm;
        cnt_nnz += __popc(pm);
        unsigned now = pm << quarter;
        now |= __shfl_xor_sync(kFull, now, 1);
        now |= __shfl_xor_sync(kFull, now, 2);
        if (!on) continue;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const bool p = (pm >> s) & 1u, moved = ((pm ^ pm0) >> s) & 1u;
            if (p && (touched || moved)) store_amp<T>(t.amps, at + s, x.v[s]);
            if (moved) t.keys[at + s] = p ? (h.group << kSlotBits) | (unsigned)(quarter + s) : empty_key(quarter + s);
        }
        if (quarter == 0) {
            if (now != h.aux) t.hdr[b].aux = now;
            if (now == 0) cnt_empty += 1;
        }
    }
}

}  // namespace
}  // namespace sqc
