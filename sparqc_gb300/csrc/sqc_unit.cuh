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
#include "sqc_pass_dev.cuh"

namespace sqc {
namespace {

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
    const bool two = op >= UO_RX_PAIR;   // H has one coefficient
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
template <bool TWO>
__device__ __forceinline__ void products(const UGate<float>& g, Cx<float> x, Cx<float>& C, Cx<float>& P) {
    C.r = __fmul_rn(g.c, x.r);
    C.i = __fmul_rn(g.c, x.i);
    if (TWO) {
        P.r = __fmul_rn(g.s, x.r);
        P.i = __fmul_rn(g.s, x.i);
    }
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

// Whether a branching result is kept (negligible's complement). FP64 looks at the high words
// first: the 64-bit compares otherwise issue on the FP64 pipe.
__device__ __forceinline__ bool kept(Cx<float> v, const PruneBits& pb) { return !negligible(v, pb); }
__device__ __forceinline__ bool kept(Cx<double> v, const PruneBits& pb) {
    const uint32_t th = (uint32_t)(pb.d >> 32), tl = (uint32_t)pb.d;
    const uint32_t r = (uint32_t)__double2hiint(v.r) & 0x7FFFFFFFu, i = (uint32_t)__double2hiint(v.i) & 0x7FFFFFFFu;
    if (r > th || i > th) return true;
    return (r == th && (uint32_t)__double2loint(v.r) >= tl) || (i == th && (uint32_t)__double2loint(v.i) >= tl);
}

template <class T>
__device__ __forceinline__ Cx<T> shfl_cx(Cx<T> a, int off) {
    return Cx<T>{__shfl_xor_sync(kFull, a.r, off), __shfl_xor_sync(kFull, a.i, off)};
}

// U's fused multiply-add chain (branch_update), `uniform`: the own bit is the warp's. The bit-0 row's own coefficient is real: its imaginary terms add +-0, which changes
// nothing unless the sum so far is itself 0.
__device__ __forceinline__ float u_coef(const UGate<float>& g, const GateDesc*, int i) { return g.m[i]; }
__device__ __forceinline__ double u_coef(const UGate<double>&, const GateDesc* gd, int i) { return __ldg(&gd->m[i]); }
__device__ __forceinline__ bool is_zero(float x) { return x == 0.f; }
__device__ __forceinline__ bool is_zero(double x) {   // no FP64 compare
    return (((uint32_t)__double2hiint(x) & 0x7FFFFFFFu) | (uint32_t)__double2loint(x)) == 0;
}
template <class T>
__device__ __forceinline__ Cx<T> u_update(const UGate<T>& g, const GateDesc* gd, bool bit, bool uniform, Cx<T> a,
                                          Cx<T> b) {
    using A = Arith<T>;
    auto m = [&](int i) { return u_coef(g, gd, i); };
    const T msr = bit ? m(6) : m(0), mor = bit ? m(4) : m(2), moi = bit ? m(5) : m(3);
    T r = A::mul(msr, a.r), i = A::mul(msr, a.i);
    if (!uniform || bit || is_zero(r) || is_zero(i)) {
        const T msi = bit ? m(7) : m(1);
        r = A::fma(neg(msi), a.i, r);
        i = A::fma(msi, a.r, i);
    }
    return Cx<T>{A::fma(neg(moi), b.i, A::fma(mor, b.r, r)), A::fma(moi, b.r, A::fma(mor, b.i, i))};
}

// ---- one gate on the slots a lane holds ---------------------------------------------------------
// Formulas and rounding are branch_update's, swap_update's and diag_update's (sqc_device.cuh): an
// Rx, Ry, Rz or Phase result is C + P', C = c * own, P' the s-product of the own or the partner
// amplitude with its sign flipped and its components exchanged as the kind asks (a - b and a + (-b),
// and (-s) * x and -(s * x), round alike).
template <class T, int S> struct Slots {
    Cx<T> v[S];
    unsigned pm;   // presence bits
};

// Store branching results into slots (s the lane word's slots to change). Results below the prune
// threshold are rare in the slots that hold keys: every result is stored as present, and the few
// that are not kept are cleared on a branch.
template <class T, int S>
__device__ __forceinline__ void put(Slots<T, S>& x, int s, Cx<T> o, const PruneBits& pb) {
    x.v[s] = o;
    if (!kept(o, pb)) {
        x.v[s] = czero<T>();
        x.pm &= ~(1u << s);
    }
}

template <class T, uint32_t K, int S>
__device__ __forceinline__ void swap_pair(uint32_t w, Slots<T, S>& x) {
    const bool flip = (w >> 31) != 0;
#pragma unroll
    for (int s = 0; s < S; s += 2) {
        if (!(w & (1u << s))) continue;
        const Cx<T> a = x.v[s], b = x.v[s + 1];
        x.v[s] = swap_update<T, K>(flip, b);
        x.v[s + 1] = swap_update<T, K>(!flip, a);
        x.pm = (x.pm & ~(3u << s)) | ((x.pm >> 1) & (1u << s)) | ((x.pm << 1) & (2u << s));
    }
}

template <class T, uint32_t K, int S>
__device__ __forceinline__ void swap_shfl(uint32_t loc, uint32_t w, Slots<T, S>& x) {
    const int off = 1 << ((loc >> kLocBit) & 31u);
    const unsigned pp = __shfl_xor_sync(kFull, x.pm, off);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (!(loc & (1u << (kLocSlots + s)))) continue;
        const Cx<T> b = shfl_cx(x.v[s], off);
        if (w & (1u << s)) x.v[s] = swap_update<T, K>((w >> 31) != 0, b);
    }
    x.pm = (x.pm & ~(w & 15u)) | (pp & w & 15u);
}

// Rx, Ry: results of the two members from their products (C: c * own, P: s * partner); Ry subtracts
// where minus has bit 31 set.
template <class T, uint32_t K>
__device__ __forceinline__ Cx<T> rot(Cx<T> C, Cx<T> P, uint32_t minus) {
    using A = Arith<T>;
    if constexpr (K == KRX) return Cx<T>{A::add(C.r, P.i), A::sub(C.i, P.r)};
    else return Cx<T>{A::add(C.r, flip_sign(P.r, minus)), A::add(C.i, flip_sign(P.i, minus))};
}

template <class T, uint32_t K, int S, class G>
__device__ __forceinline__ void branch_pair(const G& g, const GateDesc* gd, uint32_t w, Slots<T, S>& x,
                                            const PruneBits& pb) {
    using A = Arith<T>;
    x.pm |= w & ((1u << S) - 1u);
#pragma unroll
    for (int s = 0; s < S; s += 2) {
        if (!(w & (1u << s))) continue;
        Cx<T> a = x.v[s], b = x.v[s + 1], o0, o1;
        if constexpr (K == KH) {   // logical bit 0: v0 + v1, bit 1: v0 - v1
            const Cx<T> y0{A::add(b.r, flip_sign(a.r, w)), A::add(b.i, flip_sign(a.i, w))};
            const Cx<T> y1{A::add(a.r, flip_sign(b.r, ~w)), A::add(a.i, flip_sign(b.i, ~w))};
            Cx<T> none;
            products<false>(g, y0, o0, none);
            products<false>(g, y1, o1, none);
        } else if constexpr (K == KU) {
            o0 = u_update<T>(g, gd, (w >> 31) != 0, true, a, b);
            o1 = u_update<T>(g, gd, (w >> 31) == 0, true, b, a);
        } else {
            Cx<T> C0, C1, P0, P1;
            products<true>(g, a, C0, P0);
            products<true>(g, b, C1, P1);
            o0 = rot<T, K>(C0, P1, ~w);
            o1 = rot<T, K>(C1, P0, w);
        }
        put<T, S>(x, s, o0, pb);
        put<T, S>(x, s + 1, o1, pb);
    }
}

template <class T, uint32_t K, int S, class G>
__device__ __forceinline__ void branch_shfl(const G& g, const GateDesc* gd, uint32_t loc, uint32_t w, Slots<T, S>& x,
                                            const PruneBits& pb) {
    using A = Arith<T>;
    const int off = 1 << ((loc >> kLocBit) & 31u);
    x.pm |= w & ((1u << S) - 1u);
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (!(loc & (1u << (kLocSlots + s)))) continue;
        const Cx<T> a = x.v[s];
        Cx<T> o;
        if constexpr (K == KH) {
            const Cx<T> b = shfl_cx(a, off);
            const Cx<T> y{A::add(b.r, flip_sign(a.r, w)), A::add(b.i, flip_sign(a.i, w))};
            Cx<T> none;
            products<false>(g, y, o, none);
        } else if constexpr (K == KU) {
            o = u_update<T>(g, gd, (w >> 31) != 0, false, a, shfl_cx(a, off));
        } else {
            Cx<T> C, P;
            products<true>(g, a, C, P);   // the partner lane needs this lane's s-product
            o = rot<T, K>(C, shfl_cx(P, off), ~w);
        }
        if (w & (1u << s)) put<T, S>(x, s, o, pb);
    }
}

// Diagonal gates: e has bit s set where the gate acts on slot s and its logical target bit is 1.
template <class T, uint32_t K, int S, class G>
__device__ __forceinline__ void diag(const G& g, unsigned e, unsigned act, Slots<T, S>& x) {
    using A = Arith<T>;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        Cx<T>& v = x.v[s];
        if constexpr (K == KZ) {
            const uint32_t m = e << (31 - s);
            v = Cx<T>{flip_sign(v.r, m), flip_sign(v.i, m)};
        } else if constexpr (K == KS || K == KSDG) {   // S: i * v, Sdg: -i * v
            if (e & (1u << s)) v = K == KSDG ? Cx<T>{v.i, neg(v.r)} : Cx<T>{neg(v.i), v.r};
        } else if constexpr (K == KYPH) {              // bit 1: i * v, bit 0: -i * v
            const uint32_t m = e << (31 - s);
            if (act & (1u << s)) v = Cx<T>{flip_sign(v.i, m), flip_sign(v.r, ~m)};
        } else if (K == KRZ ? (act & (1u << s)) : (e & (1u << s))) {
            Cx<T> C, P;
            products<true>(g, v, C, P);
            if constexpr (K == KRZ) {   // bit 1: c*r - s*i, c*i + s*r; bit 0: + and -
                const uint32_t m = e << (31 - s);
                v = Cx<T>{A::add(C.r, flip_sign(P.i, m)), A::add(C.i, flip_sign(P.r, ~m))};
            } else {
                v = Cx<T>{A::sub(C.r, P.i), A::add(C.i, P.r)};
            }
        }
    }
}

template <class T, int S>
__device__ __forceinline__ void swap_slots12(Slots<T, S>& x) {
    const Cx<T> y = x.v[S == 4 ? 1 : 0];
    x.v[S == 4 ? 1 : 0] = x.v[S == 4 ? 2 : 0];
    x.v[S == 4 ? 2 : 0] = y;
    x.pm = (x.pm & 9u) | ((x.pm & 2u) << 1) | ((x.pm & 4u) >> 1);
}

// The gates of a pass on the unit a warp holds; uid is the unit's base index. Absent slots hold
// +-0, which no gate makes present (sqc_pass_dev.cuh).
template <class T, int S>
__device__ __forceinline__ void run_unit(const UGates<T>& sg, const GateDesc* __restrict__ gates, uint32_t ng,
                                         uint32_t uid, int lane, Slots<T, S>& x, bool& touched,
                                         const PruneBits& pb, unsigned long long& upd) {
    unsigned n = __popc(x.pm);
#pragma unroll 1
    for (uint32_t gi = 0; gi < ng; ++gi) {
        const UGate<T>& g = sg.g[gi];
        const uint4 head = *reinterpret_cast<const uint4*>(&g);   // om, ov, loc, weight
        upd += (unsigned long long)n * head.w;
        if ((uid & head.x) != head.y) continue;   // a control outside the unit excludes all of it
        const uint32_t w = (uint32_t)(int)sg.lw[gi][lane];
        const uint32_t loc = head.z;
        const GateDesc* gd = gates + gi;
        touched = true;
        const bool exchange = S == 4 && (loc & kLocPair3);   // dimension 2: exchange slots around the pair code
        if (exchange) swap_slots12<T, S>(x);
        if ((loc >> kLocOp) < UO_Z) {
            switch (loc >> kLocOp) {
            case UO_X_PAIR: swap_pair<T, KX, S>(w, x); break;
            case UO_X_SHFL: swap_shfl<T, KX, S>(loc, w, x); break;
            case UO_Y_PAIR: swap_pair<T, KY, S>(w, x); break;
            case UO_Y_SHFL: swap_shfl<T, KY, S>(loc, w, x); break;
            case UO_H_PAIR: branch_pair<T, KH, S>(g, gd, w, x, pb); break;
            case UO_H_SHFL: branch_shfl<T, KH, S>(g, gd, loc, w, x, pb); break;
            case UO_RX_PAIR: branch_pair<T, KRX, S>(g, gd, w, x, pb); break;
            case UO_RX_SHFL: branch_shfl<T, KRX, S>(g, gd, loc, w, x, pb); break;
            case UO_RY_PAIR: branch_pair<T, KRY, S>(g, gd, w, x, pb); break;
            case UO_RY_SHFL: branch_shfl<T, KRY, S>(g, gd, loc, w, x, pb); break;
            case UO_U_PAIR: branch_pair<T, KU, S>(g, gd, w, x, pb); break;
            default: branch_shfl<T, KU, S>(g, gd, loc, w, x, pb); break;
            }
            if (exchange) swap_slots12<T, S>(x);
            n = __popc(x.pm);
        } else {
            const unsigned act = w & 15u;
            const unsigned e = ((w >> 4) & 15u) ^ (((uid >> ((loc >> kLocBit) & 31u)) & 1u) && !(loc & kLocLane) ? act : 0u);
            switch (loc >> kLocOp) {
            case UO_Z: diag<T, KZ, S>(g, e, act, x); break;
            case UO_S: diag<T, KS, S>(g, e, act, x); break;
            case UO_SDG: diag<T, KSDG, S>(g, e, act, x); break;
            case UO_YPH: diag<T, KYPH, S>(g, e, act, x); break;
            case UO_RZ: diag<T, KRZ, S>(g, e, act, x); break;
            default: diag<T, KPHASE, S>(g, e, act, x); break;
            }
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
template <class T, int DIMS>
__device__ __forceinline__ void do_unit(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up, unsigned base,
                                        const UGates<T>& sg, const GateDesc* gates, uint32_t ng, int lane,
                                        const PruneBits& pb, unsigned long long& cnt_nnz, unsigned long long& cnt_empty,
                                        unsigned long long& upd) {
    constexpr int S = 1 << (DIMS - 1);
    const int j = lane & 15;
    const unsigned b0 = base | ((unsigned)(lane >> 4) << up.dim[1]);
    unsigned bk[S];
    uint2 h[S];
    Slots<T, S> x;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        bk[s] = b0 | ((s & 1) ? 1u << up.dim[0] : 0u) | ((s & 2) ? 1u << up.dim[2] : 0u);
        h[s] = *reinterpret_cast<const uint2*>(&t.hdr[bk[s]].epoch);
        const typename AmpT<T>::V a = reinterpret_cast<const typename AmpT<T>::V*>(t.amps)[(size_t)bk[s] * kSlots + j];
        x.v[s] = Cx<T>{a.x, a.y};
    }
    x.pm = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const bool p = h[s].x == ep && ((h[s].y >> j) & 1u);
        x.pm |= (unsigned)p << s;
        x.v[s] = pick(p, x.v[s], czero<T>());
    }
    bool touched = false;
    const unsigned pm0 = x.pm;
    if (__any_sync(kFull, pm0 != 0)) run_unit<T, S>(sg, gates, ng, base, lane, x, touched, pb, upd);
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
    } else {
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (j == 0 && h[s].x == ep && h[s].y == 0) cnt_empty += 1;
    }
}

// Units [u0, u1) step `stride` of a table whose live buckets fill it.
template <class T, int DIMS>
__device__ __forceinline__ void walk_units(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up,
                                           unsigned long long u0, unsigned long long u1, unsigned long long stride,
                                           const UGates<T>& sg, const GateDesc* gates, uint32_t ng, int lane,
                                           const PruneBits& pb, unsigned long long& cnt_nnz,
                                           unsigned long long& cnt_empty, unsigned long long& upd) {
    for (unsigned long long u = u0; u < u1; u += stride)
        do_unit<T, DIMS>(t, mq, ctl, ep, up, unit_base<DIMS>((unsigned)u, up.lo), sg, gates, ng, lane, pb, cnt_nnz, cnt_empty,
                         upd);
}

// The units of list entries [e0, e0 + 32) below n, for tables whose live buckets are few among
// the mapped ones: lane l takes entry e0 + l; the unit belongs to its live member of smallest index
// (members a pass creates are made by the unit's owner, after its own check), found by reading
// the headers of the smaller members.
template <class T, int DIMS>
__device__ __forceinline__ void walk_entries(const TableDev& t, const uint8_t* mq, Ctl* ctl, unsigned ep, const UnitPass& up,
                                             unsigned long long e0, unsigned long long n, const UGates<T>& sg,
                                             const GateDesc* gates, uint32_t ng, int lane, const PruneBits& pb,
                                             unsigned long long& cnt_nnz, unsigned long long& cnt_empty,
                                             unsigned long long& upd) {
    constexpr int K = 1 << DIMS;
    unsigned base = 0;
    bool own = false;
    if (e0 + lane < n) {
        const unsigned b = t.list[e0 + lane];
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
        do_unit<T, DIMS>(t, mq, ctl, ep, up, __shfl_sync(kFull, base, l), sg, gates, ng, lane, pb, cnt_nnz, cnt_empty, upd);
    }
}

// Whether a pass walks the list (live buckets below an eighth of the mapped ones) or every unit:
// a unit without keys costs its headers and amplitudes (about an eighth of a unit of a ten-gate
// pass), a list entry its ownership check.
__device__ __forceinline__ bool walk_list(unsigned long long list_n, uint32_t dn) {
    return dn >= 6 && list_n < (1ULL << (dn - 3));
}

}  // namespace
}  // namespace sqc
