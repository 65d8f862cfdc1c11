// Host-side gate planning: see sqc_plan.h.
#include "sqc_plan.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace sqc {

const char* check_gate(const sqc_gate& g, uint32_t nq) {
    if (g.kind > SQC_U) return "unknown gate kind";
    if (g.target >= nq) return "target qubit out of range";
    if (nq < 64 && (g.controls >> nq)) return "control qubit out of range";
    if ((g.controls >> g.target) & 1ULL) return "target qubit among the controls";
    return nullptr;
}

GateDesc make_desc(const Planner& p, uint32_t kind, uint32_t target, unsigned long long ctrl, const sqc_gate& g) {
    GateDesc d;
    std::memset(&d, 0, sizeof d);
    d.kind = kind;
    d.target = target;
    d.ctrl = ctrl;
    d.cval = ctrl & ~p.frame;
    d.flip = (uint32_t)((p.frame >> target) & 1ULL);
    switch (kind) {
    case KPHASE: d.c = std::cos(g.theta); d.s = std::sin(g.theta); break;
    case KRZ: case KRX: case KRY: {
        const double h = g.theta / 2.;   // the reference passes par/2 (table_manager.cuh:333-336)
        d.c = std::cos(h);
        d.s = std::sin(h);
        break;
    }
    case KT: d.c = 0.70710678118654752440; d.s = 0.70710678118654752440; break;
    case KTDG: d.c = 0.70710678118654752440; d.s = -0.70710678118654752440; break;
    case KH: d.c = 1. / std::sqrt(2.); break;   // as in h_core (device_data.cuh:205)
    case KU: {
        const double c = std::cos(g.theta / 2.), s = std::sin(g.theta / 2.);
        const double cl = std::cos(g.lambda), sl = std::sin(g.lambda);
        const double cp = std::cos(g.phi), sp = std::sin(g.phi);
        const double cpl = std::cos(g.phi + g.lambda), spl = std::sin(g.phi + g.lambda);
        d.m[0] = c;         d.m[1] = 0.;
        d.m[2] = -(cl * s); d.m[3] = -(sl * s);
        d.m[4] = cp * s;    d.m[5] = sp * s;
        d.m[6] = cpl * c;   d.m[7] = spl * c;
        break;
    }
    default: break;
    }
    d.cf = (float)d.c;
    d.sf = (float)d.s;
    for (int i = 0; i < 8; ++i) d.mf[i] = (float)d.m[i];
    return d;
}

namespace {

// What plan_gate decides, without the descriptor: whether the gate needs the device, as which kind
// and with which controls still to test per key.
bool resolve_gate(Planner& p, const sqc_gate& g, uint32_t* kind, unsigned long long* ctrl) {
    const unsigned long long bq = 1ULL << g.target;
    const unsigned long long kc = g.controls & p.kmask;
    if ((p.kval & kc) != kc) { ++p.credit; return false; }   // a control is known to be 0
    *ctrl = g.controls & ~p.kmask;
    *kind = g.kind;
    if (is_swap_kind(g.kind) && *ctrl == 0) {
        p.frame ^= bq;
        if (p.kmask & bq) p.kval ^= bq;
        if (g.kind == KX) { ++p.credit; return false; }
        *kind = KYPH;   // Y = relabel + diag(-i, +i)
        return true;
    }
    if (is_one_sided_kind(g.kind) && (p.kmask & bq) && !(p.kval & bq)) { ++p.credit; return false; }
    return true;
}

}  // namespace

bool plan_gate(Planner& p, const sqc_gate& g, GateDesc* out) {
    uint32_t kind;
    unsigned long long ctrl;
    if (!resolve_gate(p, g, &kind, &ctrl)) return false;
    *out = make_desc(p, kind, g.target, ctrl, g);
    if (!is_diag_kind(kind)) p.kmask &= ~(1ULL << g.target);
    return true;
}

void encode_pass(GateDesc* d, size_t g0, size_t g1, uint32_t q1, uint32_t q3) {
    for (size_t k = g0; k < g1; ++k) {
        GateDesc& g = d[k];
        uint32_t op = g.flip & kOpFlip;
        const bool branch = is_branch_kind(g.kind), swap = is_swap_kind(g.kind);
        if (g.ctrl) op |= kOpCtrl;
        if (branch) op |= kOpBranch;
        if (swap) op |= kOpSwap;
        if (is_one_sided_kind(g.kind)) op |= kOpOneSided;
        if (g.target < (uint32_t)kSlotBits) op |= kOpLowBit;
        if (branch || swap) {
            if (g.target == q1 && g.target >= (uint32_t)kSlotBits) {
                op |= kOpPair;
            } else if (g.target == q3 && g.target >= (uint32_t)kSlotBits) {
                op |= kOpPair3;
            } else {
                // qubits 0..3: a lane of the same half; the pass's second cross-group qubit:
                // the other half of the warp
                const uint32_t off_log2 = g.target < (uint32_t)kSlotBits ? g.target : 4u;
                op |= kOpShfl | (off_log2 << kOpOffShift);
            }
        }
        g.flip = op;
    }
}

bool GroupMap::extend(unsigned long long kmask, uint32_t nq) {
    const unsigned long long reg = nq >= 64 ? ~0ULL : ((1ULL << nq) - 1);
    unsigned long long add = ~kmask & reg & ~15ULL;
    for (uint32_t i = 0; i < n; ++i) add &= ~(1ULL << (q[i] + kSlotBits));
    if (n + (uint32_t)__builtin_popcountll(add) > kMaxMapBits) return false;
    for (; add; add &= add - 1) q[n++] = (uint8_t)(__builtin_ctzll(add) - kSlotBits);
    return true;
}

// Whether a coefficient is not finite (an angle was infinite or NaN).
static bool odd_gate(const GateDesc& g) {
    bool odd = !std::isfinite(g.c) || !std::isfinite(g.s);
    for (double m : g.m) odd = odd || !std::isfinite(m);
    return odd;
}

// The op code of a gate kind (pairing kinds: on slots 0-1 and 2-3).
static uint32_t unit_op(uint32_t kind) {
    switch (kind) {
    case KX: return UO_X_PAIR;
    case KY: return UO_Y_PAIR;
    case KH: return UO_H_PAIR;
    case KRX: return UO_RX_PAIR;
    case KRY: return UO_RY_PAIR;
    case KU: return UO_U_PAIR;
    case KZ: return UO_Z;
    case KS: return UO_S;
    case KSDG: return UO_SDG;
    case KYPH: return UO_YPH;
    case KRZ: return UO_RZ;
    default: return UO_PHASE;   // Phase, T, Tdg
    }
}

void encode_unit_pass(GateDesc* d, size_t g0, size_t g1, const uint32_t q[3], const GroupMap& map, uint32_t dims,
                      uint32_t dim[3]) {
    // the cross-group qubit with the fewest gates goes to the lane dimension (1), whose gates
    // shuffle; the others pair slots of one lane, the most used in dimension 0 (dimension 2 costs
    // an exchange of slots around each gate)
    uint32_t order[3] = {q[0], q[1], q[2]}, uses[3] = {0, 0, 0};
    for (size_t k = g0; k < g1; ++k)
        for (int i = 0; i < 3; ++i)
            if (!streamable(d[k]) && d[k].target == q[i]) ++uses[i];
    int nx = 0;
    while (nx < 3 && q[nx] != kNoQubit) ++nx;
    if ((uint32_t)nx == dims) {
        int least = 0;
        for (int i = 1; i < nx; ++i)
            if (uses[i] < uses[least]) least = i;
        std::swap(order[1], order[least]);
        std::swap(uses[1], uses[least]);
    } else if (nx == 2) {   // three dimensions, two qubits: both pair slots
        order[2] = order[1];
        uses[2] = uses[1];
        order[1] = kNoQubit;
    }
    if (dims == 3 && nx >= 2 && uses[2] > uses[0]) std::swap(order[0], order[2]);
    unsigned long long taken = 0;
    int bit[3] = {-1, -1, -1};
    for (uint32_t i = 0; i < dims; ++i) {
        if (order[i] == kNoQubit) continue;
        bit[i] = map.bit_of(order[i]);
        taken |= 1ULL << bit[i];
    }
    for (uint32_t i = 0; i < 3; ++i) {
        if (i < dims && bit[i] < 0) {
            int b = 0;
            while ((taken >> b) & 1ULL) ++b;
            bit[i] = b;
            taken |= 1ULL << b;
        }
        dim[i] = i < dims ? (uint32_t)bit[i] : 31u;
    }
    for (size_t k = g0; k < g1; ++k) {
        GateDesc& g = d[k];
        g.om = g.ov = 0;
        uint32_t lmask = 0, lval = 0, smask = 0, sval = 0;
        for (unsigned long long c = g.ctrl; c; c &= c - 1) {
            const uint32_t qb = (uint32_t)__builtin_ctzll(c);
            const uint32_t v = (uint32_t)((g.cval >> qb) & 1ULL);
            if (qb < (uint32_t)kSlotBits) {
                lmask |= 1u << qb;
                lval |= v << qb;
                continue;
            }
            const uint32_t b = (uint32_t)map.bit_of(qb);
            if (b == dim[0]) { smask |= 1u; sval |= v; }
            else if (b == dim[1]) { lmask |= 16u; lval |= v << 4; }
            else if (b == dim[2]) { smask |= 2u; sval |= v << 1; }
            else { g.om |= 1u << b; g.ov |= v << b; }
        }
        // the target: a lane bit, a slot bit (0 or 1), or a bit of the unit's base; a diagonal gate
        // on a bit that never differed reads stored 0 (no bit of the base)
        uint32_t lane_bit = kNoQubit, slot_bit = kNoQubit, outer = kMaxMapBits;
        if (g.target < (uint32_t)kSlotBits) {
            lane_bit = g.target;
        } else {
            const int b = map.bit_of(g.target);
            if (b >= 0 && (uint32_t)b == dim[0]) slot_bit = 0;
            else if (b >= 0 && (uint32_t)b == dim[1]) lane_bit = 4;
            else if (b >= 0 && (uint32_t)b == dim[2]) slot_bit = 1;
            else if (b >= 0) outer = (uint32_t)b;
        }
        const bool flip = (g.flip & kOpFlip) != 0, pairs = is_branch_kind(g.kind) || is_swap_kind(g.kind);
        const bool pair3 = pairs && slot_bit == 1;
        uint32_t slots = 0, bits = 0;
        for (uint32_t s = 0; s < 4; ++s) {
            if (((s ^ sval) & smask) == 0) slots |= 1u << s;
            if ((slot_bit != kNoQubit && ((s >> slot_bit) & 1u)) != flip) bits |= 1u << s;
        }
        const uint32_t shfl = lane_bit != kNoQubit ? 1u : 0u;
        uint32_t op = unit_op(g.kind) + (pairs ? shfl : 0u);
        const bool all = pairs && !lmask && !smask;   // no controls inside the unit
        if (pairs && (all || pair3)) op += all ? (pair3 ? UO_ALL3 : UO_ALL) : UO_PAIR3;
        if (odd_gate(g)) op = UO_ODD + (pair3 ? 2u : pairs ? shfl : 0u);
        const uint32_t tb = lane_bit != kNoQubit ? lane_bit : slot_bit != kNoQubit ? kMaxMapBits : outer;
        g.loc = lmask | (lval << kLocLaneVal) | (slots << kLocSlots) | (bits << kLocSlotBit) | (tb << kLocBit) |
                (shfl ? kLocLane : 0u) | (flip ? kLocFlip : 0u) |
                (op << kLocOp);
    }
}

// One gate's place in a pass over a hashed table whose lanes hold the four keys that differ in qubits q0 and q1:
// controls on them by slot, all others by key; op is the gate's op code (pairing gates on q0 or q1: with the
// form on q1 added).
static void encode_in_lane(GateDesc& g, uint32_t q0, uint32_t q1, uint32_t lane_bit) {
    g.om = g.ov = 0;
    const uint32_t q[2] = {q0, q1};   // (kNoQubit: none)
    uint32_t smask = 0, sval = 0, slot_bit = kNoQubit;
    for (uint32_t i = 0; i < 2; ++i) {
        if (q[i] == kNoQubit) continue;
        if (g.target == q[i]) slot_bit = i;
        if (!((g.ctrl >> q[i]) & 1ULL)) continue;
        smask |= 1u << i;
        sval |= (uint32_t)((g.cval >> q[i]) & 1ULL) << i;
    }
    const bool flip = (g.flip & kOpFlip) != 0, pairs = is_branch_kind(g.kind) || is_swap_kind(g.kind);
    uint32_t slots = 0, bits = 0;
    for (uint32_t s = 0; s < 4; ++s) {
        if (((s ^ sval) & smask) == 0) slots |= 1u << s;
        if ((slot_bit != kNoQubit && ((s >> slot_bit) & 1u)) != flip) bits |= 1u << s;
    }
    const bool pair3 = pairs && slot_bit == 1, lanes = pairs && slot_bit == kNoQubit;
    const uint32_t op = odd_gate(g) ? UO_ODD + (pair3 ? 2u : lanes ? 1u : 0u) : unit_op(g.kind) + (pair3 ? UO_PAIR3 : lanes ? 1u : 0u);
    const uint32_t bit = lanes ? lane_bit : g.target & 31u;
    g.loc = (slots << kLocSlots) | (bits << kLocSlotBit) | (slot_bit != kNoQubit ? kLocLane : 0u) | (bit << kLocBit) |
            (!lanes && g.target >= 32u ? kLocHigh : 0u) | (flip ? kLocFlip : 0u) | (op << kLocOp);
}

void encode_column_pass(GateDesc* d, size_t g0, size_t g1, const uint32_t q[2], uint32_t dim[3]) {
    dim[0] = q[0];
    dim[1] = q[1];
    dim[2] = 64u;
    for (int i = 0; i < 2; ++i)   // (2^16 groups of 16 keys, 24 diagonal gates, FP64: 747 us with one key to a column)
        if (dim[i] == kNoQubit) dim[i] = dim[1 - i] == 0u ? 1u : 0u;
    for (size_t k = g0; k < g1; ++k) encode_in_lane(d[k], dim[0], dim[1], 0);
}

void encode_slot_pass(GateDesc* d, size_t g0, size_t g1, uint32_t form, const uint32_t q[3], uint32_t dim[3]) {
    for (int i = 0; i < 3; ++i) dim[i] = q[i] == kNoQubit ? 64u : q[i];
    // lane bits: qubits 0 to 3, then the first cross-group one; the others are in a lane
    for (size_t k = g0; k < g1; ++k) {
        if (form == 2) encode_in_lane(d[k], 0, 1, d[k].target - 2);   // (lanes: qubits 2 and 3)
        else encode_in_lane(d[k], q[1], q[2], std::min(d[k].target, 4u));
    }
}

namespace {

// A gate as the scheduler sees it: the qubits it touches (target and controls), the qubit it changes
// (its target, unless it is diagonal), its target bit when the device pairs keys across groups
// for it, and whether the device runs it at all.
struct SchedGate {
    unsigned long long sup, moves, cross;
    uint32_t dev;
};

// The gates of a scheduling window: those not yet placed, in order, and their positions in the input.
struct SchedWindow {
    std::vector<SchedGate> g;
    std::vector<uint32_t> idx;
};

// One pass over the window's gates (in order, the first one first): a gate joins when it
// commutes with every gate left behind so far and fits the pass (cross-group qubits: those of
// fixed_q when nonzero, else the first max_nx used; at most max_run device gates), over the
// first nscan gates. Two gates commute when neither changes a qubit the other touches: gates
// act diagonally on their controls, and a diagonal gate on its target too, and operators that
// are diagonal on their shared qubits and change disjoint ones commute. Writes the positions
// taken to took (room for nscan + 1; their number to *ntook) if given, and returns the number of device gates among them; *limited (if
// given) tells whether a gate was refused for want of a cross-group qubit.
size_t sched_pass(const SchedWindow& w, size_t nscan, uint32_t max_nx, size_t max_run, unsigned long long fixed_q,
                  uint32_t* took, size_t* ntook, bool* limited) {
    unsigned long long qmask = fixed_q;
    uint32_t nx = 0;
    const bool fixed = fixed_q != 0;
    size_t run = 0;
    bool lim = false;
    size_t nt = 0;
    uint32_t sink[2];
    uint32_t* to = took ? took : sink;
    const size_t step = took ? 1 : 0;
    unsigned long long left_sup = 0, left_moves = 0;   // of the gates left behind
    // written without data-dependent branches: whether a gate joins is close to a coin flip
    for (size_t r = 0; r < nscan && run < max_run; ++r) {
        const SchedGate& g = w.g[r];
        const unsigned long long blocked = (g.moves & left_sup) | (g.sup & left_moves);
        const unsigned long long new_q = g.cross & ~qmask;
        const bool refused = (new_q != 0) & (fixed | (nx >= max_nx));
        const bool take = (blocked == 0) & !refused;
        lim |= (blocked == 0) & refused;
        const unsigned long long behind = take ? 0ULL : ~0ULL;
        left_sup |= g.sup & behind;
        left_moves |= g.moves & behind;
        qmask |= new_q & ~behind;
        nx += (unsigned)(take & (new_q != 0));
        run += (size_t)(take & (g.dev != 0));
        to[nt] = w.idx[r];
        nt += take ? step : 0;
    }
    if (limited) *limited = lim;
    if (ntook) *ntook = nt;
    return run;
}

}  // namespace

namespace {

// Device gates a pass takes over the first nscan gates of the window for each of nset (at most 32)
// choices of its cross-group qubits, as sched_pass counts them for one choice (nscan <= max_run, so
// no choice stops early). All choices advance together: bit s of a word belongs to choice s, and
// for every qubit there is one word of the choices whose gates left behind touch it and one of those
// whose change it. A gate costs a few words per qubit it touches instead of a step per choice (2000
// gates of 48 qubits: 1.16 -> 0.37 ms in all).
void sched_trials(const SchedWindow& w, size_t nscan, const unsigned long long* sets, uint32_t nset, uint32_t* runs) {
    uint32_t left_sup[64] = {}, left_moves[64] = {};
    uint32_t plane[7] = {};   // bit k of every choice's count (counts stay below 128)
    uint32_t without[64];     // choices a qubit is not in
    for (uint32_t& m : without) m = ~0u;
    for (uint32_t s = 0; s < nset; ++s)
        for (unsigned long long m = sets[s]; m; m &= m - 1) without[__builtin_ctzll(m)] &= ~(1u << s);
    for (size_t r = 0; r < nscan; ++r) {
        const SchedGate& g = w.g[r];
        uint32_t blocked = 0;
        if (g.moves) blocked = left_sup[__builtin_ctzll(g.moves)];
        for (unsigned long long m = g.sup; m; m &= m - 1) blocked |= left_moves[__builtin_ctzll(m)];
        if (g.cross) blocked |= without[__builtin_ctzll(g.cross)];
        for (unsigned long long m = g.sup; m; m &= m - 1) left_sup[__builtin_ctzll(m)] |= blocked;
        if (g.moves) left_moves[__builtin_ctzll(g.moves)] |= blocked;
        if (g.dev) {
            uint32_t carry = ~blocked;
            for (int k = 0; k < 7 && carry; ++k) {
                const uint32_t t = plane[k] & carry;
                plane[k] ^= carry;
                carry = t;
            }
        }
    }
    for (uint32_t s = 0; s < nset; ++s) {
        runs[s] = 0;
        for (int k = 0; k < 7; ++k) runs[s] |= ((plane[k] >> s) & 1u) << k;
    }
}

}  // namespace

void schedule_gates(const sqc_gate* g, size_t n, uint32_t max_nx, size_t max_run, size_t window, uint32_t* perm) {
    // what each gate is, planned in the given order: a move below only passes gates that change
    // none of the key bits the moved gate's planning reads (its target and controls), and the
    // moved gate changes none of theirs, so every gate plans the same in the new order
    std::vector<SchedGate> sg(n);
    std::vector<unsigned char> done(n, 0);
    Planner p;
    for (size_t i = 0; i < n; ++i) {
        const unsigned long long t = 1ULL << g[i].target;
        uint32_t kind = g[i].kind;
        unsigned long long ctrl;
        sg[i].dev = resolve_gate(p, g[i], &kind, &ctrl) ? 1 : 0;
        const bool pairs = sg[i].dev && !is_diag_kind(kind);
        if (pairs) p.kmask &= ~t;
        sg[i].cross = pairs && g[i].target >= (uint32_t)kSlotBits ? t : 0ULL;
        sg[i].sup = t | g[i].controls;
        sg[i].moves = is_diag_kind(g[i].kind) ? 0ULL : t;
    }
    if (max_nx > 3) max_nx = 3;
    size_t out = 0, first = 0;
    SchedWindow w;
    std::vector<uint32_t> best(window + 1);
    size_t next = 0;   // the first gate the window has not reached
    while (first < n) {
        if (done[first]) {
            ++first;
            continue;
        }
        size_t keep = 0;   // drop the gates the last pass took, add those the window reaches now
        for (size_t r = 0; r < w.idx.size(); ++r) {
            w.idx[keep] = w.idx[r];
            w.g[keep] = w.g[r];
            keep += done[w.idx[r]] ? 0 : 1;
        }
        w.idx.resize(keep);
        w.g.resize(keep);
        for (; next < std::min(n, first + window); ++next) {
            w.idx.push_back((uint32_t)next);
            w.g.push_back(sg[next]);
        }
        // the pass's cross-group qubits: the first-use choice, or any max_nx of the first
        // kSchedCandidates qubits the window's gates pair across, whichever takes the most
        // device gates over the first kSchedTrialWindow gates (earliest choice on ties). A
        // first-use pass that refused no gate for want of a qubit took every gate it reached (the
        // first refusal of any other kind needs a gate left behind), so no choice does better.
        const size_t ntrial = std::min(w.idx.size(), (size_t)kSchedTrialWindow);
        bool limited = false;
        size_t best_run = sched_pass(w, ntrial, max_nx, max_run, 0ULL, nullptr, nullptr, &limited);
        unsigned long long best_q = 0;
        if (limited) {
            unsigned long long cand[kSchedCandidates];
            uint32_t m = 0;
            unsigned long long seen = 0;
            for (size_t r = 0; r < w.idx.size() && m < kSchedCandidates; ++r) {
                if (w.g[r].cross & ~seen) cand[m++] = w.g[r].cross;
                seen |= w.g[r].cross;
            }
            const uint32_t k = std::min(max_nx, m);
            if (k > 0 && m > k) {
                uint32_t ix[3] = {0, 1, 2};
                unsigned long long sets[32];
                uint32_t runs[32], nset = 0;
                for (;;) {   // every k-subset of the candidates (20 at most), in lexicographic order
                    unsigned long long set = 0;
                    for (uint32_t a = 0; a < k; ++a) set |= cand[ix[a]];
                    sets[nset++] = set;
                    int a = (int)k - 1;
                    while (a >= 0 && ix[a] == m - k + (uint32_t)a) --a;
                    if (a < 0) break;
                    ++ix[a];
                    for (uint32_t b = (uint32_t)a + 1; b < k; ++b) ix[b] = ix[b - 1] + 1;
                }
                if (ntrial <= max_run) {
                    sched_trials(w, ntrial, sets, nset, runs);
                } else {
                    for (uint32_t s = 0; s < nset; ++s)
                        runs[s] = (uint32_t)sched_pass(w, ntrial, max_nx, max_run, sets[s], nullptr, nullptr, nullptr);
                }
                for (uint32_t s = 0; s < nset; ++s) {
                    if (runs[s] > best_run) {   // earliest choice on ties, the first-use one first
                        best_run = runs[s];
                        best_q = sets[s];
                    }
                }
            }
        }
        size_t taken = 0;   // the chosen pass over the whole window
        sched_pass(w, w.idx.size(), max_nx, max_run, best_q, best.data(), &taken, nullptr);
        if (!taken) best[taken++] = (uint32_t)first;   // (never: the first gate always fits the first-use pass)
        for (size_t k = 0; k < taken; ++k) {
            done[best[k]] = 1;
            perm[out++] = best[k];
        }
    }
}

unsigned long long group_bound(const Planner& p, uint32_t nq) {
    const unsigned long long reg = nq >= 64 ? ~0ULL : ((1ULL << nq) - 1);
    const unsigned long long var = ~p.kmask & reg & ~15ULL;
    const int bits = __builtin_popcountll(var);
    return bits >= 63 ? (1ULL << 63) : (1ULL << bits);
}

}  // namespace sqc
