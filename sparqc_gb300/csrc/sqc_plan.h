// Host-side gate planning shared by the single-state engine and the many-circuit batch:
// resolution of gates against what is known about the keys, descriptor construction
// (coefficients on the host) and the split of a descriptor sequence into passes.
#pragma once
#include <cstddef>
#include <algorithm>
#include <cstdint>

#include "../../include/sparqc.h"
#include "sqc_types.h"

namespace sqc {

// What the host knows about the keys without looking at them: stored key = actual key ^
// frame; bits in kmask are identical across all keys and equal kval. Gates whose effect
// follows from this are resolved here: an uncontrolled X flips a frame bit, a gate with a
// known-zero control or a one-sided diagonal gate on a known-zero bit is the identity.
// kmask only loses bits, so ~kmask is every bit that has ever differed between keys.
struct Planner {
    unsigned long long frame = 0;
    unsigned long long kmask = ~0ULL;
    unsigned long long kval = 0;
    uint32_t credit = 0;   // resolved gates not yet credited to a device gate
};

inline bool is_diag_kind(uint32_t k) {
    return k == KZ || k == KPHASE || k == KRZ || k == KS || k == KSDG || k == KT || k == KTDG || k == KYPH;
}
inline bool is_one_sided_kind(uint32_t k) {
    return k == KZ || k == KPHASE || k == KS || k == KSDG || k == KT || k == KTDG;
}
inline bool is_branch_kind(uint32_t k) { return k == KH || k == KRX || k == KRY || k == KU; }
inline bool is_swap_kind(uint32_t k) { return k == KX || k == KY; }
// A gate that never pairs keys of different 16-key groups.
inline bool streamable(const GateDesc& d) { return d.target < (uint32_t)kSlotBits || is_diag_kind(d.kind); }

// Check one gate against a register of nq qubits; nullptr when valid, else the reason.
const char* check_gate(const sqc_gate& g, uint32_t nq);

// Descriptor of one device gate in the stored-key frame of p, coefficients resolved here.
GateDesc make_desc(const Planner& p, uint32_t kind, uint32_t target, unsigned long long ctrl, const sqc_gate& g);

// Resolve one gate against p. Returns true and a descriptor when the gate needs the device;
// otherwise the gate was applied here (identity, or an uncontrolled X as a frame flip) and
// is counted in p.credit, to be credited to the next device gate.
bool plan_gate(Planner& p, const sqc_gate& g, GateDesc* out);

// Passes of a descriptor sequence. A pass is a run of at most max_run consecutive gates whose
// cross-group gates (gates that pair keys of different 16-key groups) target at most
// max_nx (<= 3) distinct qubits; streamable gates may sit anywhere in it. Passes are cut
// greedily. f(g0, g1, nx, q1, q2, q3, keys_fixed) is called per pass, q1..q3 the cross-group
// qubits in order of first use (kNoQubit when absent).
// With columns, gates on the low four qubits pair too (passes over hashed tables).
template <class F>
void split_passes(const GateDesc* d, size_t n, size_t max_run, uint32_t max_nx, F&& f, bool columns = false) {
    size_t i = 0;
    while (i < n) {
        const size_t start = i;
        uint32_t q[3] = {kNoQubit, kNoQubit, kNoQubit};
        uint32_t nx = 0;
        while (i < n && i - start < max_run) {
            if (columns ? !is_diag_kind(d[i].kind) : !streamable(d[i])) {
                const uint32_t t = d[i].target;
                if (t != q[0] && t != q[1] && t != q[2]) {
                    if (nx >= max_nx || nx >= 3) break;
                    q[nx++] = t;
                }
            }
            ++i;
        }
        bool fixed = true;
        for (size_t k = start; k < i; ++k) fixed = fixed && is_diag_kind(d[k].kind);
        f(start, i, nx, q[0], q[1], q[2], fixed);
    }
}

// A summary of descriptors [g0, g1), one pass with cross-group qubits q1, q2, q3 (in order of first use;
// kNoQubit when absent), by kind and qubits (GateDesc.flip kOp* bits): gates on q1 and q3 pair slots, gates on
// q2 and on qubits 0..3 lanes. For checks of pass splits: how passes apply their gates is in om, ov and loc.
void encode_pass(GateDesc* d, size_t g0, size_t g1, uint32_t q1, uint32_t q3 = kNoQubit);

// The group bits a mapped table addresses its buckets by (TableDev::map_q): bucket bit i is group
// bit q[i]. Bits join in the order they begin to differ between keys, so a table that gains a bit
// keeps every bucket where it is.
struct GroupMap {
    uint32_t n = 0;
    uint8_t q[kMaxMapBits + 1] = {};
    void clear() { n = 0; }
    // Add the qubits >= 4 that may differ between keys (not in kmask, below nq) and are not mapped
    // yet, lowest first. False when they would not fit.
    bool extend(unsigned long long kmask, uint32_t nq);
    int bit_of(uint32_t qubit) const {   // bucket bit of a qubit >= 4, or -1
        for (uint32_t i = 0; i < n; ++i)
            if (q[i] + (uint32_t)kSlotBits == qubit) return (int)i;
        return -1;
    }
    void store(TableDev* t) const {
        t->map_on = 1;
        t->map_n = n;
        for (uint32_t i = 0; i < n; ++i) t->map_q[i] = q[i];
    }
};

// Choose the bucket bits of a unit pass's dimensions and record in descriptors [g0, g1) (one pass
// with cross-group qubits q[0..2], kNoQubit when absent, at most dims of them) how the pass
// applies each gate (GateDesc.om, ov, loc). Every qubit >= 4 a gate tests or changes must be
// mapped. Dimensions without a cross-group qubit take the lowest free bucket bits.
void encode_unit_pass(GateDesc* d, size_t g0, size_t g1, const uint32_t q[3], const GroupMap& map, uint32_t dims,
                      uint32_t dim[3]);

// The same for a pass over a hashed table, whose columns (sqc_unit.cuh) are the keys that differ in its
// pairing qubits q[0..1], any qubits (split_passes with columns; kNoQubit when absent: a low qubit takes its
// place, so that a column always has four keys); dim gets them.
void encode_column_pass(GateDesc* d, size_t g0, size_t g1, const uint32_t q[2], uint32_t dim[3]);

// The same for a slot pass (walk_slots) with cross-group qubits q[0..2] (kNoQubit when absent); dim as above.
// form 1: a slot to a lane (walk_slots), 2: four (walk_low; no cross-group qubits).
void encode_slot_pass(GateDesc* d, size_t g0, size_t g1, uint32_t form, const uint32_t q[3], uint32_t dim[3]);

// Passes of a descriptor sequence over a hashed table: column passes (split_passes with columns, at most `two`
// (1 or 2) pairing qubits) or slot passes (at most max_nx cross-group qubits). A slot pass runs the absent slots
// of its units along. It is taken where the state is small (groups) or its groups hold enough keys, those that
// branching gates on low qubits will add among them, and it takes the gates of at least two column passes, or `spare`
// when it needs lookups (a cross-group qubit); a pass that is one column pass either way where the state is small,
// or FP64 groups hold enough keys. (us, start
// of the sequence to its end, columns against slots: 24 gates on low qubits, FP64, 2^12 groups of 16 keys 169
// and 45, 2^16 478 and 255; 36 gates on the low and two other qubits, 2^11 groups of 16 keys 344 and 69, 30000 of one key
// 1018 and 492; but a million keys in groups of one or two, 60 gates, few branching: 7.4 ms and 14.)
// f(g0, g1, form, q1, q2, q3, keys_fixed): form 0, a column pass and its pairing qubits, or a slot pass (encode_slot_pass)
// and its cross-group ones.
constexpr unsigned long long kSlotSmall = 1ULL << 15;   // groups of a small state
template <class F>
void plan_hashed(const GateDesc* d, size_t n, size_t max_run, uint32_t max_nx, uint32_t two, uint32_t spare, bool dbl,
                 unsigned long long groups, unsigned long long keys, F&& f) {
    for (size_t i = 0; i < n;) {
        // the slot pass from here, and the column passes over the same gates
        struct { size_t g1; uint32_t nx, q[3]; bool fixed; } slot{}, col{};
        split_passes(d + i, std::min(n - i, max_run), max_run, max_nx, [&](size_t g0, size_t g1, uint32_t nx, uint32_t q1, uint32_t q2, uint32_t q3, bool fixed) {
            if (g0 == 0) slot = {i + g1, nx, {q1, q2, q3}, fixed};
        });
        size_t cols = 0;
        split_passes(d + i, slot.g1 - i, max_run, two, [&](size_t g0, size_t g1, uint32_t nx, uint32_t q1, uint32_t q2, uint32_t q3, bool fixed) {
            if (g0 == 0) col = {i + g1, nx, {q1, q2, q3}, fixed};
            ++cols;
        }, true);
        uint32_t low = 0;   // low qubits with a branching gate
        for (size_t k = i; k < slot.g1; ++k)
            if (is_branch_kind(d[k].kind) && d[k].target < (uint32_t)kSlotBits) low |= 1u << d[k].target;
        const unsigned long long held = std::min(keys << __builtin_popcount(low), 16 * groups);   // (keys: at most 2^62)
        const bool slots = slot.nx ? cols >= spare && (groups <= kSlotSmall || held >= 8 * groups)
                                   : cols >= 2 ? groups <= kSlotSmall || held >= 4 * groups : groups <= kSlotSmall / 4 || (dbl && held >= 4 * groups);
        const auto& p = slots ? slot : col;
        const uint32_t form = !slots ? 0u : !dbl && !slot.nx && groups > kSlotSmall / 2 ? 2u : 1u;
        f(i, p.g1, form, p.q[0], p.q[1], p.q[2], p.fixed);
        i = p.g1;
    }
}

// Whether an encoded pass has a gate with a coefficient that is not finite.
inline bool odd_pass(const GateDesc* d, size_t g0, size_t g1) {
    for (size_t k = g0; k < g1; ++k)
        if (d[k].loc >> kLocOp >= UO_ODD) return true;
    return false;
}

// An order of gates g[0..n) that passes fuse better, as a permutation: perm[i] is the index of
// the i-th gate to apply. Passes are built greedily from the first gate not yet placed: a gate
// within the next `window` joins the pass when it commutes with every gate it moves ahead of
// (neither changes a qubit the other touches: a gate changes its target, unless it is
// diagonal, and only reads its controls) and the pass still has room for it (at most max_nx
// cross-group qubits, max_run device gates). The pass's cross-group qubits are the set, among
// the first-use choice and the max_nx-subsets of the first kSchedCandidates qubits gates pair
// across, that takes the most device gates over the first kSchedTrialWindow gates of the
// window. Commuting gates give the same state in either order; rounding and pruning follow the
// new order. Deterministic: a function of the gates.
void schedule_gates(const sqc_gate* g, size_t n, uint32_t max_nx, size_t max_run, size_t window, uint32_t* perm);
constexpr uint32_t kSchedCandidates = 6;
constexpr uint32_t kSchedTrialWindow = 64;   // gates the candidate choices are compared over
constexpr size_t kScheduleWindow = 256;
// Longer gate arrays (indices no longer fit 32 bits) keep the order given.
constexpr uint64_t kScheduleMaxGates = 0xFFFFFFFFULL;

// Largest number of 16-key groups a state can ever hold while running a gate sequence whose
// planning ended in p (starting from keys that agreed on every bit of the starting kmask):
// 2^(bits >= 4 that have ever differed between keys).
unsigned long long group_bound(const Planner& p, uint32_t nq);

}  // namespace sqc
