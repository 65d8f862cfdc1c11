// Plain data structures shared by the host engine and the kernels (no device code).
#pragma once
#include <cstdint>

namespace sqc {

constexpr int kSlots = 16;
constexpr int kSlotBits = 4;
constexpr uint32_t kMaxProbe = 4096;  // buckets probed before a claim reports the table full
constexpr int kThreads = 256;
constexpr int kMaxRun = 64;           // gates fused into one pass at most
constexpr unsigned kFull = 0xffffffffu;

enum Status : unsigned int {
    ST_OK = 0,
    ST_TABLE_FULL = 1,   // a claim found no free bucket within kMaxProbe (state no longer valid)
    ST_DUPLICATE = 2,    // set_state saw the same key twice
    ST_GROW = 3,         // a pair pass refused to start: the table might overflow (state intact)
    ST_TIMEOUT = 4,      // a bounded wait inside a pass ran out (state no longer valid)
    ST_BAD_KEY = 5       // a loaded key has a bit at or above the register's qubit count
};

// gate kinds (0..12 = sqc_gate.kind); KYPH is internal: the diagonal left over when an
// uncontrolled Y is turned into a relabelling of the keys (bit 0 -> -i, bit 1 -> +i).
enum Kind : uint32_t { KX = 0, KY, KZ, KH, KPHASE, KRZ, KRX, KRY, KS, KSDG, KT, KTDG, KU, KCOUNT, KYPH = 13 };

struct alignas(16) Header {
    unsigned long long group;   // key >> 4 of the bucket's keys
    unsigned int epoch;         // live iff equal to the state's epoch
    unsigned int aux;           // presence mask: bit j is set iff key (group << 4) | j is held
};

constexpr unsigned kNoBucket = 0xFFFFFFFFu;   // no bucket: the group is absent

// Where a group's bucket is. A *mapped* table addresses groups directly: bucket bit i is group
// bit map_q[i], for the map_n group bits that may differ between keys (in the order they began
// to); every other bit of a stored group is 0, so the address is exact and no probing is needed.
// A *hashed* table (map_on 0) probes linearly from a hash of the group.
constexpr uint32_t kMaxMapBits = 31;

struct TableDev {
    Header* hdr;
    unsigned long long* keys;
    void* amps;
    unsigned int* list;         // live buckets, in claim order
    unsigned long long mask;    // nb - 1
    uint32_t map_on;            // 1: mapped, 0: hashed
    uint32_t map_n;             // mapped group bits
    uint8_t map_q[kMaxMapBits + 1];
};

// Device-resident control block of one state. Per-pass bookkeeping happens here, on the
// device, so a recorded sequence of passes replays without host involvement.
struct Ctl {
    unsigned int epoch;             // live-bucket epoch of the table
    unsigned int status;            // Status; nonzero stops every later pass until the host repairs
    unsigned int done;              // blocks finished in the running pass
    unsigned int bar;               // blocks that have met between the passes of a run (0 outside one)
    unsigned long long seq;         // passes completed since the last reset
    unsigned long long nnz;         // keys held
    unsigned long long list_n;      // live buckets (list entries) committed at the last pass end
    unsigned long long list_tail;   // list entries appended so far
    unsigned long long empty_groups;  // live buckets without a key after the last pass
    unsigned long long acc_nnz, acc_upd, acc_empty;
    unsigned long long amp_updates; // sum over gates of input nonzeros, since the last reset
    unsigned long long alg_bytes;   // algorithmic bytes of the passes, since the last reset
    unsigned long long alg_bytes_pair;  // the part of alg_bytes moved by pair passes
    unsigned long long out_count;   // readout counter
    double acc[6];                  // reductions: norm, compare
    unsigned long long acc_max;     // bit pattern of a non-negative double (max |a-b|)
    unsigned long long bar_len;     // a run's live buckets before a pass that walks the list, tagged with the pass
                                    // (0 outside a run)
};

// Gate descriptor with host-resolved coefficients (std::cos/std::sin on the host, so the
// device and the CPU oracle use identical values) in the stored-key frame: the gate acts on
// a stored key s iff (s & ctrl) == cval, and the member's logical target bit is
// ((s >> target) & 1) ^ flip.
struct alignas(16) GateDesc {
    uint32_t kind, target;
    unsigned long long ctrl, cval;
    uint32_t flip, pad;
    double c, s;          // phase/T/Tdg: cos, sin; rz/rx/ry: cos, sin of theta/2; h: 1/sqrt(2)
    double m[8];          // u: m00, m01, m10, m11 as (re, im)
    float cf, sf;         // float copies for FP32 states
    float mf[8];
    // how its pass (sqc_unit.cuh) applies the gate, set by encode_unit_pass on the host: in a mapped
    // table the unit's base bucket u satisfies the controls outside the unit iff (u & om) == ov (in a
    // hashed one the column's key is tested against ctrl and cval); loc holds the rest (kLoc* fields)
    uint32_t om, ov, loc, pad2;
};

// GateDesc.loc: what a unit pass does for the gate, by place in the unit.
constexpr uint32_t kLocLaneVal = 5;        // bits 0..4: controlled lane bits (qubits 0..3, dimension 1), 5..9: their values
constexpr uint32_t kLocSlots = 10;         // bits 10..13: slots whose controls (dimensions 0 and 2) hold
constexpr uint32_t kLocSlotBit = 14;       // bits 14..17: diagonal gates: logical target bit per slot, before the next two
constexpr uint32_t kLocBit = 18;           // bits 18..22: the target's bit of the lane index or of the unit's base (31: none)
constexpr uint32_t kLocLane = 1u << 23;    // ... of the lane index
constexpr uint32_t kLocFlip = 1u << 24;    // the stored frame flips the target bit (pairing gates)
constexpr uint32_t kLocHigh = 1u << 25;    // hashed tables: kLocBit counts from bit 32 of the column's key
constexpr uint32_t kLocOp = 26;            // bits 26..31: UOp
// Pairing gates come as their controls inside the unit ask, on slots 0-1 and 2-3 or (UO_PAIR3) 0-2 and
// 1-3, and, when they have none there (every lane and slot takes part), straight through (UO_ALL,
// UO_ALL3).
enum UOp : uint32_t {
    UO_X_PAIR = 0, UO_X_SHFL, UO_Y_PAIR, UO_Y_SHFL, UO_H_PAIR, UO_H_SHFL, UO_RX_PAIR, UO_RX_SHFL, UO_RY_PAIR,
    UO_RY_SHFL, UO_U_PAIR, UO_U_SHFL, UO_Z, UO_S, UO_SDG, UO_YPH, UO_RZ, UO_PHASE,
    UO_ALL = 18,    // + 0..11: the forms above
    UO_ALL3 = 30,   // + 0, 2, .., 10: UO_X_PAIR .. UO_U_PAIR on dimension 2
    UO_PAIR3 = 31,  // + 0, 2, .., 10: the same with controls inside the unit
    UO_ODD = 61     // a gate with a coefficient that is not finite; + 1: pairs lanes, + 2: on dimension 2
};

// GateDesc.flip bits: the frame's flip (the only one passes read), and encode_pass's summary of a gate.
constexpr uint32_t kOpFlip = 1u << 0;      // the stored frame flips the target bit
constexpr uint32_t kOpPair = 1u << 1;      // pairs the a and b slots (first cross-group qubit)
constexpr uint32_t kOpShfl = 1u << 2;      // partner slot in lane ^ (1 << off_log2)
constexpr uint32_t kOpOffShift = 3;        // off_log2: bits 3..5
constexpr uint32_t kOpCtrl = 1u << 6;      // controls to test per key
constexpr uint32_t kOpBranch = 1u << 7;    // H, Rx, Ry, U
constexpr uint32_t kOpSwap = 1u << 8;      // X, Y
constexpr uint32_t kOpOneSided = 1u << 9;  // diagonal gate that leaves bit-0 keys unchanged
constexpr uint32_t kOpLowBit = 1u << 10;   // target < 4: the target bit is in the slot index
constexpr uint32_t kOpPair3 = 1u << 11;    // pairs slots a with c and b with d (third cross-group qubit)

struct PruneBits {
    unsigned long long d;   // bit pattern of thr (double)
    unsigned int f;         // bit pattern of the largest float below thr
};

constexpr uint32_t kNoQubit = 0xFFFFFFFFu;
constexpr unsigned long long kKeysUnknown = 1ULL << 62;

// Exact sums of products (sqc_exact.cuh): fixed-point numbers with their least significant bit
// at 2^kSumLsb, kSumChunks 32-bit pieces each held in a 64-bit counter.
constexpr int kSumChunks = 10;
constexpr int kSumLsb = -256;
enum SumIndex { SUM_NORM = 0, SUM_ORE, SUM_OIM, SUM_NA, SUM_NB, SUM_NB_ONLY, kSums };
struct ExactSums {
    unsigned long long c[kSums][kSumChunks];
};

// Where a gate of a unit pass acts: GateDesc.om, ov, loc, and the amp updates a present key counts.
struct alignas(16) UnitHead {
    uint32_t om, ov, loc, weight;
};

struct PassArgs {
    TableDev t;
    Ctl* ctl;
    const GateDesc* gates;
    uint32_t g0, g1;        // gate range [g0, g1) of this pass
    uint32_t nx;            // cross-group qubits of the pass
    uint32_t keys_fixed;    // 1: every gate of the pass is diagonal (no key changes)
    uint32_t amp_bytes;     // 16 (FP64) or 8 (FP32)
    unsigned long long max_groups;   // a pass that pairs groups refuses to start when its groups could
                                     // exceed this: min(grow_bound, n << nx, n + key_bound) > max_groups
    PruneBits prune;
    unsigned long long grow_bound;   // groups the state can hold after the pass, at most
    unsigned long long key_bound;    // keys it can hold after the pass, at most: a pass makes no more
                                     // groups than that (hashed tables; at most kKeysUnknown)
    // mapped bits in use after the pass (mapped tables), dimensions of a unit (2 or 3) and the bucket
    // bit (mapped) or qubit (hashed; 64: none) of each dimension
    uint32_t dn, dims, dim[3];
    uint32_t odd;           // 1: a gate is UO_ODD (never in a run)
    uint32_t slots;         // 1: a slot pass (hashed tables; never in a run): dim holds its cross-group qubits;
                            // 2: one without any, four slots to a lane (FP32)
    uint32_t plain;         // slot passes: FP64 products by the FP64 instruction
    UnitHead heads[kMaxRun];   // mapped tables: those of the pass's gates (read from the parameter bank)
};

// A run of passes in one launch (run_kernel). words holds the passes one after another: a record (om:
// gates in bits 0..7, the flags below, from bit 16 the mapped bits after the pass or, in a hashed
// table, its cross-group qubits; ov: the dimensions' bits, a byte each; loc: the pass's
// first gate), then the heads of its gates (mapped) or grow_bound and key_bound (hashed; PassArgs).
// All of it is read from the parameter bank.
constexpr uint32_t kRunWords = 496;        // 8 KB of parameters
constexpr uint32_t kRunFixed = 1u << 8;    // every gate is diagonal
constexpr uint32_t kRunPair = 1u << 9;     // the pass pairs groups
struct RunArgs {
    TableDev t;
    Ctl* ctl;
    const GateDesc* gates;
    PruneBits prune;
    uint32_t np, amp_bytes;
    unsigned long long max_groups;   // hashed tables: as in PassArgs
    UnitHead words[kRunWords];
};

}  // namespace sqc
