"""How passes apply their gates by place (GateDesc.om, ov, loc), on the CPU: random gates are planned into
passes and encoded for unit passes over mapped tables, and for column and slot passes over hashed ones; the
encoded words, followed place by place as the kernels follow them, must do to a state what the gates do to its keys.
"""
import pytest

from test_host_engine import engine_objects, run  # noqa: F401  (the fixture)

EMULATE = r"""
    // A unit's places: bit i of a lane is key bit lane_q[i], bit i of a slot slot_q[i] (64: no such bit, the place
    // must stay empty); `base` has those bits 0. uid: the base bucket of a unit pass, else hashed.
    struct Place { std::vector<uint32_t> lane_q, slot_q; };
    auto follow = [&](State& st, const GateDesc& g, const Place& pl, unsigned long long base, bool hashed, uint32_t uid) {
        const uint32_t L = 1u << pl.lane_q.size(), S = 1u << pl.slot_q.size();
        auto key = [&](uint32_t lane, uint32_t slot, bool* ok) {
            unsigned long long k = base;
            *ok = true;
            for (size_t i = 0; i < pl.lane_q.size(); ++i) if (lane >> i & 1) { if (pl.lane_q[i] > 63) *ok = false; else k |= 1ULL << pl.lane_q[i]; }
            for (size_t i = 0; i < pl.slot_q.size(); ++i) if (slot >> i & 1) { if (pl.slot_q[i] > 63) *ok = false; else k |= 1ULL << pl.slot_q[i]; }
            return k;
        };
        unsigned long long in_lane = 0;
        for (uint32_t q : pl.slot_q) if (q < 64) in_lane |= 1ULL << q;
        const uint32_t loc = g.loc, op = loc >> kLocOp, tb = (loc >> kLocBit) & 31u;
        if (!hashed && (uid & g.om) != g.ov) return;
        std::vector<uint32_t> act(L), bit(L), one(L);
        for (uint32_t l = 0; l < L; ++l) {
            const bool flip = loc & kLocFlip;
            if (hashed) {
                bool ok;
                const unsigned long long kb = key(l, 0, &ok);
                const bool on = (kb & (g.ctrl & ~in_lane)) == (g.cval & ~in_lane);
                act[l] = on ? (loc >> kLocSlots) & 15u : 0u;
                const uint32_t word = loc & kLocHigh ? (uint32_t)(kb >> 32) : (uint32_t)kb;
                one[l] = (((loc >> kLocSlotBit) & 15u) ^ (!(loc & kLocLane) && (word >> tb & 1u) ? 15u : 0u)) & act[l];
                bit[l] = (flip ? 1u : 0u) | (flip != ((l >> tb & 1u) != 0) ? 2u : 0u);   // bit 0: pairs of slots, bit 1: of lanes
            } else {
                const bool on = (((loc >> kLocLaneVal) ^ l) & loc & 31u) == 0, at = (loc & kLocLane) && (l >> tb & 1u);
                act[l] = on ? (loc >> kLocSlots) & 15u : 0u;
                one[l] = ((((loc >> kLocSlotBit) & 15u) ^ (at ? 15u : 0u)) & act[l]) ^ ((uid >> tb & 1u) && !(loc & kLocLane) ? act[l] : 0u);
                bit[l] = at != flip ? 3u : 0u;
            }
        }
        // the form of the op code: 0 diagonal, 1 pairs of slots s and s + 1, 2 of s and s + 2, 3 of lanes
        int form;
        if (op >= UO_ODD) form = is_diag_kind(g.kind) ? 0 : op == UO_ODD + 1 ? 3 : op == UO_ODD + 2 ? 2 : 1;
        else if (op >= UO_Z && op <= UO_PHASE) form = 0;
        else if (op < UO_Z) form = op & 1 ? 3 : 1;
        else if (op >= UO_ALL3 && (op - UO_ALL3) % 2 == 0) form = 2;
        else if (op >= UO_PAIR3 && (op - UO_PAIR3) % 2 == 0) form = 2;
        else form = (op - UO_ALL) & 1 ? 3 : 1;
        if (op >= UO_ALL && op < UO_ODD && !(op >= UO_PAIR3 && (op - UO_PAIR3) % 2 == 0))
            for (uint32_t l = 0; l < L; ++l) CHECK((act[l] & (S - 1)) == S - 1);   // straight-line forms take every place
        GateDesc h = g;   // the gate on one pair at a time, its place known
        h.ctrl = h.cval = 0;
        for (uint32_t l = 0; l < L; ++l)
            for (uint32_t s = 0; s < S; ++s) {
                if (!(act[l] >> s & 1u)) continue;
                const uint32_t st2 = form == 2 ? 2u : 1u;
                const uint32_t pl2 = form == 3 ? l ^ (1u << tb) : l, ps = form == 1 || form == 2 ? s ^ st2 : s;
                if (form && (pl2 < l || ps < s)) continue;   // each pair once, from its first place
                bool ok, ok2;
                const unsigned long long k = key(l, s, &ok), kp = form ? key(pl2, ps, &ok2) : k;
                if (!ok) continue;
                const bool one_bit = form == 0 ? one[l] >> s & 1u : form == 3 ? bit[l] & 2u : bit[l] & 1u;
                State two;
                auto a = st.amp.find(k), b = st.amp.find(kp);
                // as a state of one qubit: bit 0 the logical target bit
                if (a != st.amp.end()) two.amp[one_bit] = a->second;
                if (form && b != st.amp.end()) two.amp[!one_bit] = b->second;
                h.target = 0;
                h.flip = 0;
                apply_desc(two, h, 1e-14);
                auto put = [&](unsigned long long q, bool v) {
                    auto it = two.amp.find(v);
                    if (it == two.amp.end()) st.amp.erase(q); else st.amp[q] = it->second;
                };
                put(k, one_bit);
                if (form) put(kp, !one_bit);
            }
    };
    auto same = [&](const State& x, const State& y) {
        if (x.amp.size() != y.amp.size()) return false;
        for (auto& kv : x.amp) {
            auto it = y.amp.find(kv.first);
            if (it == y.amp.end() || std::abs(it->second - kv.second) > 1e-12) return false;
        }
        return true;
    };
    unsigned long long seed = 12345;
    auto rnd = [&](unsigned long long n) { seed = seed * 6364136223846793005ULL + 1442695040888963407ULL; return (seed >> 33) % n; };
    // gates on `qubits`, planned from keys that may differ in all of them
    auto draw = [&](const std::vector<uint32_t>& qubits, size_t n, unsigned long long frame) {
        Planner p;
        p.frame = frame;
        p.kmask = ~0ULL;
        for (uint32_t q : qubits) p.kmask &= ~(1ULL << q);
        p.kval = frame & p.kmask;
        std::vector<GateDesc> d;
        while (d.size() < n) {
            sqc_gate g = gate((uint32_t)rnd(13), qubits[rnd(qubits.size())], 0, 0.1 * (double)(1 + rnd(60)));
            g.phi = 0.3; g.lambda = 0.7;
            for (int c = (int)rnd(4); c > 0; --c) { const uint32_t q = qubits[rnd(qubits.size())]; if (q != g.target) g.controls |= 1ULL << q; }
            GateDesc x;
            if (plan_gate(p, g, &x)) d.push_back(x);
        }
        return d;
    };
    auto keys_of = [&](const std::vector<uint32_t>& qubits, size_t n) {
        State st;
        for (size_t i = 0; i < n; ++i) {
            unsigned long long k = 0;
            for (uint32_t q : qubits) k |= (unsigned long long)rnd(2) << q;
            st.amp[k] = Amp(0.1 + 0.01 * (double)rnd(50), 0.01 * (double)rnd(70));
        }
        return st;
    };
    int forms[4] = {0, 0, 0, 0};
"""


def test_unit_passes_by_place(engine_objects, tmp_path):  # noqa: F811
    """Mapped tables: two and three dimensions, fewer and more mapped bits than those, in any order."""
    run(engine_objects, tmp_path, EMULATE + r"""
    const std::vector<std::vector<uint32_t>> cases = {{0, 1, 2, 3}, {2, 9}, {0, 3, 30, 5}, {1, 17, 4, 40, 6, 33}, {2, 3, 8, 12, 45, 5, 61, 20}};
    for (auto& qubits : cases)
        for (uint32_t dims = 2; dims <= 3; ++dims)
            for (int rep = 0; rep < 12; ++rep) {
                GroupMap map;
                for (uint32_t q : qubits) map.extend(~(1ULL << q), 64);   // (one by one: the order they are given in)
                unsigned long long frame = 0;
                for (uint32_t q : qubits) frame |= (unsigned long long)rnd(2) << q;
                auto d = draw(qubits, 24, frame);
                State got = keys_of(qubits, 40), want = got;
                split_passes(d.data(), d.size(), 64, dims, [&](size_t g0, size_t g1, uint32_t, uint32_t q1, uint32_t q2, uint32_t q3, bool) {
                    const uint32_t q[3] = {q1, q2, q3};
                    uint32_t dim[3];
                    encode_unit_pass(d.data(), g0, g1, q, map, dims, dim);
                    auto qubit = [&](uint32_t b) { return b < map.n ? map.q[b] + 4u : 64u; };
                    const Place pl{{0, 1, 2, 3, qubit(dim[1])}, dims == 3 ? std::vector<uint32_t>{qubit(dim[0]), qubit(dim[2])} : std::vector<uint32_t>{qubit(dim[0])}};
                    std::set<uint32_t> units;
                    for (uint32_t b = 0; b < 1u << map.n; ++b) {
                        uint32_t u = b;
                        for (uint32_t i = 0; i < dims; ++i) u &= ~(1u << dim[i]);
                        units.insert(u);
                    }
                    for (uint32_t u : units) {
                        unsigned long long base = 0;
                        for (uint32_t i = 0; i < map.n; ++i) base |= (unsigned long long)(u >> i & 1u) << (map.q[i] + 4);
                        for (size_t k = g0; k < g1; ++k) follow(got, d[k], pl, base, false, u);
                    }
                    for (size_t k = g0; k < g1; ++k) apply_desc(want, d[k], 1e-14);
                    ++forms[dims];
                });
                CHECK(same(got, want));
            }
    CHECK(forms[2] >= 60 && forms[3] >= 60);
    """)


@pytest.mark.parametrize("max_nx", [1, 2, 3])
def test_hashed_passes_by_place(engine_objects, tmp_path, max_nx):  # noqa: F811
    """Hashed tables: column passes with none, one and two pairing qubits, slot passes of both forms with up to
    three cross-group qubits, as plan_hashed chooses them for small, dense and thin states in both precisions."""
    run(engine_objects, tmp_path, EMULATE + r"""
    const std::vector<std::vector<uint32_t>> cases = {{0, 1, 2, 3}, {0, 2, 50}, {1, 3, 20, 47, 5}, {0, 1, 2, 3, 33, 8}, {3, 63, 32, 31, 4, 12, 0, 2, 40}};
    const unsigned long long sizes[3][2] = {{100, 100}, {1 << 20, 1 << 24}, {1 << 20, 1 << 20}};
    for (auto& qubits : cases)
        for (auto& size : sizes)
            for (int dbl = 0; dbl < 2; ++dbl)
                for (int rep = 0; rep < 8; ++rep) {
                    unsigned long long frame = 0;
                    for (uint32_t q : qubits) frame |= (unsigned long long)rnd(2) << q;
                    auto d = draw(qubits, 24, frame);
                    State got = keys_of(qubits, 30), want = got;
                    size_t at = 0;
                    plan_hashed(d.data(), d.size(), 16, MAXNX, MAXNX < 2 ? MAXNX : 2, 3, dbl != 0, size[0], size[1],
                                [&](size_t g0, size_t g1, uint32_t form, uint32_t q1, uint32_t q2, uint32_t q3, bool fixed) {
                        CHECK(g0 == at && g1 > g0 && g1 - g0 <= 16);
                        at = g1;
                        const uint32_t q[3] = {q1, q2, q3};
                        uint32_t dim[3];
                        Place pl;
                        auto opt = [](uint32_t x) { return x == kNoQubit ? 64u : x; };
                        if (form) {
                            encode_slot_pass(d.data(), g0, g1, form, q, dim);
                            CHECK(form == 1 || (!dbl && q1 == kNoQubit));
                            pl = form == 2 ? Place{{2, 3}, {0, 1}} : Place{{0, 1, 2, 3, opt(q1)}, {opt(q2), opt(q3)}};
                        } else {
                            encode_column_pass(d.data(), g0, g1, q, dim);
                            CHECK(dim[0] < 64 && dim[1] < 64 && dim[0] != dim[1]);
                            pl = Place{{}, {dim[0], dim[1]}};
                        }
                        unsigned long long inside = 0;
                        for (uint32_t x : pl.lane_q) if (x < 64) inside |= 1ULL << x;
                        for (uint32_t x : pl.slot_q) if (x < 64) inside |= 1ULL << x;
                        std::set<unsigned long long> bases;
                        for (auto& kv : got.amp) bases.insert(kv.first & ~inside);
                        for (unsigned long long b : bases)
                            for (size_t k = g0; k < g1; ++k) follow(got, d[k], pl, b, true, 0);
                        bool diag = true;
                        for (size_t k = g0; k < g1; ++k) { diag = diag && is_diag_kind(d[k].kind); apply_desc(want, d[k], 1e-14); }
                        CHECK(diag == fixed);
                        ++forms[form];
                    });
                    CHECK(at == d.size() && same(got, want));
                }
    CHECK(forms[0] > 100 && forms[1] > 100 && forms[2] > 5);
    """.replace("MAXNX", str(max_nx)))
