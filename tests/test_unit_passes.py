"""Unit passes over mapped tables, and their FP64 products on the integer pipes.

CPU part: the product code (sparqc_gb300/csrc/sqc_dmul.cuh) compiled for the host gives the
hardware's product for every operand pair it does not refuse, and refuses only pairs whose product
is not a normal number by exponent or with an operand that is not a finite normal number or zero.
GPU part: states at the edges of what a unit pass handles, bit for bit against the oracle.
"""
import os
import subprocess

import numpy as np
import pytest

from oracle.sparse import SparseOracle
from sparqc_gb300 import circuits, gates as G
from test_oracle import assert_identical

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sparqc_gb300", "csrc")

PROGRAM = r'''
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "sqc_dmul.cuh"
using namespace sqc;
static uint64_t bits(double x) { uint64_t u; std::memcpy(&u, &x, 8); return u; }
static double from(uint64_t u) { double x; std::memcpy(&x, &u, 8); return x; }
int main() {
    std::mt19937_64 r(7);
    unsigned long long done = 0, refused = 0, bad = 0, wrong_refusal = 0;
    auto mantissa = [&]() -> uint64_t {
        uint64_t m = r() & 0xFFFFFFFFFFFFFULL;
        switch (r() % 8) {
        case 0: return 0;
        case 1: return 0xFFFFFFFFFFFFFULL;
        case 2: return m & ~0x3FFFFFFULL;              // few significant bits: exact products and ties
        case 3: return 1ULL << (r() % 52);
        case 4: return m & ~((1ULL << (r() % 52)) - 1);
        default: return m;
        }
    };
    for (int ci = 0; ci < 4000; ++ci) {
        double c;
        switch (ci % 5) {
        case 0: c = std::cos(0.37 * ci); break;
        case 1: c = std::ldexp(1.0, -(ci % 40)); break;
        case 2: c = std::nextafter(1.0, 0.0) * ((ci & 8) ? -1 : 1); break;
        case 3: c = ci % 7 ? std::sqrt(0.5) : 0.0; break;
        default: c = from((r() & 0x8000000000000000ULL) | ((600 + r() % 500) << 52) | mantissa()); break;
        }
        const DCoef k = dcoef(bits(c));
        if (!k.ok) {
            const double a = std::fabs(c);
            wrong_refusal += a <= 1.0 && a >= 0x1p-400;
            continue;
        }
        for (int i = 0; i < 4000; ++i) {
            uint64_t e = r() % 4 ? 963 + r() % 64 : r() % 2048;
            uint64_t u = (r() & 0x8000000000000000ULL) | (e << 52) | mantissa();
            if (r() % 16 == 0) u &= 0x8000000000000000ULL;
            const double a = from(u), want = a * c;
            const DUnpacked x = dunpack((uint32_t)(u >> 32), (uint32_t)u, k.min_exp);
            if (x.slow) {
                ++refused;
                const int pe = (int)e + (int)((bits(c) >> 52) & 0x7FF) - 1023;   // product exponent, or one less
                wrong_refusal += e > 0 && e < 2047 && pe >= 2;
                continue;
            }
            uint32_t hi, lo;
            dproduct(x, k.hi, k.lo, k.exp, (uint32_t)(bits(c) >> 32), &hi, &lo);
            ++done;
            bad += (((uint64_t)hi << 32) | lo) != bits(want);
        }
    }
    std::printf("%llu %llu %llu %llu\n", done, refused, bad, wrong_refusal);
    return 0;
}
'''


def test_integer_products_equal_the_hardware(tmp_path):
    src = tmp_path / "dmul.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "dmul"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-x", "c++", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True)
    done, refused, bad, wrong = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert bad == 0 and wrong == 0
    assert done > 5_000_000 and refused > 10_000


def _both(nq, gates, precision, init=None, **kw):
    from sparqc_gb300.engine import State
    st = State(nq, precision=precision, **kw)
    o = SparseOracle(precision)
    if init is not None:
        st.set_state(*init)
        o.set_state(*init)
    st.apply(gates)
    o.apply(gates)
    got, want = st.state(sorted=True), o.state(sorted=True)
    stats = st.stats()
    st.close()
    assert_identical(got, want)
    assert stats["amp_updates"] == o.amp_updates
    return got


KINDS = ((G.Z, G.S, G.SDG, G.T, G.TDG, G.RZ, G.PHASE), (G.X, G.Y), (G.H, G.RX, G.RY, G.U))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("cross", [0, 3])
@pytest.mark.parametrize("nq", [1, 4, 5, 6, 7, 8, 9, 12, 13])
def test_small_registers(nq, cross, precision):
    """Fewer mapped bits than a unit has dimensions, and the first sizes past the single launch."""
    rng = circuits.SplitMix64(circuits.stream_seed("unit-small", nq, precision))
    g = circuits.random_circuit(nq, nq, 150, min(3, nq - 1), rng, kinds=KINDS)
    _both(nq, g, precision, max_cross_qubits=cross)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("seed", range(3))
def test_loaded_states(seed, precision):
    """States whose constant bits are set (the stored frame), with thin spans and with empty slots."""
    rng = np.random.default_rng(seed)
    nq, free = 40, [2, 3, 5, 11, 17, 18, 30, 39][:6 + seed]
    sub = rng.choice(1 << len(free), 1 << (len(free) - seed), replace=False)
    keys = np.full(sub.size, (1 << 4) | (1 << 20) | (1 << 33), np.uint64)
    for i, q in enumerate(free):
        keys |= ((sub >> i) & 1).astype(np.uint64) << np.uint64(q)
    a = rng.standard_normal((2, keys.size))
    g = circuits.random_circuit(nq, 12, 120, 2, circuits.SplitMix64(seed), prefix_h=False, kinds=KINDS)
    _both(nq, g, precision, init=(keys, a[0], a[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_thin_states_walk_the_list_and_leave_the_map(precision):
    """Keys that spread over ever more qubits: few live buckets among the mapped ones, then more
    mapped bits than the table holds (the state moves to a hashed table)."""
    nq = 60
    gs = [(G.H, q) for q in range(6)] + [(G.RX, 3, (), 0.3)]
    for i, t in enumerate(range(6, 50)):
        gs += [(G.X, t, (i % 6, (i + 1) % 6)[: 1 + i % 2]), (G.RZ, t, (i % 5,), 0.1 * i)]
        if i % 9 == 4:
            gs += [(G.RY, i % 6, (t,), 0.7), (G.H, t)]
    _both(nq, G.gate_array(gs), precision)


@pytest.mark.gpu
def test_fp64_products_beyond_the_integer_path():
    """Amplitudes and coefficients the integer products leave to the FP64 instruction: subnormal and
    tiny values, zero and one as coefficients, next to ordinary ones."""
    rng = np.random.default_rng(5)
    n = 1 << 9
    keys = np.arange(n, dtype=np.uint64)
    scale = 10.0 ** rng.choice([0, -5, -150, -290, -300, -308, -320], (2, n))
    a = rng.standard_normal((2, n)) * scale
    a[:, rng.random(n) < 0.2] = 0.0
    a[1, rng.random(n) < 0.2] = -0.0
    tiny = [0.0, np.pi, 2 * np.pi, 1e-5, 1e-140, 1e-300, np.pi / 2, 1.234]
    gs = []
    for i, th in enumerate(tiny):
        gs += [(G.RZ, i % 9, (), th), (G.PHASE, (i + 2) % 9, (), th), (G.T, i % 9)]
    diag = G.gate_array(gs)
    _both(9, diag, 64, init=(keys, a[0], a[1]))
    big = a.copy()
    big[0] += rng.standard_normal(n)   # every key survives the pruning of branching gates
    gs += [(k, (i + 3 * j) % 9, (), th) for j, k in enumerate((G.RX, G.RY, G.U, G.H)) for i, th in enumerate(tiny)]
    _both(9, G.gate_array(gs), 64, init=(keys, big[0], big[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_measured_bits_keep_the_masks(precision):
    """A measurement removes keys behind the passes' back: the presence masks follow it."""
    from sparqc_gb300.engine import State
    nq = 12
    g = circuits.random_circuit(nq, 10, 120, 2, circuits.SplitMix64(3), kinds=KINDS)
    st = State(nq, precision=precision)
    st.apply(g)
    for q in (1, 7):
        st.measure(q, 0.4)
    k, r, i = st.state(sorted=True)
    st.apply(g)
    o = SparseOracle(precision)
    o.set_state(k, r, i)
    o.apply(g)
    assert_identical(st.state(sorted=True), o.state(sorted=True))
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_batch_of_thin_and_tiny_circuits(precision):
    """Circuits whose keys are few among their mapped bits (their passes walk the list), circuits
    smaller than a unit, and one large enough for many chunks, in one launch."""
    from sparqc_gb300.engine import Batch
    thin = []
    for n in (10, 14, 18):
        gs = [(G.H, q) for q in range(5)] + [(G.X, 5 + i, (i % 5, (i + 2) % 5)[: 1 + i % 2]) for i in range(n)]
        gs += [(G.RZ, 5 + i, (i % 5,), 0.3 + i) for i in range(0, n, 3)] + [(G.RY, 5 + n - 1, (1,), 0.4), (G.H, 2)]
        thin.append((40, G.gate_array(gs)))
    rng = circuits.SplitMix64(circuits.stream_seed("unit-batch", precision))
    small = [(nq, circuits.random_circuit(nq, nq, 40, min(2, nq - 1), rng, kinds=KINDS)) for nq in (1, 3, 4, 5, 6, 7)]
    big = [(20, circuits.random_circuit(20, 16, 120, 2, rng, kinds=KINDS))]
    cs = thin + small + big
    b = Batch(precision=precision)
    b.prepare(cs)
    b.run()
    b.sync()
    upd = 0
    for i, (_, g) in enumerate(cs):
        o = SparseOracle(precision)
        o.apply(g)
        assert_identical(b.state(i), o.state(sorted=True))
        upd += o.amp_updates
    assert b.stats()["amp_updates"] == upd
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nq,k", [(3, 3), (5, 5), (16, 9), (30, 15), (64, 17)])
def test_key_ordered_readout(nq, k, precision):
    """Readouts of mapped tables come in key order without a sort: whole, by pattern (bits in and
    outside the map, patterns nothing matches), without negligible entries, and sampled."""
    from sparqc_gb300.engine import State
    rng = circuits.SplitMix64(circuits.stream_seed("rank", nq, precision))
    gs = circuits.random_circuit(nq, k, 60 + k, min(2, nq - 1), rng, kinds=KINDS)
    gs = np.concatenate([gs, G.gate_array([(G.X, q) for q in range(0, nq, 2)])])   # a frame on every other bit
    st, o = State(nq, precision=precision), SparseOracle(precision)
    st.apply(gs)
    o.apply(gs)
    full = o.state(sorted=True)
    assert_identical(st.state(sorted=True), full)
    assert_identical(st.state(sorted=False), full)
    top, low = 1 << (nq - 1), 1
    key = int(full[0][full[0].size // 2])
    for mask, value in ((low, low), (top, key & top), (top, ~key & top), (low | top, key & (low | top)), (2 % (1 << nq), 1),
                        ((1 << nq) - 1, key), (6, key & 6)):
        want = (full[0] & np.uint64(mask)) == np.uint64(value)
        assert_identical(st.state_where(mask, value), tuple(x[want] for x in full))
    keep = ~((np.abs(full[1]) < 1e-14) & (np.abs(full[2]) < 1e-14))
    assert_identical(st.state(drop_negligible=True), tuple(x[keep] for x in full))
    assert np.isin(st.sample(200, seed=3), full[0]).all()
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("k,depth", [(14, 300), (17, 900)])
def test_first_run_of_a_full_state_is_mapped(k, depth):
    """A new state whose keys fill their span grows a mapped table (its refused passes are replayed)
    however many branching gates the circuit has, and the next run of it does the same work."""
    from sparqc_gb300.engine import State
    g = circuits.random_circuit(30, k, depth, 2, circuits.SplitMix64(k), kinds=KINDS)
    st, o = State(30), SparseOracle()
    o.apply(g)
    st.apply(g)
    first = st.state(sorted=True)
    passes = st.stats()["passes"]
    assert st.stats()["replays"] > 0
    st.set_zero()
    st.apply(g)
    assert_identical(first, o.state(sorted=True))
    assert_identical(st.state(sorted=True), first)
    assert st.stats()["passes"] == 2 * passes
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("nq,k,depth", [(8, 5, 60), (12, 9, 200), (16, 12, 700), (18, 16, 300), (24, 20, 120), (24, 23, 60)])
def test_runs_of_passes_equal_single_passes(nq, k, depth, precision):
    """The passes of a flush in one launch leave what a launch each leaves (timed passes are launched
    one by one): keys, amplitudes, counts; one block, several, a full wave, and states too large."""
    from sparqc_gb300 import engine
    g = circuits.random_circuit(nq, k, depth, 3, circuits.SplitMix64(circuits.stream_seed("runs", nq * 100 + k)))
    one = engine.State(nq, precision=precision, time_passes=True)
    run = engine.State(nq, precision=precision)
    for st in (one, run):
        st.apply(g)
        st.sync()
    a, b = one.stats(), run.stats()
    for f in ("passes", "amp_updates", "alg_bytes", "alg_bytes_pair", "passes_pair", "replays"):
        assert a[f] == b[f], f
    assert_identical(run.state(), one.state())


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("keys", [40, 300, 1500])
def test_runs_that_walk_the_list(keys, precision):
    """Few live buckets among the mapped ones: every pass of a run walks the list, whose length
    changes from pass to pass; with 1500 keys later passes walk every unit."""
    from sparqc_gb300 import engine
    rng = np.random.default_rng(keys)
    key = np.unique(rng.integers(0, 1 << 16, keys, dtype=np.uint64))
    amp = rng.standard_normal((2, key.size)) / np.sqrt(key.size)
    c = circuits.SplitMix64(circuits.stream_seed("list", keys))
    g = [(G.X, 4 + int(c.next() % 12), [int(c.next() % 4)], 0.0) if i % 5 else
         (G.RY, int(c.next() % 16), [(int(c.next() % 3) + 13)], 0.4) for i in range(80)]
    g = G.gate_array([(a, t, [q for q in ctl if q != t], th) for a, t, ctl, th in g])
    states = []
    for timed in (True, False):
        st = engine.State(16, precision=precision, time_passes=timed)
        st.set_state(key, amp[0], amp[1])
        st.apply(g)
        st.sync()
        states.append((st.state(), st.stats()))
    (sa, a), (sb, b) = states
    assert [a[f] for f in ("passes", "amp_updates", "alg_bytes")] == [b[f] for f in ("passes", "amp_updates", "alg_bytes")]
    assert_identical(sb, sa)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("cross", [0, 1])
@pytest.mark.parametrize("keys", [1, 31, 700, 20000])
def test_column_passes(keys, cross, precision):
    """Keys spread over 64 qubits (hashed tables): passes whose two pairing qubits are low, high or one of
    each, passes with none, controls on many qubits, inside the column and out, diagonal targets in
    either half of the key; groups that appear and that empty."""
    rng = np.random.default_rng(keys)
    spread = np.uint64(0xFEDCBA9876543210)
    key = np.unique(np.concatenate([rng.integers(0, 1 << 63, keys, dtype=np.uint64) * np.uint64(2) + np.uint64(keys & 1),
                                    np.array([0, 0xFFFFFFFFFFFFFFFF, int(spread)][: 1 if keys == 1 else 3], np.uint64)]))
    amp = rng.standard_normal((2, key.size))
    c = circuits.SplitMix64(circuits.stream_seed("columns", keys))
    pick = lambda n: c.next() % n
    gs = []
    for i in range(48):
        t = [pick(4), 4 + pick(28), 32 + pick(32), 63, 35, 36][i % 6]
        ctl = tuple({q for q in [pick(4), pick(64), 35, 3][: pick(5)] if q != t})
        if i % 12 == 7:
            ctl = tuple(q for q in range(20, 60) if q != t)
        group = KINDS[pick(3)]
        gs.append((group[pick(len(group))], t, ctl, 0.3 + 0.1 * i) if i % 8 else (G.X, t, ctl[:1], 0.0))
    _both(64, G.gate_array(gs[: 48 if keys < 20000 else 14]), precision, max_cross_qubits=cross, init=(key, amp[0], amp[1]))


@pytest.mark.gpu
@pytest.mark.parametrize("k,buckets", [(10, 1024), (14, 64)])
def test_questions_after_one_long_call(k, buckets):
    """More gates in one call than the engine's descriptors hold: the state, its key count and its norm
    are the whole circuit's, asked for without a sync."""
    from sparqc_gb300.engine import State
    g = circuits.random_circuit(20, k, 9000, 2, circuits.SplitMix64(k), kinds=KINDS)
    st, o = State(20, initial_buckets=buckets), SparseOracle()
    o.apply(g)
    st.apply(g)
    want = o.state(sorted=True)
    assert st.nnz == want[0].size
    assert abs(st.norm2() - float((want[1] ** 2 + want[2] ** 2).sum())) < 1e-9
    assert_identical(st.state(sorted=True), want)
    st.close()


def _same(got, want):
    """Equal keys, and equal parts where neither is NaN; NaN in the same places."""
    assert np.array_equal(got[0], want[0])
    for a, b in zip(got[1:], want[1:]):
        assert np.array_equal(a, b, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("hashed", [False, True])
@pytest.mark.parametrize("kind", [G.U, G.H, G.RX, G.RY])
def test_infinite_and_nan_amplitudes(kind, hashed, precision):
    """Infinite and NaN parts follow the formulas wherever the pass puts the target: in a slot of the lane,
    in another lane (the second of two such qubits), in the bucket, in a column."""
    from sparqc_gb300.engine import State
    rng = np.random.default_rng(11)
    nq = 60 if hashed else 9
    keys = np.unique(rng.integers(0, 1 << nq, 300, dtype=np.uint64)) if hashed else np.arange(1 << nq, dtype=np.uint64)
    for qubits in ((7,), (5, 6), (6, 5, 4), (2,), (1, 8)):
        a = rng.standard_normal((2, keys.size))
        odd = rng.choice(keys.size, 24, replace=False)
        a[0, odd[:12]] = np.array([np.inf, -np.inf, np.nan, 0.0] * 3)
        a[1, odd[6:18]] = np.array([np.inf, -np.inf, np.nan, 0.0] * 3)
        gs = G.gate_array([(kind, q, ((q + 3) % nq,) if i else (), 0.9 + i, 0.4, 1.1) if kind == G.U else
                           (kind, q, (), 0.9 + i) for i, q in enumerate(qubits)])
        st, o = State(nq, precision=precision), SparseOracle(precision)
        st.set_state(keys, a[0], a[1])
        o.set_state(keys, a[0], a[1])
        st.apply(gs)
        o.apply(gs)
        _same(st.state(sorted=True), o.state(sorted=True))
        st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("where", ["mapped", "hashed", "batch"])
@pytest.mark.parametrize("gate", [(G.RX, np.nan), (G.RY, np.inf), (G.RZ, -np.inf), (G.PHASE, np.nan), (G.U, np.nan, 0.3, 0.2),
                                  (G.U, 0.7, np.nan, 0.2), (G.U, 0.7, 0.3, np.inf)])
def test_angles_that_are_not_finite(gate, where, precision):
    """A NaN or infinite angle turns amplitudes to NaN; it makes no key out of pairs that hold none, and
    absent keys stay 0 for the gates that follow."""
    from sparqc_gb300.engine import Batch, State
    nq, prefix = (60, 5) if where == "hashed" else (9, 5)
    spread = [8 * q + 3 for q in range(prefix)] if where == "hashed" else [0, 2, 4, 5, 8]
    first = [(G.H, q) for q in spread] + [(G.X, (q + 5) % nq, (q,)) for q in spread]
    for qubits in ((6,), (5, 6), (6, 5, 4), (1,), (3, 7)):
        odd = [(gate[0], q, ((q + 2) % 9,) if i else ()) + gate[1:] for i, q in enumerate(qubits)]
        after = [(G.H, (qubits[0] + 1) % 9), (G.RY, (qubits[0] + 2) % 9, (), 0.4), (G.X, qubits[0], ((qubits[0] + 4) % 9,))]
        gs = G.gate_array(first + odd + after)
        o = SparseOracle(precision)
        o.apply(gs)
        if where == "batch":
            st = Batch(precision=precision)
            st.prepare([(nq, gs)])
            st.run()
            st.sync()
            got = st.state(0)
        else:
            st = State(nq, precision=precision)
            st.apply(gs)
            got = st.state(sorted=True)
        _same(got, o.state(sorted=True))
        st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("keys", [40, 300])
def test_recorded_runs_replay(keys, precision):
    """Passes recorded on the caller's stream into a CUDA graph (two passes that walk the list, in one
    launch) do the same again at every replay: their meeting does not take the last replay's for its own."""
    import torch
    from sparqc_gb300.engine import State
    rng = np.random.default_rng(keys)
    key = np.unique(rng.integers(0, 1 << 16, keys, dtype=np.uint64))
    amp = rng.standard_normal((2, key.size)) / np.sqrt(key.size)
    gs = G.gate_array([(G.X, 4, (9,)), (G.RZ, 10, (2,), 0.4), (G.X, 5, (4, 11)), (G.RY, 6, (7, 12, 15), 0.3), (G.X, 8, (6,))]
                      if precision == 64 else
                      [(G.X, 4, (9,)), (G.X, 5, (4, 11)), (G.X, 10, (13,)), (G.RY, 6, (7, 12, 15), 0.3), (G.X, 8, (6,))])
    s = torch.cuda.Stream()
    st, o = State(16, precision=precision, initial_buckets=1 << 13, stream=s.cuda_stream), SparseOracle(precision)
    st.set_state(key, amp[0], amp[1])
    o.set_state(key, amp[0], amp[1])
    st.apply(gs)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        st.flush()
    with torch.cuda.stream(s):
        for _ in range(50):
            graph.replay()
    for _ in range(50):
        o.apply(gs)
    s.synchronize()
    assert st.stats()["passes"] == 2
    assert_identical(st.state(sorted=True), o.state(sorted=True))
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_comparing_states_on_different_bits(precision):
    """Two states whose keys differ in a bit neither maps share no key; telling that takes one look per key
    in a dense table too, about what a comparison of equal states takes (16 times it: far below the
    thousands of neighbours that a search would visit)."""
    import time
    from sparqc_gb300.engine import State
    gs = [(G.RY, q, (), 0.3 + q) for q in range(18)]
    a, b, c = State(40, precision=precision), State(40, precision=precision), State(40, precision=precision)
    a.apply(G.gate_array(gs))
    b.apply(G.gate_array(gs))
    c.apply(G.gate_array(gs + [(G.X, 30)]))

    def best(other):
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            r = a.compare(other)
            t.append(time.perf_counter() - t0)
        return r, min(t)

    (same, t_same), (apart, t_apart) = best(b), best(c)
    assert same[0] > 1 - 1e-6 and same[1] == 0.0
    assert apart[0] == 0.0 and apart[1] > 0.0
    assert t_apart < 16 * t_same


def _slot_gates(cross, seed, n=40):
    """Gates that go back and forth between the four low qubits and `cross` others, controls and phases anywhere."""
    c = circuits.SplitMix64(circuits.stream_seed("slots", seed))
    pick = lambda k: c.next() % k
    pairing = [0, 1, 2, 3] + [20, 47, 5][:cross]
    gs = []
    for i in range(n):
        group = KINDS[pick(3)]
        diag = group is KINDS[0]
        t = pick(64) if diag else pairing[pick(len(pairing))] if i >= len(pairing) else pairing[i]
        ctl = tuple({q for q in [pick(4), pick(64), pairing[pick(len(pairing))], 63][: pick(5)] if q != t})
        gs.append((group[pick(len(group))], t, ctl, 0.3 + 0.1 * i, 0.2, 0.7))
    return G.gate_array(gs)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("cross", [0, 1, 2, 3])
@pytest.mark.parametrize("groups,per", [(1, 1), (1, 16), (31, 5), (33, 16), (700, 1), (3000, 12)])
def test_slot_passes(groups, per, cross, precision):
    """Hashed tables, gates on the low qubits and up to three others in turns: units of one to eight groups, one
    to eight of them to a warp, with groups that appear and that empty; few passes for many gates."""
    from sparqc_gb300.engine import State
    rng = np.random.default_rng(groups * 100 + per)
    g = np.unique(rng.integers(0, 1 << 59, groups, dtype=np.uint64)) * np.uint64(2) + np.uint64(1)
    key = (g[:, None] << np.uint64(4)) + rng.permuted(np.tile(np.arange(16, dtype=np.uint64), (g.size, 1)), axis=1)[:, :per]
    key = np.unique(np.concatenate([key.ravel(), np.array([0, 0xFFFFFFFFFFFFFFFF], np.uint64)]))
    amp = rng.standard_normal((2, key.size))
    gs = _slot_gates(cross, cross + groups)
    _both(64, gs, precision, init=(key, amp[0], amp[1]))
    st = State(64, precision=precision)
    st.set_state(key, amp[0], amp[1])
    st.apply(gs)
    st.sync()
    assert st.stats()["passes"] <= (1 if cross <= 2 or precision == 32 else 40)
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_slot_passes_that_empty_groups_and_odd_angles(precision):
    """A slot pass that moves every key of a group away, one with NaN angles in lanes and slots."""
    key = (np.arange(200, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15)) | np.uint64(1 << 20)
    key = np.unique(key)
    amp = np.random.default_rng(2).standard_normal((2, key.size))
    move = [(G.X, 20, (q,)) for q in range(4)] + [(k, q, (20,)) for k in (G.Y, G.X) for q in range(4)] + [(G.X, 20, (63,)), (G.RY, 2), (G.RX, 1)]
    _both(64, G.gate_array(move), precision, init=(key, amp[0], amp[1]))
    from sparqc_gb300.engine import State
    odd = [(G.RX, q, (33,), np.nan) for q in (0, 3, 20)] + [(G.U, 2, (40,), 0.4, np.inf, 0.1), (G.RZ, 3, (41,), np.nan), (G.U, 1, (50,), 0.4, 0.1, np.nan)]
    gs = G.gate_array([(G.H, 0), (G.RY, 1, (), 0.4)] + odd + [(G.H, q) for q in (3, 2, 20, 1, 0)])
    st, o = State(64, precision=precision), SparseOracle(precision)
    st.set_state(key, amp[0], amp[1])
    o.set_state(key, amp[0], amp[1])
    st.apply(gs)
    o.apply(gs)
    _same(st.state(sorted=True), o.state(sorted=True))
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_a_thin_circuit_of_a_batch_spreads_over_warps(precision):
    """A circuit whose passes walk their list takes a batch about as long as a state of its own (three times it
    at most; a warp for every 32 entries takes six times it)."""
    import time
    from sparqc_gb300.engine import Batch, State
    c = circuits.SplitMix64(circuits.stream_seed("thin-batch"))
    gs = [(G.H, q) for q in range(9)] + [(G.X, 9 + i, (i % 9, (i + 4) % 9)[: 1 + i % 2]) for i in range(14)]
    for j in range(120):
        t, a, b = 9 + c.next() % 14, c.next() % 23, c.next() % 23
        gs.append((G.X, t, tuple({q for q in (a, b) if q != t})) if j % 4 else (G.RZ, t, tuple({a} - {t}), 0.3))
    gs = G.gate_array(gs)
    o = SparseOracle(precision)
    o.apply(gs)
    b = Batch(precision=precision)
    b.prepare([(40, gs)])
    st = State(40, precision=precision, initial_buckets=1 << 17)   # mapped, as the batch's slice

    def best(f):
        t = []
        for _ in range(7):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return min(t)

    def alone():
        st.set_zero()
        st.apply(gs)
        st.sync()

    def batch():
        b.run()
        b.sync()

    t_alone, t_batch = best(alone), best(batch)
    assert_identical(b.state(0), o.state(sorted=True))
    assert t_batch < 3 * t_alone, (t_batch, t_alone)
    b.close()
    st.close()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", [64, 32])
def test_readouts_of_thin_circuits_go_by_the_list(precision):
    """A few keys among 2^20 mapped groups: a batch's and a server's readout visits the live buckets in one
    launch, in key order when asked; with more keys, or fewer groups, it stays the ranked one (three)."""
    from sparqc_gb300.engine import Batch, Server
    thin = G.gate_array([(G.H, q) for q in range(4)] + [(G.X, 4 + i, (i % 4,)) for i in range(20)] + [(G.X, 7), (G.Y, 2)])
    dense = G.gate_array([(G.H, q) for q in range(9)])
    b, sv = Batch(precision=precision), Server(precision=precision, memory_budget=4 << 30)
    b.prepare([(40, thin), (40, dense)])
    b.run()
    b.sync()
    ids = [sv.submit(40, g) for g in (thin, dense)]
    while any(sv.status(r)[0] != 2 for r in ids):
        sv.step()
    for i, (g, launches) in enumerate(((thin, 1), (dense, 3))):
        o = SparseOracle(precision)
        o.apply(g)
        want = o.state(sorted=True)
        for read, stats in ((lambda **k: b.state(i, **k), b.stats), (lambda **k: sv.state(ids[i], **k), sv.stats)):
            before = stats()["kernel_launches"]
            assert_identical(read(sorted=True), want)
            assert stats()["kernel_launches"] == before + launches
            got = read(sorted=False)
            order = np.argsort(got[0])
            assert_identical(tuple(x[order] for x in got), want)
    b.prepare([(40, thin)])   # the only circuit of a batch, by the call that reads all
    b.run()
    b.sync()
    before = b.stats()["kernel_launches"]
    o = SparseOracle(precision)
    o.apply(thin)
    assert_identical(b.states(sorted=True)[0], o.state(sorted=True))
    assert b.stats()["kernel_launches"] == before + 1
    b.close()
    sv.close()
