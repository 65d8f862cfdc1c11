"""What this framework's users run, as measurable cases.

A sparse-statevector user starts a register in |0...0> (or loads a state), applies circuits and
reads the state, its probabilities or samples back; with many circuits they go to a batch or to
the serving loop. The sizes are those of the repository's own configurations
(sparqc_gb300/circuits.py: 20 to 64 qubits, 10 to 26 branching qubits, 200 to 2000 gates, batches
of mixed circuits, a served stream with some large circuits) and of its tests.

Most circuits follow the configurations' rules: H on qubits 0..k-1, then 30% diagonal, 30%
permutation and 40% branching gates with 0 to 3 controls; such a state fills the 2**k keys its
first k qubits span. The "logic" circuits are the other kind of sparse state: reversible logic on
superposed inputs, whose keys spread thinly over many qubits.
"""
import ctypes
import math

import numpy as np
import torch

from sparqc_gb300 import engine
from sparqc_gb300 import gates as G

DIAG = np.array([G.Z, G.S, G.T, G.RZ, G.PHASE], np.uint32)
PERM = np.array([G.X, G.Y], np.uint32)
BRANCH = np.array([G.H, G.RX, G.RY, G.U], np.uint32)
PRUNE = 1e-14


def listed():
    return [
        # a small register run and read back, as in an interactive session: latency
        dict(name="small_fp64", kind="circuit", nq=20, k=10, depth=200, controls=2, precision=64, schedule=False,
             pinned=False),
        # the Fourier transform written gate by gate through the Circuit methods
        dict(name="qft_calls", kind="qft", nq=14),
        # the 40-qubit configuration: a mid-size state, long circuit, bit-exact FP64 order
        dict(name="mid_fp64", kind="circuit", nq=40, k=20, depth=2000, controls=3, precision=64, schedule=False,
             pinned=True),
        # the same in single precision with the gates in scheduled order (odd size)
        dict(name="mid_fp32", kind="circuit", nq=41, k=19, depth=1501, controls=3, precision=32, schedule=True,
             pinned=True),
        # the 64-qubit configuration at half its largest state: the heavy FP64 run
        dict(name="large_fp64", kind="circuit", nq=64, k=25, depth=500, controls=3, precision=64, schedule=False,
             pinned=True),
        # the large circuit of the serving configuration, run alone in FP32
        dict(name="large_fp32", kind="circuit", nq=48, k=24, depth=2000, controls=3, precision=32, schedule=True,
             pinned=True),
        # reversible logic on 2**17 superposed inputs over 60 qubits: keys spread thinly
        dict(name="logic_fp64", kind="logic", nq=60, k=17, depth=300, precision=64),
        # a state held on the host (a million keys), continued on the GPU and read back
        dict(name="load_fp64", kind="load", nq=36, keys=1000003, depth=60, precision=64),
        # the batching configuration in FP32, prepared once and run again; every state read back
        dict(name="batch_fp32", kind="batch", count=128, kmin=8, kmax=18, precision=32, schedule=True, fresh=False),
        # new circuits every time: plan, upload, run, read (FP64)
        dict(name="batch_new_fp64", kind="batch", count=24, kmin=8, kmax=14, precision=64, schedule=False, fresh=True),
        # the serving loop: a burst of requests with a large one among them
        dict(name="serve_fp32", kind="serve", count=20, large=1, large_k=22, large_depth=1000, precision=32),
        # questions put to a finished state: norm, probabilities, a selected readout, samples
        dict(name="analysis_fp64", kind="analysis", nq=40, k=20, depth=200, precision=64, shots=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["circuit", "circuit", "circuit", "qft", "logic", "load", "batch", "serve", "analysis"])
    precision = rng.choice([64, 32])
    if kind == "circuit":
        k = rng.randint(6, 24)
        depth = _log_int(rng, 60, 500 if k > 22 else 2000)
        return dict(kind=kind, nq=rng.randint(max(k, 12), 64), k=k, depth=depth, controls=rng.randint(0, 3),
                    precision=precision, schedule=rng.random() < 0.4, pinned=k > 16)
    if kind == "qft":
        return dict(kind=kind, nq=rng.randint(6, 18))
    if kind == "logic":
        return dict(kind=kind, nq=rng.randint(30, 64), k=rng.randint(8, 17), depth=_log_int(rng, 50, 400),
                    precision=precision)
    if kind == "load":
        return dict(kind=kind, nq=rng.randint(24, 64), keys=_log_int(rng, 300, 1000000), depth=rng.randint(10, 80),
                    precision=precision)
    if kind == "batch":
        kmin = rng.randint(5, 10)
        return dict(kind=kind, count=_log_int(rng, 2, 64), kmin=kmin, kmax=kmin + rng.randint(0, 7),
                    precision=precision, schedule=rng.random() < 0.5, fresh=rng.random() < 0.5)
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(3, 20), large=rng.randint(0, 1), large_k=rng.randint(20, 22),
                    large_depth=rng.randint(200, 1000), precision=precision)
    return dict(kind=kind, nq=rng.randint(24, 64), k=rng.randint(8, 20), depth=_log_int(rng, 60, 400),
                precision=precision, shots=_log_int(rng, 100, 10000))


# ---- circuits -------------------------------------------------------------------------------


def _controls(rng, counts, allowed):
    """Per gate, `counts` distinct qubits drawn from its allowed ones, as a mask."""
    depth, nq = allowed.shape
    order = np.where(allowed, rng.random((depth, nq)), 2.0)
    rank = order.argsort(axis=1)
    mask = np.zeros(depth, np.uint64)
    for j in range(int(counts.max(initial=0))):
        q = rank[:, j]
        take = (j < counts) & allowed[np.arange(depth), q]
        mask |= np.where(take, np.uint64(1) << q.astype(np.uint64), np.uint64(0))
    return mask


def _mixed(nq, k, depth, controls, rng, prefix=True):
    """A circuit by the configurations' rules (see sparqc_gb300/circuits.py)."""
    u = rng.random(depth)
    diag, perm = u < 0.3, (u >= 0.3) & (u < 0.6)
    kind = np.where(diag, DIAG[rng.integers(0, 5, depth)],
                    np.where(perm, PERM[rng.integers(0, 2, depth)], BRANCH[rng.integers(0, 4, depth)]))
    target = np.where(diag | perm, rng.integers(0, nq, depth), rng.integers(0, k, depth))
    n = min(k, depth) if prefix else 0
    kind[:n], target[:n], perm[:n], diag[:n] = G.H, np.arange(n), False, False
    q = np.arange(nq)[None, :]
    allowed = (q != target[:, None]) & ~((perm & (target >= k))[:, None] & (q < k))
    counts = rng.integers(0, controls + 1, depth)
    counts[:n] = 0
    return _gates(kind, target, _controls(rng, counts, allowed), rng)


def _gates(kind, target, controls, rng):
    g = np.zeros(len(kind), G.GATE_DTYPE)
    g["kind"], g["target"], g["controls"] = kind, target, controls
    angles = rng.random((3, len(kind))) * (2.0 * math.pi)
    turned = np.isin(kind, [G.RZ, G.RX, G.RY, G.PHASE, G.U])
    g["theta"] = np.where(turned, angles[0], 0.0)
    g["phi"] = np.where(kind == G.U, angles[1], 0.0)
    g["lambda"] = np.where(kind == G.U, angles[2], 0.0)
    return g


def _logic(nq, k, depth, rng):
    """H on the k input qubits, then X, CX and Toffoli gates onto all the others with phases
    between them, and a rotation of an input qubit now and then."""
    u = rng.random(depth)
    flip, phase = u < 0.75, (u >= 0.75) & (u < 0.97)
    kind = np.where(flip, np.uint32(G.X), np.where(phase, DIAG[rng.integers(0, 5, depth)], np.uint32(G.H)))
    target = np.where(flip, rng.integers(k, nq, depth), np.where(phase, rng.integers(0, nq, depth), 0))
    counts = np.where(flip, rng.integers(1, 3, depth), np.where(phase, rng.integers(0, 3, depth), 0))
    turns = np.flatnonzero(~flip & ~phase)
    kind[turns[1:]] = G.Z   # one branching gate at most: it may double the keys
    target[turns] = rng.integers(0, k, len(turns))
    kind[:k], target[:k], counts[:k] = G.H, np.arange(k), 0
    allowed = np.arange(nq)[None, :] != target[:, None]
    return _gates(kind, target, _controls(rng, counts, allowed), rng)


def _loaded(nq, keys, depth, rng):
    """A random sparse state in key order, and gates that keep it about as large."""
    step = (1 << min(nq, 62)) // keys
    k = np.arange(keys, dtype=np.uint64) * np.uint64(step) + rng.integers(0, step, keys, dtype=np.uint64)
    a = rng.standard_normal((2, keys))
    a /= math.sqrt(float(np.sum(a * a)))
    u = rng.random(depth)
    kind = np.where(u < 0.45, DIAG[rng.integers(0, 5, depth)], np.where(u < 0.95, PERM[rng.integers(0, 2, depth)],
                                                                       np.uint32(G.RY)))
    few = np.flatnonzero(u >= 0.95)
    kind[few[1:]] = G.S   # one branching gate at most
    target = rng.integers(0, nq, depth)
    target[few] = rng.integers(0, 4, len(few))
    allowed = np.arange(nq)[None, :] != target[:, None]
    return k, a[0].copy(), a[1].copy(), _gates(kind, target, _controls(rng, rng.integers(0, 3, depth), allowed), rng)


def _batch_circuits(case, rng):
    """The sizes are the case's, spread over their ranges; the gates follow the seed."""
    out, sizes = [], np.random.default_rng(case["count"] * 100 + case["kmax"])
    for _ in range(case["count"]):
        nq = int(sizes.integers(16, 49))
        k = min(int(sizes.integers(case["kmin"], case["kmax"] + 1)), nq)
        out.append((nq, k, _mixed(nq, k, int(sizes.integers(100, 1001)), 3, rng)))
    return out


def _served_circuits(case, rng):
    out = [(nq, k, g) for nq, k, g in _batch_circuits(dict(count=case["count"] - case["large"], kmin=8, kmax=16), rng)]
    for _ in range(case["large"]):
        k = case["large_k"]
        out.insert(len(out) // 2, (48, k, _mixed(48, k, case["large_depth"], 3, rng)))
    return out


def _qft(nq, rng):
    """(basis state, gate list) of a Fourier transform: H and controlled phases."""
    start = int(rng.integers(1, 1 << nq))
    calls = [(G.X, q, 0, 0.0) for q in range(nq) if (start >> q) & 1]
    for t in reversed(range(nq)):
        calls.append((G.H, t, 0, 0.0))
        calls += [(G.PHASE, t, 1 << c, math.pi / (1 << (t - c))) for c in range(t)]
    return calls


# ---- the cases ------------------------------------------------------------------------------


def _arrays(n, pinned=False):
    """A caller's own arrays for n entries (keys, re, im), page-locked or not."""
    types = (torch.int64, torch.float64, torch.float64)
    return tuple(torch.zeros(n, dtype=t, pin_memory=pinned).numpy() for t in types)


def _into(call, handle, *args, out, flags=engine.READ_SORTED):
    """A readout of the C interface into the caller's arrays: their entry count, and the arrays."""
    n = ctypes.c_uint64()
    p = [a.ctypes.data_as(ctypes.c_void_p) for a in out]
    rc = getattr(engine.load(), call)(handle, *args, p[0], p[1], p[2], out[0].size, ctypes.byref(n), flags)
    if rc != engine.OK:
        raise RuntimeError("%s: status %d" % (call, rc))
    return (n.value,) + out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "circuit":
        s["gates"] = _mixed(case["nq"], case["k"], case["depth"], case["controls"], rng)
        s["state"] = engine.State(case["nq"], precision=case["precision"], schedule_gates=case["schedule"])
        s["out"] = _arrays(1 << case["k"], pinned=case["pinned"])
    elif kind == "qft":
        s["calls"] = _qft(case["nq"], rng)
        s["state"] = engine.Circuit(case["nq"])
    elif kind == "logic":
        s["gates"] = _logic(case["nq"], case["k"], case["depth"], rng)
        s["state"] = engine.State(case["nq"], precision=case["precision"])
        s["out"] = _arrays(2 << case["k"])
    elif kind == "load":
        s["loaded"] = _loaded(case["nq"], case["keys"], case["depth"], rng)
        s["state"] = engine.State(case["nq"], precision=case["precision"])
        s["out"] = _arrays(2 * case["keys"], pinned=True)
    elif kind == "batch":
        cs = _batch_circuits(case, rng)
        s["circuits"] = [(nq, g) for nq, _, g in cs]
        s["out"] = _arrays(sum(1 << k for _, k, _ in cs), pinned=True)
        s["batch"] = engine.Batch(precision=case["precision"], schedule_gates=case["schedule"])
        if not case["fresh"]:
            s["batch"].prepare(s["circuits"])
    elif kind == "serve":
        cs = _served_circuits(case, rng)
        s["circuits"] = [(nq, g) for nq, _, g in cs]
        s["outs"] = [_arrays(1 << k, pinned=True) for _, k, _ in cs]
        s["server"] = engine.Server(precision=case["precision"], memory_budget=16 << 30, slice_ms=1.0,
                                    schedule_gates=True, overlap_steps=True)
    else:
        g = _mixed(case["nq"], case["k"], case["depth"], 3, rng)
        s["state"] = engine.State(case["nq"], precision=case["precision"])
        s["state"].apply(g)
        s["state"].sync()
        s["out"] = _arrays(1 << (case["k"] - 3))
    return s


def _patterns(case):
    """(mask, value) patterns on the branching qubits."""
    low, high = 1, 1 << (case["k"] - 1)
    return [(low, low), (high, 0), (low | high, high), (0b1110, 0b0110)]


def run(s):
    kind = s["case"]["kind"]
    if kind == "circuit" or kind == "logic":
        st = s["state"]
        st.set_zero()
        st.apply(s["gates"])
        return _into("sqc_get_state", st.handle, out=s["out"])
    if kind == "qft":
        c = s["state"]
        c.set_zero()
        for g, t, controls, angle in s["calls"]:
            if g == G.X:
                c.x(t)
            elif g == G.H:
                c.h(t)
            else:
                c.controlled(g, t, [q for q in range(t) if (controls >> q) & 1], angle)
        return c.state()
    if kind == "load":
        st = s["state"]
        k, r, i, g = s["loaded"]
        st.set_state(k, r, i)
        st.apply(g)
        return _into("sqc_get_state", st.handle, out=s["out"])
    if kind == "batch":
        b = s["batch"]
        if s["case"]["fresh"]:
            b.prepare(s["circuits"])
        b.run()
        b.sync()
        keys, re, im = s["out"]
        counts = [x[0].size for x in b.states(sorted=True, out=(keys.view(np.uint64), re, im))]
        return np.array(counts), keys, re, im
    if kind == "serve":
        sv = s["server"]
        ids = [sv.submit(nq, g) for nq, g in s["circuits"]]
        out, got = dict(zip(ids, s["outs"])), {}
        while len(got) < len(ids):
            sv.step()
            for rid in sv.completed():
                got[rid] = _into("sqc_server_get_state", sv._h, rid, out=out[rid])[1:]
                sv.release(rid)
        return [got[rid] for rid in ids]
    st = s["state"]
    pats = _patterns(s["case"])
    return {"norm": st.norm2(), "probability": [st.probability(m, v) for m, v in pats],
            "selected": _into("sqc_get_state_where", st.handle, *pats[3], out=s["out"]),
            "samples": st.sample(s["case"]["shots"], seed=11).view(np.int64)}


# ---- what a pass cannot do without ----------------------------------------------------------

# multiplications and additions per amplitude held, by kind (one-sided kinds act on half of them)
_FLOPS = {G.H: 4, G.RX: 6, G.RY: 6, G.U: 14, G.RZ: 6, G.PHASE: 3, G.T: 3}


def _circuit_work(k, depth):
    mean = 0.4 * (4 + 6 + 6 + 14) / 4 + 0.3 * (6 + 3 + 3) / 5
    return {"bytes": 40.0 * depth + 24.0 * 2 ** k, "flops": mean * max(depth - k, 1) * 2.0 ** k}


def _sum(works):
    works = list(works)
    return {"bytes": sum(w["bytes"] for w in works), "flops": sum(w["flops"] for w in works)}


def work(case):
    kind = case["kind"]
    if kind == "circuit":
        return _circuit_work(case["k"], case["depth"])
    if kind == "qft":
        n = case["nq"]
        return {"bytes": 40.0 * n * (n + 1) / 2 + 24.0 * 2 ** n, "flops": (4 * n + 3 * n * (n - 1) / 2) * 2.0 ** n / 2}
    if kind == "logic":
        n = 2.0 ** (case["k"] + 1)
        return {"bytes": 40.0 * case["depth"] + 24.0 * n, "flops": 0.22 * 12 / 5 * case["depth"] * n}
    if kind == "load":
        return {"bytes": 48.0 * case["keys"] + 40.0 * case["depth"], "flops": 0.45 * 12 / 5 * case["depth"] * case["keys"]}
    if kind == "batch":
        ks = range(case["kmin"], case["kmax"] + 1)
        w = _sum(_circuit_work(k, 550) for k in ks)
        return {m: v * case["count"] / len(ks) for m, v in w.items()}
    if kind == "serve":
        w = _sum(_circuit_work(k, 550) for k in range(8, 17))
        w = {m: v * (case["count"] - case["large"]) / 9 for m, v in w.items()}
        return _sum([w] + [_circuit_work(case["large_k"], case["large_depth"])] * case["large"])
    n, amp = 2.0 ** case["k"], 16.0 if case["precision"] == 64 else 8.0
    return {"bytes": n * (8 + amp) + 24.0 * n / 8 + 8.0 * case["shots"], "flops": 4.0 * n}


# ---- the same in 64 bits, in plain torch and numpy --------------------------------------------


def _matrix(g):
    """(2x2 matrix) of a gate record, as four complex numbers m00, m01, m10, m11."""
    kind, th, ph, lm = int(g["kind"]), float(g["theta"]), float(g["phi"]), float(g["lambda"])
    c, s = math.cos(th / 2), math.sin(th / 2)
    e = lambda x: complex(math.cos(x), math.sin(x))  # noqa: E731
    r = math.sqrt(0.5)
    return {G.X: (0, 1, 1, 0), G.Y: (0, -1j, 1j, 0), G.Z: (1, 0, 0, -1), G.H: (r, r, r, -r), G.PHASE: (1, 0, 0, e(th)),
            G.RZ: (e(-th / 2), 0, 0, e(th / 2)), G.RX: (c, -1j * s, -1j * s, c), G.RY: (c, -s, s, c), G.S: (1, 0, 0, 1j),
            G.T: (1, 0, 0, complex(r, r)), G.U: (c, -e(lm) * s, e(ph) * s, e(ph + lm) * c)}[kind]


def _dense(nq, k, gates):
    """The final state of a circuit whose bits >= k are the same in every key: a dense vector over
    the first k qubits, the other bits classical."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v = torch.zeros(1 << k, dtype=torch.complex128, device=dev)
    v[0] = 1
    high = 0
    for g in gates:
        t, ctrl = int(g["target"]), int(g["controls"])
        if (ctrl >> k) & ~(high >> k):
            continue
        m = _matrix(g)
        low = [q for q in range(k) if (ctrl >> q) & 1]
        split = sorted(low + ([t] if t < k else []), reverse=True)
        shape, at, prev = [], [], k
        for q in split:
            shape += [1 << (prev - q - 1), 2]
            at += [slice(None), 1 if q in low else slice(None)]
            prev = q
        shape.append(1 << prev)
        sub = v.view(shape)[tuple(at) + (slice(None),)]
        if t >= k:
            bit = (high >> t) & 1
            if m[1] == 0:
                sub *= m[3] if bit else m[0]
            else:
                sub *= m[1] if bit else m[2]
                high ^= 1 << t
            continue
        axis = 1 + 2 * split.index(t) - sum(1 for q in split[:split.index(t)] if q in low)
        a, b = sub.select(axis, 0), sub.select(axis, 1)
        if m[1] == 0:
            if m[0] != 1:
                a *= m[0]
            b *= m[3]
        else:
            na = a * m[0] + b * m[1]
            b.copy_(a * m[2] + b * m[3])
            a.copy_(na)
    v = torch.view_as_real(v)
    keep = (v.abs() >= PRUNE).any(dim=1)
    v = v[keep].cpu().numpy()
    return np.ascontiguousarray(v[:, 0]), np.ascontiguousarray(v[:, 1]), keep


def _sparse(keys, amp, gates):
    """Gates on a sorted sparse state (uint64 keys, complex128 amplitudes)."""
    for g in gates:
        t, ctrl = np.uint64(1) << np.uint64(g["target"]), np.uint64(g["controls"])
        m = _matrix(g)
        on = (keys & ctrl) == ctrl
        if m[1] == 0:
            amp = np.where(on, amp * np.where((keys & t) != 0, m[3], m[0]), amp)
        elif m[0] == 0:
            amp = np.where(on, amp * np.where((keys & t) != 0, m[1], m[2]), amp)
            keys = np.where(on, keys ^ t, keys)
        else:
            base, at = np.unique(keys[on] & ~t, return_inverse=True)
            two = np.zeros((2, base.size), np.complex128)
            two[((keys[on] & t) != 0).astype(np.int64), at] = amp[on]
            new = np.concatenate([m[0] * two[0] + m[1] * two[1], m[2] * two[0] + m[3] * two[1]])
            nk = np.concatenate([base, base | t])
            live = (np.abs(new.real) >= PRUNE) | (np.abs(new.imag) >= PRUNE)
            keys, amp = np.concatenate([keys[~on], nk[live]]), np.concatenate([amp[~on], new[live]])
    order = np.argsort(keys)
    return np.ascontiguousarray(amp.real[order]), np.ascontiguousarray(amp.imag[order])


def _pad(n, *arrays):
    return tuple(np.concatenate([a, np.zeros(n - a.size)]) for a in arrays)


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "circuit":
        g = _mixed(case["nq"], case["k"], case["depth"], case["controls"], rng)
        return (None, None) + _pad(1 << case["k"], *_dense(case["nq"], case["k"], g)[:2])
    if kind == "qft":
        g = G.gate_array([(a, t, c, th) for a, t, c, th in _qft(case["nq"], rng)])
        return (None,) + _dense(case["nq"], case["nq"], g)[:2]
    if kind == "logic":
        g = _logic(case["nq"], case["k"], case["depth"], rng)
        return (None, None) + _pad(2 << case["k"], *_sparse(np.zeros(1, np.uint64), np.ones(1, np.complex128), g))
    if kind == "load":
        k, r, i, g = _loaded(case["nq"], case["keys"], case["depth"], rng)
        return (None, None) + _pad(2 * case["keys"], *_sparse(k, r + 1j * i, g))
    if kind == "batch":
        cs = _batch_circuits(case, rng)
        got = [_dense(nq, k, g)[:2] for nq, k, g in cs]
        n = sum(1 << k for _, k, _ in cs)
        return (None, None) + _pad(n, *[np.concatenate([x[j] for x in got]) for j in range(2)])
    if kind == "serve":
        return [(None,) + _pad(1 << k, *_dense(nq, k, g)[:2]) for nq, k, g in _served_circuits(case, rng)]
    re, im, keep = _dense(case["nq"], case["k"], _mixed(case["nq"], case["k"], case["depth"], 3, rng))
    key = torch.nonzero(keep).flatten().cpu().numpy().astype(np.int64)
    p = re * re + im * im
    pats = _patterns(case)
    mask, value = pats[3]
    sel = (key & mask) == value
    return {"norm": float(p.sum()), "probability": [float(p[(key & m) == v].sum()) for m, v in pats],
            "selected": (None, None) + _pad(1 << (case["k"] - 3), re[sel], im[sel]), "samples": None}
