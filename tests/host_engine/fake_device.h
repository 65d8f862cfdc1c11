// A device on the host for tests of the engine's host code (sqc_engine.cpp, sqc_plan.cpp): the CUDA
// runtime calls and kernel launchers they use, over ordinary memory. Work happens at the call, in
// order; device memory is checked (a copy or a kernel write outside an allocation is counted in
// dev.bad), allocations may be made to fail, and a state is kept as a map from stored key to
// amplitude under its control block. Passes follow the descriptors as the kernels do, with the same
// refusals; the list of live buckets is kept as the set of groups that were ever claimed.
#pragma once
#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <vector>

#include "sqc_engine.h"
#include "sqc_kernels.h"

namespace fake {

using Amp = std::complex<double>;

struct State {
    std::map<unsigned long long, Amp> amp;
    std::set<unsigned long long> live;   // groups with a bucket
};

struct Device {
    std::map<unsigned char*, size_t> mem;        // device allocations
    std::map<const void*, State> state;          // by control block
    size_t held = 0, peak = 0;                   // bytes allocated
    size_t total = (size_t)284 << 30;            // bytes of the device
    size_t big_limit = 0;                        // allocations of at least this many bytes fail (0: none)
    int fail_big = 0;                            // ... while this is positive
    int fail_copies = 0;                         // copies to the device that fail
    long bad = 0;                                // accesses outside an allocation, misuse of events
    cudaError_t last = cudaSuccess;              // what cudaGetLastError answers, once
    long syncs = 0, passes = 0, runs = 0;
    unsigned long long items = 0;                // most items a run was launched for
    bool capturing = false;
    std::vector<long> events;                    // time of each event's last record, 0: never
    long now = 0;
    bool inside(const void* p, size_t n) const {
        auto it = mem.upper_bound((unsigned char*)p);
        if (it == mem.begin()) return false;
        --it;
        return (unsigned char*)p + n <= it->first + it->second;
    }
};
inline Device dev;
inline int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); ++fake::fails; } } while (0)

// Large tables are not backed by memory: nothing here reads them (the amplitudes are in State).
constexpr size_t kBacked = (size_t)1 << 26;

inline void apply_desc(State& st, const sqc::GateDesc& g, double thr) {
    using namespace sqc;
    const Amp i1(0, 1);
    Amp m[4] = {1, 0, 0, 1};
    const Amp e(g.c, g.s);
    switch (g.kind) {
    case KX: m[0] = m[3] = 0; m[1] = m[2] = 1; break;
    case KY: m[0] = m[3] = 0; m[1] = -i1; m[2] = i1; break;
    case KZ: m[3] = -1; break;
    case KH: m[0] = m[1] = m[2] = g.c; m[3] = -g.c; break;
    case KS: m[3] = i1; break;
    case KSDG: m[3] = -i1; break;
    case KYPH: m[0] = -i1; m[3] = i1; break;
    case KRZ: m[0] = std::conj(e); m[3] = e; break;
    case KPHASE: case KT: case KTDG: m[3] = e; break;
    case KRX: m[0] = m[3] = g.c; m[1] = m[2] = -i1 * g.s; break;
    case KRY: m[0] = m[3] = g.c; m[1] = -g.s; m[2] = g.s; break;
    default: for (int k = 0; k < 4; ++k) m[k] = Amp(g.m[2 * k], g.m[2 * k + 1]);
    }
    const unsigned long long bit = 1ULL << g.target;
    std::set<unsigned long long> base;
    for (auto& kv : st.amp)
        if ((kv.first & g.ctrl) == g.cval) base.insert(kv.first & ~bit);
    for (unsigned long long b : base) {
        const unsigned long long k0 = (g.flip & kOpFlip) ? b | bit : b, k1 = k0 ^ bit;
        auto p0 = st.amp.find(k0), p1 = st.amp.find(k1);
        const bool h0 = p0 != st.amp.end(), h1 = p1 != st.amp.end();
        const Amp v0 = h0 ? p0->second : 0.0, v1 = h1 ? p1->second : 0.0;
        const Amp o0 = m[0] * v0 + m[1] * v1, o1 = m[2] * v0 + m[3] * v1;
        bool n0 = h0, n1 = h1;
        if (is_swap_kind(g.kind)) { n0 = h1; n1 = h0; }
        if (is_branch_kind(g.kind)) {
            n0 = !(std::fabs(o0.real()) < thr && std::fabs(o0.imag()) < thr);
            n1 = !(std::fabs(o1.real()) < thr && std::fabs(o1.imag()) < thr);
        }
        auto put = [&](unsigned long long k, bool on, Amp v) {
            if (!on) { st.amp.erase(k); return; }
            st.amp[k] = v;
            st.live.insert(k >> kSlotBits);
        };
        put(k0, n0, o0);
        put(k1, n1, o1);
    }
}

inline double threshold(const sqc::PruneBits& p) { double t; std::memcpy(&t, &p.d, 8); return t; }

inline void publish(sqc::Ctl* ctl, State& st) {
    ctl->nnz = st.amp.size();
    ctl->list_n = ctl->list_tail = st.live.size();
    std::set<unsigned long long> used;
    for (auto& kv : st.amp) used.insert(kv.first >> sqc::kSlotBits);
    ctl->empty_groups = st.live.size() - used.size();
    ctl->seq += 1;
    ++dev.passes;
}

inline bool pass(sqc::Ctl* ctl, const sqc::GateDesc* gates, uint32_t g0, uint32_t g1, const sqc::PruneBits& pb, bool refuse) {
    if (ctl->status) return false;
    if (refuse) { ctl->status = sqc::ST_GROW; return false; }
    State& st = dev.state[ctl];
    for (uint32_t i = g0; i < g1; ++i) {
        ctl->amp_updates += st.amp.size() * (gates[i].pad + 1ULL);
        apply_desc(st, gates[i], threshold(pb));
    }
    publish(ctl, st);
    return true;
}

inline bool overflow(unsigned long long n, uint32_t nx, unsigned long long bound, unsigned long long keys, unsigned long long max) {
    return nx > 0 && std::min(std::min(bound, n << nx), n + keys) > max;
}

// The same gates on actual keys, without the engine: what the state must be.
inline std::map<unsigned long long, Amp> expected(const std::vector<sqc_gate>& gs, std::map<unsigned long long, Amp> amp = {{0, 1.0}}) {
    State st;
    st.amp = std::move(amp);
    for (const sqc_gate& g : gs) {
        sqc::Planner p;
        p.kmask = 0;
        apply_desc(st, sqc::make_desc(p, g.kind, g.target, g.controls, g), 1e-14);
    }
    return st.amp;
}

inline sqc_gate gate(uint32_t kind, uint32_t t, uint64_t ctrl = 0, double th = 0.3) {
    sqc_gate x;
    std::memset(&x, 0, sizeof x);
    x.kind = kind;
    x.target = t;
    x.controls = ctrl;
    x.theta = th;
    return x;
}

// The engine's answers about its state against `want`.
inline bool holds(sqc::Engine& e, const std::map<unsigned long long, Amp>& want) {
    uint64_t n = 0;
    if (e.nnz(&n) != SQC_OK || n != want.size()) { std::printf("nnz %llu, not %zu: %s\n", (unsigned long long)n, want.size(), e.err.c_str()); return false; }
    std::vector<uint64_t> k(n + 1);
    std::vector<double> r(n + 1), i(n + 1);
    uint64_t got = 0;
    if (e.get_state(k.data(), r.data(), i.data(), n, &got, SQC_READ_SORTED) != SQC_OK || got != n) { std::printf("readout: %s\n", e.err.c_str()); return false; }
    size_t at = 0;
    for (auto& kv : want) {
        if (k[at] != kv.first || std::abs(Amp(r[at], i[at]) - kv.second) > 1e-9) { std::printf("entry %zu differs\n", at); return false; }
        ++at;
    }
    return true;
}

inline void make(sqc::Engine& e, uint32_t nq, const sqc_options* o = nullptr) {
    if (e.init(nq, nullptr, o) != SQC_OK) { std::printf("init: %s\n", e.err.c_str()); std::exit(2); }
}

}  // namespace fake

extern "C" {
void sqc_default_options(sqc_options* o) {
    std::memset(o, 0, sizeof *o);
    o->precision = SQC_FP64;
    o->prune_threshold = 1e-14;
    o->load_factor = 0.5;
}

// ---- runtime ----
cudaError_t cudaMalloc(void** p, size_t n) {
    using namespace fake;
    *p = nullptr;
    if (dev.held + n > dev.total) return dev.last = cudaErrorMemoryAllocation;
    if (dev.big_limit && n >= dev.big_limit && dev.fail_big > 0) { --dev.fail_big; return dev.last = cudaErrorMemoryAllocation; }
    // a range that is not backed is only an address
    static unsigned char* next = reinterpret_cast<unsigned char*>(1ULL << 60);
    unsigned char* q = n <= kBacked ? (unsigned char*)std::calloc(1, n) : next;
    if (n > kBacked) next += (n + 4095) & ~(size_t)4095;
    dev.mem[q] = n;
    dev.held += n;
    dev.peak = std::max(dev.peak, dev.held);
    *p = q;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    using namespace fake;
    if (!p) return cudaSuccess;
    auto it = dev.mem.find((unsigned char*)p);
    if (it == dev.mem.end()) { ++dev.bad; return cudaErrorInvalidValue; }
    dev.held -= it->second;
    if (it->second <= kBacked) std::free(p);
    dev.mem.erase(it);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (!fake::dev.inside(p, n)) { ++fake::dev.bad; return cudaSuccess; }
    if ((size_t)p < (1ULL << 60)) std::memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (k == cudaMemcpyHostToDevice && fake::dev.fail_copies > 0) { --fake::dev.fail_copies; return cudaErrorUnknown; }
    if (!fake::dev.inside(k == cudaMemcpyHostToDevice ? d : s, n)) { ++fake::dev.bad; return cudaSuccess; }
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    ++fake::dev.syncs;
    return fake::dev.capturing ? cudaErrorStreamCaptureUnsupported : cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = fake::dev.capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    fake::dev.events.push_back(0);
    *e = reinterpret_cast<cudaEvent_t>(fake::dev.events.size());
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { fake::dev.events[(size_t)e - 1] = ++fake::dev.now; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t a, cudaEvent_t b) {
    const long x = fake::dev.events[(size_t)a - 1], y = fake::dev.events[(size_t)b - 1];
    if (!x || !y || x >= y) ++fake::dev.bad;   // a pass ends after it begins
    *ms = (float)(y - x);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::dev.last;
    fake::dev.last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = fake::dev.total - fake::dev.held; *t = fake::dev.total; return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { a->type = cudaMemoryTypeHost; return cudaSuccess; }
}

// ---- launchers (as theirs do, they answer with the last error) ----
namespace sqc {
using namespace fake;

cudaError_t launch_set_zero(const TableDev&, Ctl* ctl, bool, cudaStream_t) {
    const unsigned ep = ctl->epoch + 1;
    std::memset(ctl, 0, sizeof *ctl);
    ctl->epoch = ep;
    State& st = fake::dev.state[ctl];
    st.amp = {{0, 1.0}};
    st.live = {0};
    ctl->nnz = ctl->list_n = ctl->list_tail = 1;
    return cudaGetLastError();
}
cudaError_t launch_set_state(const unsigned long long* keys, const double* re, const double* im, unsigned long long n,
                             unsigned long long frame, const TableDev&, Ctl* ctl, bool, int, cudaStream_t) {
    launch_set_zero(TableDev(), ctl, true, nullptr);
    State& st = fake::dev.state[ctl];
    st.amp.clear();
    st.live.clear();
    for (unsigned long long i = 0; i < n; ++i) {
        st.amp[keys[i] ^ frame] = Amp(re[i], im[i]);
        st.live.insert((keys[i] ^ frame) >> kSlotBits);
    }
    ctl->nnz = n;
    ctl->list_n = ctl->list_tail = st.live.size();
    return cudaGetLastError();
}
int launch_unit_pass(const PassArgs& a, bool, int, cudaStream_t) {
    fake::pass(a.ctl, a.gates, a.g0, a.g1, a.prune, (1ULL << a.dn) > a.max_groups);
    return 1;
}
int launch_hash_pass(const PassArgs& a, unsigned long long, bool, int, cudaStream_t) {
    fake::pass(a.ctl, a.gates, a.g0, a.g1, a.prune, overflow(a.ctl->list_n, a.nx, a.grow_bound, a.key_bound, a.max_groups));
    return 1;
}
int launch_run_passes(const RunArgs& a, uint32_t, unsigned long long items, bool, int, cudaStream_t) {
    ++fake::dev.runs;
    fake::dev.items = std::max(fake::dev.items, items);
    uint32_t o = 0;
    for (uint32_t p = 0; p < a.np; ++p) {
        const UnitHead r = a.words[o];
        const uint32_t ng = r.om & 0xFFu;
        bool refuse = false;
        if (!a.t.map_on) {
            unsigned long long b[2];
            std::memcpy(b, &a.words[o + 1], sizeof b);
            refuse = overflow(a.ctl->list_n, r.om >> 16, b[0], b[1], a.max_groups);
        }
        if (!fake::pass(a.ctl, a.gates, r.loc, r.loc + ng, a.prune, refuse)) break;
        o += a.t.map_on ? 1 + ng : 2;
    }
    return 1;
}
cudaError_t launch_refresh_masks(const TableDev&, Ctl*, unsigned long long, int, cudaStream_t) { return cudaGetLastError(); }
static void emit(const TableDev&, Ctl* ctl, unsigned long long frame, unsigned long long* ok, double* re, double* im,
                 unsigned long long cap, unsigned long long smask, unsigned long long sval) {
    std::vector<std::pair<unsigned long long, Amp>> out;
    for (auto& kv : fake::dev.state[ctl].amp)
        if ((kv.first & smask) == sval) out.push_back({kv.first ^ frame, kv.second});
    std::sort(out.begin(), out.end(), [](auto& x, auto& y) { return x.first < y.first; });
    ctl->out_count = out.size();
    for (size_t i = 0; i < out.size() && i < cap; ++i) {
        ok[i] = out[i].first;
        re[i] = out[i].second.real();
        im[i] = out[i].second.imag();
    }
}
cudaError_t launch_readout(const TableDev& t, Ctl* ctl, unsigned long long, unsigned long long frame, bool,
                           unsigned long long* ok, double* re, double* im, unsigned long long cap, bool, PruneBits, int,
                           cudaStream_t, unsigned long long smask, unsigned long long sval) {
    emit(t, ctl, frame, ok, re, im, cap, smask, sval);
    return cudaGetLastError();
}
RankJob rank_job(const TableDev& t, const Ctl* ctl, unsigned long long frame, unsigned long long, unsigned long long) {
    RankJob j;
    std::memset(&j, 0, sizeof j);
    j.t = t;
    j.ctl = ctl;
    j.frame = frame;
    return j;
}
cudaError_t RankScratch::need(size_t, size_t) { return cudaGetLastError(); }
void RankScratch::release() {}
cudaError_t launch_ranked(const RankJob& one, const RankJob*, uint32_t, unsigned long long, unsigned long long*, bool,
                          unsigned long long* k, double* re, double* im, unsigned long long cap, bool, PruneBits,
                          unsigned long long*, unsigned long long*, cudaStream_t) {
    emit(one.t, const_cast<Ctl*>(one.ctl), one.frame, k, re, im, cap, 0, 0);
    return cudaGetLastError();
}
cudaError_t launch_norm(const TableDev&, Ctl*, unsigned long long, bool, ExactSums*, int, cudaStream_t) { return cudaGetLastError(); }
cudaError_t launch_compare(const TableDev&, const Ctl*, unsigned long long, bool, const TableDev&, const Ctl*, unsigned long long,
                           bool, unsigned long long, Ctl*, ExactSums*, int, cudaStream_t) { return cudaGetLastError(); }
cudaError_t measure_fp64_rate(int, double*) { return cudaGetLastError(); }
// The rebuild drops groups without keys; a hashed table takes at most what its buckets hold.
cudaError_t launch_rehash(const TableDev&, unsigned long long, const TableDev& nt, unsigned, int, Ctl* ctl, int, cudaStream_t) {
    State& st = fake::dev.state[ctl];
    st.live.clear();
    for (auto& kv : st.amp) st.live.insert(kv.first >> kSlotBits);
    ctl->list_tail = st.live.size();
    if (st.live.size() > nt.mask + 1) ctl->status = ST_TABLE_FULL;
    return cudaGetLastError();
}
cudaError_t launch_pattern_prob(const TableDev&, Ctl*, unsigned long long, bool, unsigned long long, unsigned long long, ExactSums*,
                                int, cudaStream_t) { return cudaGetLastError(); }
cudaError_t launch_collapse(const TableDev&, Ctl*, unsigned long long, bool, unsigned long long, unsigned long long, double, int,
                            cudaStream_t) { return cudaGetLastError(); }
size_t sort_scratch_bytes(unsigned long long) { return 256; }
cudaError_t sort_entries(SortBuffers& b, unsigned long long n, uint32_t, bool, int, cudaStream_t) {
    std::memcpy(b.keys_out, b.keys_in, n * 8);   // (emit writes in key order)
    std::memcpy(b.re_out, b.re_in, n * 8);
    std::memcpy(b.im_out, b.im_in, n * 8);
    return cudaGetLastError();
}
size_t cumulate_scratch_bytes(unsigned long long) { return 256; }
cudaError_t cumulate(const double*, const double*, double*, unsigned long long, void*, size_t, int, cudaStream_t) { return cudaGetLastError(); }
cudaError_t launch_sample(const unsigned long long*, const double*, unsigned long long, unsigned long long, unsigned long long,
                          unsigned long long*, int, cudaStream_t) { return cudaGetLastError(); }
}  // namespace sqc
