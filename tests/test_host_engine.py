"""The engine's host code on the CPU: sqc_engine.cpp and sqc_plan.cpp over a device made of host
memory (tests/host_engine/fake_device.h), whose allocations can be made to fail. What these tests show
is what the engine launches, waits for and keeps, not what the kernels compute.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "sparqc_gb300", "csrc")
FLAGS = ["-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", CSRC, "-I", os.path.join(HERE, "host_engine")]


def _cuda_include():
    for d in (os.environ.get("CUDA_HOME", "/usr/local/cuda"), "/usr/local/cuda"):
        if os.path.exists(os.path.join(d, "include", "cuda_runtime.h")):
            return ["-I", os.path.join(d, "include")]
    pytest.skip("no CUDA headers")


@pytest.fixture(scope="session")
def engine_objects(tmp_path_factory):
    out = tmp_path_factory.mktemp("host_engine")
    objs = []
    for src in ("sqc_engine.cpp", "sqc_plan.cpp", "sqc_devmem.cpp"):
        obj = out / (src + ".o")
        subprocess.run(["g++", *FLAGS, *_cuda_include(), "-c", os.path.join(CSRC, src), "-o", str(obj)], check=True)
        objs.append(str(obj))
    return objs


def run(engine_objects, tmp_path, body):
    """Compile and run a program whose main is `body` (fake_device.h included); its checks must hold."""
    src = tmp_path / "main.cpp"
    src.write_text('#include "fake_device.h"\nusing namespace sqc;\nusing namespace fake;\nint main() {\n' + body +
                   '\n    CHECK(fake::dev.bad == 0);\n    std::printf("fails=%d\\n", fails);\n    return fails != 0;\n}\n')
    exe = tmp_path / "main"
    r = subprocess.run(["g++", *FLAGS, *_cuda_include(), str(src), *engine_objects, "-o", str(exe)], capture_output=True, text=True)
    if r.returncode != 0:
        pytest.fail(r.stderr[-4000:])
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and "fails=0" in out.stdout, out.stdout[-4000:] + out.stderr[-2000:]


@pytest.mark.parametrize("pieces", [1, 9], ids=["one_call", "calls_of_1024"])
@pytest.mark.parametrize("buckets", [1024, 64], ids=["room", "must_grow"])
def test_questions_after_more_gates_than_descriptors(engine_objects, tmp_path, buckets, pieces):
    """More gates than the descriptor buffer holds (8192): the flush waits for what it launched before and
    launches again, and a question must wait for that. Asked without a sync: the key count, the state, and
    an asynchronous readout."""
    run(engine_objects, tmp_path, """
    for (int ask = 0; ask < 2; ++ask) {
        Engine e;
        sqc_options o;
        sqc_default_options(&o);
        o.initial_buckets = %d;
        make(e, 12, &o);
        std::vector<sqc_gate> g;
        for (uint32_t q = 4; q < 10; ++q) g.push_back(gate(KH, q));
        while (g.size() < 9215) g.push_back(gate(g.size() %% 7 ? KT : KX, 7 + g.size() %% 3, 1ULL << (4 + g.size() %% 3)));
        g.push_back(gate(KH, 10));
        const size_t step = g.size() / %d;
        for (size_t i = 0; i < g.size(); i += step) CHECK(e.apply(g.data() + i, step) == SQC_OK);
        if (ask == 1) {
            std::vector<uint64_t> k(2048);
            std::vector<double> r(2048), i(2048);
            uint64_t n = 0;
            CHECK(e.get_state_async(k.data(), r.data(), i.data(), 2048, &n) == SQC_OK);
            CHECK(e.readout_wait() == SQC_OK);
            CHECK(n == 128);
        }
        CHECK(holds(e, expected(g)));
    }
    """ % (buckets, pieces))


THIN = """
    // few keys over many qubits: a state no map is worth, which outgrows its hashed table
    std::vector<sqc_gate> g;
    for (uint32_t q = 0; q < 6; ++q) g.push_back(gate(KH, q));
    for (uint32_t i = 0; i < 26; ++i) g.push_back(gate(KX, 6 + i, 1ULL << (i % 6)));
    for (uint32_t i = 0; i < 6; ++i) g.push_back(gate(KRY, 8 + 3 * i, 0, 0.7));
"""


@pytest.mark.parametrize("lasting", [1, 2, 1000000])
def test_allocation_failure_in_a_flush_loses_no_gate(engine_objects, tmp_path, lasting):
    """The table cannot be enlarged while a flush is launching (one failed allocation, two, all of them):
    a call may say so, but the gates stay, and the state is the whole circuit's once there is memory."""
    run(engine_objects, tmp_path, THIN + """
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 64;
    make(e, 60, &o);
    dev.big_limit = 64 * e.bucket_bytes_now();
    dev.fail_big = %d;
    CHECK(e.apply(g.data(), g.size()) == SQC_OK);
    const int a = e.flush(), b = e.sync();
    CHECK(a == SQC_OK || a == SQC_ERR_OOM);
    CHECK(b == SQC_OK || b == SQC_ERR_OOM);
    if (%d > 1000) {
        CHECK(b == SQC_ERR_OOM);
        CHECK(e.sync() == SQC_ERR_OOM);   // it stays an error while there is no memory
        uint64_t n = 0;
        CHECK(e.nnz(&n) == SQC_ERR_OOM);
    }
    dev.fail_big = 0;
    CHECK(holds(e, expected(g)));
    sqc_stats st;
    e.stats(&st);
    CHECK(st.gates_applied == g.size());
    """ % (lasting, lasting))


def test_failed_copy_in_a_flush_loses_no_gate(engine_objects, tmp_path):
    """A flush that cannot upload its descriptors queues its gates again."""
    run(engine_objects, tmp_path, THIN + """
    Engine e;
    make(e, 60);
    CHECK(e.apply(g.data(), 10) == SQC_OK && e.flush() == SQC_OK);
    dev.fail_copies = 1;
    CHECK(e.apply(g.data() + 10, g.size() - 10) == SQC_OK);
    CHECK(e.flush() == SQC_ERR_CUDA);
    CHECK(holds(e, expected(g)));
    """)


def test_meeting_wait_ends_when_the_state_has_failed(tmp_path):
    """The wait of a run's blocks at a meeting (sqc_meet.h): over when the others are there, soon over when the
    state has failed (a block that saw that at its start never comes), and bounded."""
    src = tmp_path / "meet.cpp"
    src.write_text(r"""
#include <cstdio>
#include <initializer_list>
#include "sqc_meet.h"
using namespace sqc;
static int fails = 0;
#define CHECK(c) do { if (!(c)) { std::printf("FAIL line %d: %s\n", __LINE__, #c); ++fails; } } while (0)
template <bool LOOK = true>
static Meet wait(unsigned long met_at, unsigned long failed_at, unsigned long* polls) {
    unsigned long n = 0;
    const Meet m = wait_meeting<LOOK>([&] { return ++n >= met_at; }, [&] { return n >= failed_at ? ST_TABLE_FULL : ST_OK; });
    *polls = n;
    return m;
}
int main() {
    const unsigned long never = ~0UL;
    unsigned long n;
    for (unsigned long at : {1UL, 2UL, 63UL, 64UL, 65UL, 1000UL, (unsigned long)kMaxPolls}) CHECK(wait(at, never, &n) == MEET_OK && n == at);
    CHECK(wait(1, 0, &n) == MEET_OK);
    for (unsigned long at : {0UL, 1UL, 64UL, 65UL, 100000UL}) CHECK(wait(never, at, &n) == MEET_FAILED && n <= at + kStatusPolls);
    CHECK(wait(never, never, &n) == MEET_TIMEOUT && n == kMaxPolls);
    CHECK(wait<false>(1000, 0, &n) == MEET_OK && n == 1000);
    CHECK(wait<false>(never, never, &n) == MEET_TIMEOUT && n == kMaxPolls);
    std::printf("fails=%d\n", fails);
}
""")
    exe = tmp_path / "meet"
    subprocess.run(["g++", *FLAGS, str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "fails=0\n"


@pytest.mark.parametrize("groups,runs", [(1 << 17, 1), ((1 << 17) + 1, 0)])
def test_large_hashed_states_make_no_runs(engine_objects, tmp_path, groups, runs):
    """Passes go out in one launch while the state has at most 2^17 live buckets, whatever gates they hold."""
    run(engine_objects, tmp_path, """
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.max_fused_gates = 2;
    make(e, 60, &o);
    const size_t n = %d;
    std::vector<uint64_t> k(n);
    std::vector<double> r(n, 0.001), i(n, 0.0);
    for (size_t j = 0; j < n; ++j) k[j] = (j * 0x9E3779B97F4A7C15ULL) >> 4 & ~15ULL;
    CHECK(e.set_state(k.data(), r.data(), i.data(), n) == SQC_OK);
    std::vector<sqc_gate> g;
    for (int j = 0; j < 5; ++j) g.push_back(gate(KT, 59 - j, 1ULL << (10 + j)));
    CHECK(e.apply(g.data(), g.size()) == SQC_OK && e.sync() == SQC_OK);
    CHECK(dev.passes == 3 && dev.runs == %d);
    """ % (groups, runs))


def test_timed_passes_of_a_table_that_is_enlarged(engine_objects, tmp_path):
    """Enlarging a table between two passes reads the events of the passes before it: every later pass
    still spans from an event of its own to the next."""
    run(engine_objects, tmp_path, THIN + """
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 64;
    o.time_passes = 1;
    make(e, 60, &o);
    for (int k = 0; k < 3; ++k) {
        CHECK(e.set_zero() == SQC_OK);
        CHECK(e.apply(g.data(), g.size()) == SQC_OK);
        CHECK(holds(e, expected(g)));
    }
    sqc_stats st;
    e.stats(&st);
    // one tick of the fake clock per pass, and none for what lies between two
    CHECK(st.pass_ns_pair + st.pass_ns_stream == (unsigned long long)dev.passes * 1000000ULL);
    CHECK(st.buckets > 64);
    """)


def test_flush_waits_for_nothing_while_recording(engine_objects, tmp_path):
    """A flush whose launches are recorded into a graph does not stop to enlarge the table: the passes are
    recorded, one without room refuses when it runs, and the next sync repairs that."""
    run(engine_objects, tmp_path, THIN + """
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 64;
    make(e, 60, &o);
    CHECK(e.apply(g.data(), g.size()) == SQC_OK);
    dev.capturing = true;
    const long before = dev.syncs;
    CHECK(e.flush() == SQC_OK);
    CHECK(dev.syncs == before);
    dev.capturing = false;
    CHECK(holds(e, expected(g)));
    """)


MOVES = """
    // 2^10 keys that move about: the groups they leave fill the table, which is rebuilt again and again
    std::vector<sqc_gate> g;
    for (uint32_t q = 0; q < 10; ++q) g.push_back(gate(KH, q));
    for (uint32_t i = 0; i < 200; ++i) g.push_back(gate(KX, 10 + i % 40, 1ULL << (i % 10) | 1ULL << ((i * i + 3 * i + 1) % 10)));
"""


def test_kept_tables_are_counted_and_given_back(engine_objects, tmp_path):
    """The table a rebuild leaves is kept for the next one: it is in the state's bytes, another state's
    allocation gets its memory when there is no other, and so does this state's own."""
    run(engine_objects, tmp_path, MOVES + """
    auto buffers = [](size_t held, const sqc_stats& st) { return held - (size_t)st.table_bytes; };
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 1 << 12;
    Engine a;
    make(a, 60, &o);
    sqc_stats st;
    a.stats(&st);
    const size_t other = buffers(dev.held, st);
    size_t kept = 0;
    for (int k = 0; k < 3; ++k) {
        CHECK(a.set_zero() == SQC_OK && a.apply(g.data(), g.size()) == SQC_OK && a.sync() == SQC_OK);
        a.stats(&st);
        kept = (size_t)st.table_bytes - (size_t)st.buckets * a.bucket_bytes_now();
        CHECK(buffers(dev.held, st) == other);   // (no readout yet)
    }
    CHECK(kept > 0);
    dev.total = dev.held + (4 << 20);   // (another state's small buffers)
    {
        Engine b;
        o.initial_buckets = kept / a.bucket_bytes_now();
        make(b, 60, &o);
        a.stats(&st);
        CHECK(st.table_bytes == st.buckets * a.bucket_bytes_now());
        dev.total = dev.held + (4 << 20);
    }
    CHECK(holds(a, expected(g)));
    dev.total = (size_t)284 << 30;
    CHECK(a.set_zero() == SQC_OK && a.apply(g.data(), g.size()) == SQC_OK);
    CHECK(holds(a, expected(g)));
    """)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("keys", [16, 300])
def test_small_sparse_states_stay_small(engine_objects, tmp_path, keys, precision):
    """A few hundred keys over many qubits hold a few megabytes, tables kept for a rebuild included."""
    run(engine_objects, tmp_path, """
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.precision = %d;
    make(e, 60, &o);
    std::vector<uint64_t> k(%d);
    std::vector<double> r(k.size(), 0.05), i(k.size(), 0.0);
    std::map<unsigned long long, Amp> start;
    for (size_t j = 0; j < k.size(); ++j) start[k[j] = ((j + 1) * 0x9E3779B97F4A7C15ULL) >> 4] = Amp(0.05, 0.0);
    CHECK(e.set_state(k.data(), r.data(), i.data(), k.size()) == SQC_OK);
    std::vector<sqc_gate> g;
    for (uint32_t j = 0; j < 12; ++j) g.push_back(gate(j %% 6 ? KX : KRY, 7 + 4 * j, j %% 6 ? 1ULL << j : 0, 0.7));
    CHECK(e.apply(g.data(), g.size()) == SQC_OK);
    CHECK(holds(e, expected(g, start)));
    sqc_stats st;
    e.stats(&st);
    std::printf("bytes %%llu\\n", (unsigned long long)st.table_bytes);
    CHECK(st.table_bytes <= (size_t)2 * 16384 * e.bucket_bytes_now());
    """ % (precision, keys))


@pytest.mark.parametrize("mb", [160, 40, 34, 30])
def test_tables_grow_by_what_there_is(engine_objects, tmp_path, mb):
    """2^12 keys in groups of their own on a device with little memory: the table that would be best does not
    fit beside the old one, and a smaller one is taken."""
    run(engine_objects, tmp_path, """
    dev.total = (size_t)%d << 20;
    Engine e;
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 64;
    make(e, 60, &o);
    std::vector<sqc_gate> g;
    for (uint32_t q = 0; q < 12; ++q) g.push_back(gate(KH, q));
    for (uint32_t q = 0; q < 12; ++q) g.push_back(gate(KX, 12 + 4 * q, 1ULL << q));
    CHECK(e.apply(g.data(), g.size()) == SQC_OK);
    CHECK(holds(e, expected(g)));
    """ % mb)


def test_thin_maps_take_a_share_of_the_device(engine_objects, tmp_path):
    """2^14 groups that spread over 18 bits would be mapped by a table of half the device: they are hashed
    instead, and the state takes an eighth of it."""
    run(engine_objects, tmp_path, """
    dev.total = (size_t)512 << 20;
    Engine e;
    make(e, 60);
    std::vector<sqc_gate> g;
    for (uint32_t q = 4; q < 18; ++q) g.push_back(gate(KH, q));
    for (uint32_t q = 0; q < 4; ++q) g.push_back(gate(KX, 20 + 4 * q, 7ULL << (4 + 3 * q)));
    CHECK(e.apply(g.data(), g.size()) == SQC_OK);
    CHECK(holds(e, expected(g)));
    sqc_stats st;
    e.stats(&st);
    std::printf("bytes %llu peak %zu\\n", (unsigned long long)st.table_bytes, dev.peak);
    CHECK(st.table_bytes <= dev.total / 8 && dev.peak <= dev.total / 2);
    """)


def test_runs_of_thin_mapped_states_take_few_blocks(engine_objects, tmp_path):
    """A run whose passes walk the list is launched for the live buckets there can be, not for every unit of
    the map; one whose passes walk the units for those."""
    run(engine_objects, tmp_path, """
    sqc_options o;
    sqc_default_options(&o);
    o.initial_buckets = 1 << 18;
    for (uint32_t k : {4u, 14u}) {   // keys: 2^4, or 2^14 that fill the map
        Engine e;
        make(e, 40, &o);
        dev.items = 0;
        std::vector<sqc_gate> g;
        for (uint32_t q = 0; q < k; ++q) g.push_back(gate(KH, 4 + q));
        for (uint32_t q = k; q < 14; ++q) g.push_back(gate(KX, 4 + q, 1ULL << (4 + q % k)));
        CHECK(e.apply(g.data(), g.size()) == SQC_OK && e.sync() == SQC_OK);
        CHECK(dev.items == (k == 4 ? 16u * 6u : 1u << 12));
        CHECK(holds(e, expected(g)));
    }
    """)
