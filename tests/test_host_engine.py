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
    for src in ("sqc_engine.cpp", "sqc_plan.cpp"):
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
