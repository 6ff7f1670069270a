"""Launch state that belongs to a (kernel, device) pair (`csrc/per_device.hpp`), compiled for the host with a stand-in for the
CUDA call: every device is configured for itself, a limit is only ever raised, and threads do not lose one another's."""
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wick_b200", "csrc")

PROGRAM = r"""
#include <cstdio>
#include <thread>
#include <vector>
#include "per_device.hpp"
#define CHECK(c) if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; }
int main() {
    wick::RaisedPerDevice state;
    size_t limit[100] = {};
    int calls = 0, failing = 0;
    auto on = [&](int dev) { return [&, dev](size_t v) { calls++; if (failing) return 2; limit[dev] = v; return 0; }; };
    CHECK(state.raise(0, 220, on(0)) == 0 && limit[0] == 220);
    CHECK(state.raise(1, 220, on(1)) == 0 && limit[1] == 220);           // the second device is not the first
    CHECK(state.raise(0, 100, on(0)) == 0 && limit[0] == 220 && calls == 2);  // never lowered, no call
    failing = 1;
    CHECK(state.raise(2, 50, on(2)) == 2);                               // a failure is passed on and not remembered
    failing = 0;
    CHECK(state.raise(2, 50, on(2)) == 0 && limit[2] == 50);
    CHECK(state.raise(80, 50, on(80)) == 0 && state.raise(80, 40, on(80)) == 0 && limit[80] == 50);  // beyond the table
    for (int round = 0; round < 200; round++) {                          // whatever the order, the largest request is granted
        wick::RaisedPerDevice s;
        size_t now = 0;
        std::vector<std::thread> t;
        for (size_t v = 1; v <= 8; v++) t.emplace_back([&, v] { s.raise(3, v, [&](size_t x) { now = x; return 0; }); });
        for (auto& x : t) x.join();
        CHECK(now == 8);
    }
    return 0;
}
"""


def test_launch_state_is_kept_per_device(tmp_path):
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(tmp_path / "t"), str(src)])
    out = subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout


@pytest.mark.parametrize("name", ["gemm_tc.cu", "kernels_attn.cu", "kernels_batch.cu"])
def test_launchers_keep_no_state_of_their_own(name):
    """No plain function-level static in a launcher: it would be one value for all devices, unsynchronised between threads."""
    code = open(os.path.join(CSRC, name)).read()
    assert not re.findall(r"^\s+static (?:bool|int|size_t) \w+(?:\[\w+\])? = .*$", code, flags=re.M)


@pytest.mark.parametrize("name", ["gemm_tc.cu", "kernels_attn.cu", "kernels_batch.cu", "decode_mega.cu"])
def test_shared_memory_is_only_ever_raised(name):
    """A bare set of a kernel's shared-memory limit lowers it under another thread that is about to launch with more."""
    code = open(os.path.join(CSRC, name)).read()
    assert "cudaFuncAttributeMaxDynamicSharedMemorySize" not in code and "raise_dynamic_smem" in code


@pytest.mark.gpu
def test_operator_gemm_on_every_device(cuda_lib, orc):
    """The product of more than 8 columns on each device of a process (a launch was refused on all but the first)."""
    torch = pytest.importorskip("torch")
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    import numpy as np
    from wick_b200 import gguf_synth as gs, ops
    rng = np.random.default_rng(0)
    raw = gs.quantize_q4_0((rng.standard_normal((256, 128)) * 0.02).astype(np.float32))
    bs, bq = orc.quantize_q8_0(rng.standard_normal((9, 128), dtype=np.float32))
    want = orc.gemv(orc.DT_Q4_0, raw, bs[8], bq[8], 256, 128)
    for d in range(2):
        with torch.cuda.device(d):
            w = ops.QuantWeight(ops.DT_Q4_0, raw, 256, 128)
            out = ops.gemm_q8(w, torch.from_numpy(bs).cuda(), torch.from_numpy(bq).cuda())
            assert np.array_equal(out[8].cpu().numpy().view(np.uint32), want.view(np.uint32))
