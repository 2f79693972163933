"""The host side of the kernels, without a GPU: what is set up per device, and what a launch is told."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "llm_infrence_engine_b200" / "csrc"


def test_once_per_device(tmp_path):
    """Each device is served, each once, a failure is tried again, and threads that come together all find it done."""
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "t.cpp").write_text('''
#include "per_device.h"
#include <cassert>
#include <thread>
#include <vector>
int main() {
    static OncePerDevice once;
    int calls[80] = {};
    auto grant = [&](int d, int rc = 0) { return once.run(d, [&] { ++calls[d]; return rc; }); };
    for (int d : {0, 1, 0, 63, 1, 63}) assert(grant(d) == 0);
    assert(calls[0] == 1 && calls[1] == 1 && calls[63] == 1);
    assert(grant(2, 7) == 7 && grant(2) == 0 && grant(2) == 0 && calls[2] == 2);
    assert(grant(70) == 0 && grant(70) == 0 && calls[70] == 2);
    static OncePerDevice shared;
    std::atomic<int> granted[8] = {};
    std::vector<std::thread> all;
    for (int t = 0; t < 16; ++t)
        all.emplace_back([&, t] { assert(shared.run(t % 8, [&] { granted[t % 8] = 1; return 0; }) == 0); assert(granted[t % 8] == 1); });
    for (auto& t : all) t.join();
}
''')
    subprocess.run([cxx, "-std=c++17", "-pthread", "-I", str(CSRC), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True, timeout=60)


@pytest.mark.parametrize("name", ["gemm_simt.cu", "mlstm.cu"])
def test_shared_memory_is_granted_on_every_device(name):
    """A grant kept in a plain static is the first device's alone: a second device of the process would refuse the launch."""
    text = (CSRC / name).read_text()
    assert not re.search(r"static[^;\n]*cudaFuncSetAttribute", text) and "grant_shared(" in text


def _fake_kernels(monkeypatch):
    """The kernels' Python side over a library that notes what every launch is told."""
    import torch

    from llm_infrence_engine_b200.csrc import kernels

    told = []

    class Library:
        def __getattr__(self, name):
            def call(*args):
                told.append((name, [getattr(a, "value", a) for a in args]))
                return 0

            return call

    monkeypatch.setattr(torch.cuda, "is_available", lambda: True)
    monkeypatch.setattr(kernels, "load_library", Library)
    monkeypatch.setattr(kernels.CudaKernels, "_need", staticmethod(lambda *a, **k: None))
    monkeypatch.setattr(kernels.CudaKernels, "_stream", staticmethod(lambda: 0))
    made = kernels.CudaKernels()
    told.clear()
    return made, told


def test_weights_are_fetched_ahead_of_the_wait_only_where_they_lie_at_rest(monkeypatch):
    """A matrix given to a product outside a model's step may be what the kernel before is writing: then nothing of it may be read before
    that kernel has finished. Inside ``at_rest`` (a runner's forward) it may. Another thread's ``at_rest`` changes nothing here."""
    import threading

    import torch

    K, told = _fake_kernels(monkeypatch)
    x, w, row = torch.zeros(3, 512), torch.zeros(8, 512), torch.zeros(512)

    def flags():
        told.clear()
        K.linear(x, w)
        K.linear(x, w, add_to=torch.zeros(3, 8))
        K.moe_router(x, w, None, 2)
        K.group_rmsnorm_gate(x, x, 0, row, 512, 1e-5, True, torch.float32)
        K.latent_absorb(x, torch.zeros(4 * 64, 32), None, None, 4, 64, 64, 0, 32)
        K.latent_expand(x, torch.zeros(4, 128, 16), None, 0, 4, 128, 16)
        place = {"llmie_gemm_simt": -2, "llmie_moe_router": -3, "llmie_group_rmsnorm_gate": -2, "llmie_head_matmul": -3}
        assert [n for n, _ in told] == ["llmie_gemm_simt"] * 2 + ["llmie_moe_router", "llmie_group_rmsnorm_gate"] + ["llmie_head_matmul"] * 2
        return [a[place[n]] for n, a in told]

    assert flags() == [0] * 6
    with K.at_rest:
        with K.at_rest:
            pass
        assert flags() == [1] * 6
        seen = []
        t = threading.Thread(target=lambda: seen.append(K.at_rest.depth))
        t.start()
        t.join()
        assert seen == [0]
    assert flags() == [0] * 6


@pytest.mark.parametrize("name,kernel,first", [
    ("gemm_simt.cu", "small_kernel", "fetch_weights(c);"), ("gemm_simt.cu", "tile_kernel", "fetch(t, true, false);"),
    ("moe.cu", "moe_router_kernel", "(w + (size_t)e * K + k)"), ("latent.cu", "head_matmul_kernel", "cp.async.cg"),
    ("layernorm.cu", "group_rmsnorm_gate_held_kernel", "load4(w + "), ("recurrent.cu", "selective_scan_kernel", "dt_bias[stage_c]"),
    ("attention_mma.cu", "attn_mma_decode_kernel", "p.bias + (size_t)head")])
def test_a_wait_stands_before_the_first_read_of_a_weight(name, kernel, first):
    text = (CSRC / name).read_text()
    body = text[text.index(f"{kernel}(", text.index("__global__")):]
    before = body[:body.index(first)]
    assert "pdl_wait_unless(" in before or "pdl_wait();" in before
