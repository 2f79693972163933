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
