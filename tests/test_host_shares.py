"""The host threads' helper: what a share throws reaches the caller after every share has ended (left to itself it
would end the process)."""
import os
import shutil
import subprocess

import pytest

import ommgpu as G

CODE = """
#include <atomic>
#include <cstdio>
#include <functional>
#include <new>
namespace ommgpu {
void host_shares(int n, const std::function<void(int)>& f);
}
int main() {
    for (int bad = 0; bad < 4; ++bad) {
        std::atomic<int> ran{0};
        bool caught = false;
        try {
            ommgpu::host_shares(4, [&](int t) {
                ++ran;
                if (t >= bad) throw std::bad_alloc();
            });
        } catch (const std::bad_alloc&) {
            caught = true;
        }
        if (!caught || ran != 4) return 1;
    }
    std::atomic<int> sum{0};
    ommgpu::host_shares(5, [&](int t) { sum += t; });
    if (sum != 10) return 2;
    std::puts("done");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_a_share_that_throws(tmp_path):
    G.lib()
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(CODE)
    lib = os.path.dirname(G.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", str(src), "-o", str(exe), "-L" + lib, "-lommgpu", "-Wl,-rpath," + lib,
                    "-Wl,--allow-shlib-undefined", "-pthread"], check=True)
    env = dict(os.environ, LD_LIBRARY_PATH=os.environ.get("LD_LIBRARY_PATH", "") + ":/usr/local/cuda/lib64")
    r = subprocess.run([str(exe)], env=env, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "done" in r.stdout, (r.returncode, r.stdout, r.stderr)
