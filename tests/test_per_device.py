"""The once-per-device bookkeeping of the kernels' shared-memory opt-in: each
device of a process gets its own, a failure is not remembered, and callers racing
on one device run it once.  Plain C++, built with the host compiler."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "per_device.cuh"
#include <cstdio>
#include <thread>
#include <vector>
#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)
static att::OncePerDevice once;
int main() {
    int calls[80] = {};
    auto ask = [&](int d) { return once.run(d, [&] { ++calls[d]; return 0; }); };
    for (int k = 0; k < 3; ++k)
        for (int d = 0; d < 64; ++d) CHECK(ask(d) == 0 && calls[d] == 1);
    CHECK(ask(70) == 0 && ask(70) == 0 && calls[70] == 2);  // past the table: every time
    static att::OncePerDevice failing;
    int n = 0;
    CHECK(failing.run(1, [&] { ++n; return 2; }) == 2);
    CHECK(failing.run(0, [&] { ++n; return 0; }) == 0 && n == 2);  // another device: its own
    CHECK(failing.run(1, [&] { ++n; return 0; }) == 0 && n == 3);  // tried again
    CHECK(failing.run(1, [&] { ++n; return 2; }) == 0 && n == 3);
    static att::OncePerDevice raced;
    std::atomic<int> runs{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] { for (int d = 0; d < 32; ++d) raced.run(d, [&] { ++runs; return 0; }); });
    for (auto &t : threads) t.join();
    CHECK(runs == 32);
    return 0;
}
"""


def test_once_per_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "att_gb300", "csrc"), str(src),
                    "-o", str(exe)], check=True)
    done = subprocess.run([str(exe)], stdout=subprocess.PIPE, text=True)
    assert done.returncode == 0, done.stdout


def test_every_opt_in_is_per_device():
    """No kernel sets its shared-memory attribute anywhere but in dynamic_smem."""
    csrc = os.path.join(ROOT, "att_gb300", "csrc")
    found = {}
    for name in sorted(os.listdir(csrc)):
        with open(os.path.join(csrc, name)) as f:
            n = f.read().count("cudaFuncSetAttribute(")
        if n:
            found[name] = n
    assert found == {"att_common.cuh": 1}
