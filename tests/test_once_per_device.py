"""Kernel attributes are set once on every device of a process, not once a process (host logic; no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "gpumlib_gb300/csrc/once_per_device.h"
#include <cassert>
#include <thread>
#include <vector>
int main() {
    gpunmf::OncePerDevice<int> once;
    int calls[3] = {0, 0, 0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 12; t++)
        threads.emplace_back([&, t] {
            const int dev = t % 3;
            assert(once.run(dev, [&] { return ++calls[dev] + 10 * dev; }) == 1 + 10 * dev);
        });
    for (auto &t : threads) t.join();
    for (int dev = 0; dev < 3; dev++) assert(calls[dev] == 1);
    return 0;
}
"""


def test_each_device_once(tmp_path):
    src, exe = tmp_path / "once.cpp", tmp_path / "once"
    src.write_text(PROGRAM)
    r = subprocess.run(["g++", "-std=c++17", "-pthread", "-I", ROOT, str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    assert subprocess.run([str(exe)]).returncode == 0


def test_no_attribute_is_set_once_a_process():
    csrc = os.path.join(ROOT, "gpumlib_gb300", "csrc")
    for name in sorted(os.listdir(csrc)):
        assert "call_once" not in open(os.path.join(csrc, name)).read(), name
