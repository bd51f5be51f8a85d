"""Kernel attributes (more than 48 KB of shared memory) belong to one device: with handles on several devices in a process each
device gets them once. The helper is compiled and run here; more than one GPU is not used by the tests."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "parts-sim_b200", "csrc")

PROGRAM = r"""
#include <atomic>
#include <cstdio>
#include "host_util.hpp"
int main() {
    static psfea::OncePerDevice once;
    std::atomic<int> runs[4] = {};
    std::vector<std::thread> th;
    for (int t = 0; t < 16; t++)
        th.emplace_back([&, t] {
            for (int k = 0; k < 100; k++) once.run((t + k) % 4, [&] { runs[(t + k) % 4]++; });
        });
    for (auto& t : th) t.join();
    for (auto& r : runs)
        if (r != 1) return 1;
    // a failure is not remembered as done
    psfea::OncePerDevice again;
    int tries = 0;
    try {
        again.run(2, [&] { tries++; throw psfea::Error(PS_ECUDA, "no"); });
        return 2;
    } catch (const psfea::Error&) {
    }
    again.run(2, [&] { tries++; });
    again.run(2, [&] { tries++; });
    return tries == 2 ? 0 : 3;
}
"""


def test_each_device_once(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-pthread", f"-I{CSRC}", f"-I{os.path.join(HERE, '..', 'include')}", "-o", str(exe), str(tmp_path / "t.cpp")], check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0


def test_no_attribute_is_set_once_for_the_process():
    with open(os.path.join(CSRC, "solver.cu")) as f:
        src = f.read()
    assert "call_once" not in src and src.count("OncePerDevice attrOnce") == 2
