"""The shared-memory limit of a kernel under two threads that both find it too small."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include "nmg_limit.h"
#include <chrono>
#include <cstdio>
#include <thread>
int main() {
    nmg::GrowingLimit limit;
    std::atomic<int> in_force{0}, sets{0};
    std::atomic<bool> first_has_set{false}, second_is_done{false};
    std::thread second([&] {
        while (!first_has_set) std::this_thread::yield();
        limit.ensure(100, [&](int v) { in_force = v; sets++; return 0; });
        second_is_done = true;
    });
    // the larger request has been set but not recorded yet while the smaller one arrives
    limit.ensure(200, [&](int v) {
        in_force = v; sets++;
        first_has_set = true;
        for (int i = 0; i < 200 && !second_is_done; i++) std::this_thread::sleep_for(std::chrono::milliseconds(1));
        return 0;
    });
    second.join();
    limit.ensure(150, [&](int v) { in_force = v; sets++; return 0; });
    const int failed = limit.ensure(300, [&](int) { return 7; }), again = limit.ensure(300, [&](int v) { in_force = v; return 0; });
    std::printf("%d %d %d %d\n", sets.load(), in_force.load(), failed, again);
    return sets == 1 && in_force == 300 && failed == 7 && again == 0 ? 0 : 1;
}
"""


def test_the_recorded_limit_is_the_one_in_force(tmp_path):
    src, exe = tmp_path / "limit.cpp", tmp_path / "limit"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{os.path.join(ROOT, 'sten_b200', 'csrc')}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
