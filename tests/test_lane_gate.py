"""The turns of the solve service's lanes (csrc/lane_gate.h), on the CPU: in
the order in which they were asked for, at most two at a time."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "cudaplasticity_b200", "csrc")

SOURCE = r"""
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "lane_gate.h"
int main() {
    cp::LaneGate gate;
    if (gate.shared()) return 1;
    gate.busy = 1;
    if (gate.shared()) return 2;
    gate.busy = 2;
    if (!gate.shared()) return 3;
    std::atomic<int> inside{0}, most{0}, turns{0};
    std::vector<std::vector<int>> at(6);
    std::vector<std::thread> lanes;
    for (int k = 0; k < 6; ++k)
        lanes.emplace_back([&, k] {
            for (int i = 0; i < 200; ++i) {
                cp::LaneGate::Turn turn(gate);
                const int now = ++inside;
                int m = most;
                while (m < now && !most.compare_exchange_weak(m, now)) {}
                at[k].push_back(turns++);
                std::this_thread::sleep_for(std::chrono::microseconds(50));
                --inside;
            }
        });
    // an error leaves its turn like any other end
    for (int i = 0; i < 5; ++i)
        try {
            cp::LaneGate::Turn turn(gate);
            throw 1;
        } catch (int) {
        }
    for (auto& t : lanes) t.join();
    // while all six are at work no lane waits for more than a few rounds of the others
    int gap = 0;
    for (auto& v : at)
        for (size_t i = 1; i < 100; ++i) gap = gap < v[i] - v[i - 1] ? v[i] - v[i - 1] : gap;
    printf("%d %d\n", (int)most, gap);
    return 0;
}
"""


def test_turns(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    (tmp_path / "t.cpp").write_text(SOURCE)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(tmp_path / "t.cpp"), "-o", exe], check=True)
    most, gap = map(int, subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout.split())
    assert most == 2
    assert gap <= 24  # (six turns between two of a lane's; a thread that starts late asks late)
