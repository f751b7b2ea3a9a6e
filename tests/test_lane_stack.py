"""The stack that the lanes of a warp keep in common (csrc/snk_lane_stack.h), on the host: two
threads as lanes, one of them held up longer before every read.  An entry that a pop frees must not
be overwritten before every lane has read it."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "snake-vk_gb300", "csrc")

SOURCE = r"""
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include "snk_lane_stack.h"

static std::atomic<int> entries[8], arrived[64];
static bool good[2] = {true, true};

static void lane(int id) {
    int sp = 0, waits = 0;
    auto push = [&](int v) { entries[sp++] = v; };
    auto pop = [&](int want) {
        const int got = snk::lanes_pop<int>(
            [&](int k) {
                std::this_thread::sleep_for(std::chrono::milliseconds(id ? 50 : 10));
                return entries[k].load();
            },
            sp, [&] {
                const int w = waits++;
                arrived[w]++;
                while (arrived[w] < 2) std::this_thread::yield();
            });
        if (got != want) good[id] = false;
    };
    push(1); push(2); push(3);
    pop(3);
    push(4);            // over the entry just read, as an instance group does with what is left of it
    pop(4); pop(2);
    push(5); push(6);
    pop(6); pop(5); pop(1);
}

int main() {
    std::thread a(lane, 0), b(lane, 1);
    a.join();
    b.join();
    std::puts(good[0] && good[1] ? "same" : "differ");
}
"""


def test_lanes_read_the_same_entries(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "lanes.cpp", tmp_path / "lanes"
    src.write_text(SOURCE)
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.stdout.strip() == "same"
