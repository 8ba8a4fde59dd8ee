"""The host threads behind staging copies (csrc/host_pool.h), compiled for the CPU: every item runs
exactly once and before run() returns, over many short runs in a row (a worker that wakes late, in a
later run or in none, takes nothing of an earlier one), and runs of one item stay on the caller."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "cuda_ndt_matcher_gb300", "csrc")

SRC = r"""
#include "host_pool.h"
#include <cstdio>
#include <memory>
int main() {
    ndtgb::HostPool pool;
    for (int round = 0; round < 20000; ++round) {
        const uint64_t n = round % 7 == 0 ? 1 : (uint64_t)(round % 37);
        // freed and refilled at once: a late call would write into another round's counts
        std::unique_ptr<std::atomic<int>[]> hit(new std::atomic<int>[n + 1]);
        for (uint64_t i = 0; i <= n; ++i) hit[i] = 0;
        const auto me = std::this_thread::get_id();
        bool other = false;
        pool.run(n, [&](uint64_t i) {
            hit[i].fetch_add(1);
            if (n == 1) other = std::this_thread::get_id() != me;
        });
        if (other) return 2;
        for (uint64_t i = 0; i <= n; ++i)
            if (hit[i].load() != (i < n ? 1 : 0)) return 1;
    }
    std::puts("ok");
}
"""


def test_every_item_once(tmp_path):
    src, exe = tmp_path / "pool.cpp", tmp_path / "pool"
    src.write_text(SRC)
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", CSRC, "-o", str(exe), str(src)],
                   check=True)
    for _ in range(3):
        r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
        assert r.returncode == 0 and r.stdout.strip() == "ok", r
