"""The queue of the persistent groups, compiled for the host with a thread per block: every block marches the
same jobs, those that are refused are skipped by all, also where a block reads the group's slot late."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "shg_focused_gaussian_beams_gb300", "csrc")
CUDA_INCLUDE = "/usr/local/cuda/include"

PROGRAM = r"""
#include <cuda_runtime.h>
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>
#include "shg_group_queue.cuh"

int main() {
    const unsigned blocks = 4, njobs = 40;
    std::atomic<unsigned> queue{0}, slot{~0u}, arrived{0};
    std::vector<std::vector<unsigned>> marched(blocks);
    std::atomic<bool> late{false};
    auto block = [&](unsigned rank) {
        unsigned target = 0, job;
        auto meet = [&] {  // bounded, as on the device
            target += blocks;
            arrived.fetch_add(1);
            for (int i = 0; arrived.load() < target; ++i) {
                if (i > 2000000) return late = true, false;
                std::this_thread::yield();
            }
            return !late.load();
        };
        auto take = [&] {
            if (rank == 0) slot.store(queue.fetch_add(1));
        };
        auto read = [&] {
            if (rank == 2) std::this_thread::sleep_for(std::chrono::milliseconds(3));
            return slot.load();
        };
        auto good = [](unsigned j) { return j % 3 != 1; };
        while (shg::group_next(job, njobs, take, meet, read, good)) {
            marched[rank].push_back(job);
            if (!meet() || !meet()) return;  // the march's barriers
        }
    };
    std::vector<std::thread> t;
    for (unsigned r = 0; r < blocks; ++r) t.emplace_back(block, r);
    for (auto &x : t) x.join();
    std::vector<unsigned> want;
    for (unsigned j = 0; j < njobs; ++j)
        if (j % 3 != 1) want.push_back(j);
    for (unsigned r = 0; r < blocks; ++r)
        if (late || marched[r] != want) {
            std::printf("block %u marched %zu of %zu jobs%s\n", r, marched[r].size(), want.size(), late ? ", a barrier gave up" : "");
            return 1;
        }
    return 0;
}
"""


def test_every_block_marches_the_same_jobs(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None or not os.path.exists(os.path.join(CUDA_INCLUDE, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    src, exe = tmp_path / "queue.cpp", tmp_path / "queue"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-I", CUDA_INCLUDE, "-I", CSRC, "-o", str(exe), str(src)],
                   check=True, capture_output=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout
