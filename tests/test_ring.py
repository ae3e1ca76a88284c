"""The random-number ring of the FP32 electron step (omc_ring.cuh) on a warp
emulated on the host: 32 threads whose stores to shared memory are seen by
the others only after a __syncwarp, as CUDA's memory model has it (shuffles
and votes order nothing).  Lanes take streams at any position, a few of them
have their rings filled by the whole warp, and every number drawn is that of
the stream's own generator."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SRC = r'''
#include <atomic>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#define __host__
#define __device__
#define __forceinline__ inline
#define __noinline__
#define __shared__ thread_local
struct Dim { int x; };
static thread_local Dim threadIdx;
static std::atomic<int> arrived{0}, turn{0};
static void meet() {
    const int t = turn;
    if (++arrived == 32) {
        arrived = 0;
        ++turn;
    } else {
        while (turn == t) std::this_thread::yield();
    }
}
static uint32_t passed[32];
static uint32_t __shfl_sync(unsigned, uint32_t v, int src) {
    passed[threadIdx.x] = v;
    meet();
    const uint32_t r = passed[src];
    meet();
    return r;
}
static int __ffs(unsigned m) { return __builtin_ffs((int)m); }
static void __syncwarp();
#include "omc_ring.cuh"
using Store = omc::RingStore<32, HELD>;
static Store shared_memory;
static std::mutex mu;
static thread_local Store seen;
static void __syncwarp() {
    constexpr int n = sizeof(Store) / 4;
    uint32_t own[n], old[n], all[n];
    std::memcpy(own, &omc::ring<32, HELD>(), sizeof own);
    std::memcpy(old, &seen, sizeof old);
    {
        std::lock_guard<std::mutex> lock(mu);
        std::memcpy(all, &shared_memory, sizeof all);
        for (int i = 0; i < n; i++)
            if (own[i] != old[i]) all[i] = own[i];
        std::memcpy(&shared_memory, all, sizeof all);
    }
    meet();
    seen = shared_memory;
    omc::ring<32, HELD>() = seen;
    meet();
}
int main() {
    std::atomic<long> drawn{0}, bad{0};
    std::vector<std::thread> warp;
    for (int lane = 0; lane < 32; lane++)
        warp.emplace_back([&, lane] {
            threadIdx.x = lane;
            omc::RingStream<32, HELD> g{};
            omc::Philox<float> own;
            uint64_t s = 12345;   // the same choices on every lane
            for (int round = 0; round < 60; round++) {
                // one to eight lanes at work, some of them with a new stream
                s = omc::mix64(s);
                unsigned lanes = 0;
                for (uint64_t k = 0, left = 1 + s % 8; k < left; k++) lanes |= 1u << (omc::mix64(s + k) & 31);
                const bool fresh = round < 2 || (omc::mix64(s ^ lane) & 3) == 0;
                if (fresh) {
                    const uint64_t key = omc::mix64(s + 977 * lane);
                    const uint32_t at = round % 3 ? (uint32_t)(omc::mix64(s * 3 + lane) % 1000) : 0;
                    g.init(key, 7u, at);
                    own.init(key, 7u, at);
                }
                g.assist(lanes);
                int turns = (int)(omc::mix64(s * 5 + lane) % 4);
                for (int t = 0; t <= turns; t++) {
                    const int n = 1 + (int)(omc::mix64(s * 7 + lane + 100 * t) % 13);
                    g.ensure(n);
                    for (int k = 0; k < n; k++) {
                        drawn++;
                        bad += g.uni() != own.uni();
                    }
                    bad += g.position() != own.position();
                }
                __syncwarp();   // the block's barrier between two turns
            }
        });
    for (auto &t : warp) t.join();
    std::printf("%ld %ld\n", drawn.load(), bad.load());
}
'''


@pytest.mark.parametrize("rows", [16, 32, 64])
def test_numbers_are_the_streams_own(tmp_path, rows):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    src = tmp_path / "ring.cpp"
    src.write_text(SRC)
    exe = tmp_path / "ring"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", f"-DHELD={rows}", "-w", "-I",
                    str(ROOT / "ompmc_b200" / "csrc"), "-o", str(exe), str(src)], check=True)
    drawn, bad = map(int, subprocess.run([str(exe)], capture_output=True, text=True, timeout=120).stdout.split())
    assert drawn > 10_000 and bad == 0
