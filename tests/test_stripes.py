"""The host threads that take a large result over (omc_stripes.h): every stripe
runs once, also when the memory for a thread or for the list of them cannot
be had at any point; nothing escapes and nothing is terminated."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
SRC = r'''
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>
#include "omc_stripes.h"
static std::atomic<int> left{1 << 30};   // allocations that succeed before one fails
void *operator new(size_t n) {
    if (left-- == 0) throw std::bad_alloc();
    return std::malloc(n);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }
int main() {
    for (int n = 1; n <= 4; n++)
        for (int fail = -1; fail < 12; fail++) {
            std::atomic<int> ran[4]{};
            left = fail < 0 ? 1 << 30 : fail;
            omc::run_stripes(n, [&](int k) { ran[k]++; });
            left = 1 << 30;
            for (int k = 0; k < 4; k++)
                if (ran[k] != (k < n)) return std::printf("%d stripes, allocation %d: stripe %d ran %d times\n", n, fail, k, ran[k].load()), 1;
        }
    std::puts("ok");
}
'''


def test_every_stripe_runs_once(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "stripes.cpp", tmp_path / "stripes"
    src.write_text(SRC)
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", str(ROOT / "ompmc_b200" / "csrc"), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout == "ok\n", out.stdout + out.stderr
