"""The page-locked buffers a codec's readers share, on the CPU against a counting
stand-in for the two allocation calls: small buffers kept first do not keep
large ones out, what is kept is given up when memory runs out, and nothing is
leaked or freed twice."""

import os
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "fritillaria_gb300" / "csrc"
CUDA = Path(os.environ.get("CUDA_HOME", "/usr/local/cuda")) / "include"

PROGRAM = r"""
#include "pinned.h"
#include <cstdio>
#include <cstdlib>
#include <map>
static std::map<void *, size_t> held;
static size_t total = 0, limit = ~(size_t)0;
extern "C" cudaError_t cudaMallocHost(void **p, size_t n)
{
    if (total + n > limit) return cudaErrorMemoryAllocation;
    *p = malloc(64);
    held[*p] = n;
    total += n;
    return cudaSuccess;
}
extern "C" cudaError_t cudaFreeHost(void *p)
{
    if (!held.count(p)) abort();
    total -= held[p];
    held.erase(p);
    free(p);
    return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError(void) { return cudaSuccess; }
#define CHECK(x) if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; }
using namespace frt;
constexpr size_t MB = 1 << 20;
int main()
{
    {
        auto pool = std::make_shared<PinnedPool>();
        auto reader = [&](size_t bytes) {
            auto b = std::make_unique<PinnedBytes>();
            b->pool = pool;
            if (!b->reserve(bytes)) b.reset();
            return b;
        };
        { auto a = reader(1), b = reader(1), c = reader(2 * MB); } // small ones fill the pool
        CHECK(held.size() == 2 && total == 3 * MB)
        { auto a = reader(16 * MB); } // a large one takes a small one's place
        CHECK(held.size() == 2 && total == 18 * MB)
        { auto a = reader(32 * MB); }
        CHECK(held.size() == 2 && total == 48 * MB)
        void *kept = nullptr;
        { auto a = reader(20 * MB); kept = a->p; CHECK(a->cap == 32 * MB) }
        { auto a = reader(20 * MB); CHECK(a->p == kept) } // handed on
        { auto a = reader(3 * MB); CHECK(a->cap == 16 * MB) }
        { auto a = reader(128 * MB); CHECK(total == 176 * MB) } // past MAX_BYTES: not kept
        CHECK(held.size() == 2 && total == 48 * MB)
        { auto a = reader(20 * MB); a->idle = false; } // a copy may be in flight: not kept
        CHECK(held.size() == 1 && total == 16 * MB)
        { auto a = reader(10 * MB), b = reader(20 * MB); }
        CHECK(total == 48 * MB)
        limit = 100 * MB; // 64 MB more are to be had only once the kept ones go
        { auto a = reader(60 * MB); CHECK(a && a->cap == 64 * MB && total == 64 * MB) }
        { auto a = reader(128 * MB); CHECK(!a && total == 0) }
        { auto a = reader(60 * MB); CHECK(a && a->cap == 64 * MB) } // and later ones work
    }
    CHECK(held.empty() && total == 0)
    printf("ok\n");
    return 0;
}
"""


def test_pool_keeps_the_large_and_gives_up_when_asked(tmp_path):
    if not shutil.which("g++") or not (CUDA / "cuda_runtime_api.h").exists():
        pytest.skip("no compiler or CUDA headers")
    src = tmp_path / "pool.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "pool"
    subprocess.run(["g++", "-std=c++17", "-Wall", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert (r.returncode, r.stdout) == (0, "ok\n"), r.stdout
