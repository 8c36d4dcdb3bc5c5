"""Pinned host blocks (csrc/common.cuh) when an allocation fails: the block that
was there is given back once and the object is empty, so that a later, smaller
request allocates again instead of using freed memory. The allocator is a fake
that keeps count, so this needs no GPU."""
import subprocess

from clothcraft_b200 import build

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdio>
#include <cstdlib>
#include <set>

static std::set<void*> live;
static int bad_frees = 0, allocations = 0;
static bool refuse = false;
template <class T>
static cudaError_t fake_alloc(T** p, size_t bytes) {
    if (refuse) return cudaErrorMemoryAllocation;
    *p = static_cast<T*>(std::malloc(bytes));
    live.insert(*p);
    ++allocations;
    return cudaSuccess;
}
static cudaError_t fake_free(void* p) {
    if (!live.erase(p)) ++bad_frees;  // not freed twice, nor memory that is not ours
    return cudaSuccess;
}
#define cudaMallocHost fake_alloc
#define cudaFreeHost fake_free
#include "common.cuh"

int main() {
    {
        cc::Pinned<double> p;
        p.reserve(10);
        refuse = true;
        bool failed = false;
        try {
            p.reserve(20);
        } catch (const cc::Failure&) {
            failed = true;
        }
        refuse = false;
        if (!failed || p.cap != 0 || p.ptr) return 1;
        p.reserve(5);  // would fit the block that was given back
        if (p.cap != 5 || !live.count(p.ptr) || allocations != 2) return 2;
    }
    return live.empty() && bad_frees == 0 ? 0 : 3;
}
"""


def test_failed_growth_leaves_an_empty_block(tmp_path):
    src, exe = tmp_path / "pinned.cu", tmp_path / "pinned"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC, str(src), "-o", str(exe)] + build._flags(), check=True)
    assert subprocess.run([str(exe)], timeout=60).returncode == 0
