"""The device buffer (common.cuh) against an allocator that runs out of memory, compiled here with g++ and a
stand-in for the CUDA runtime: a buffer whose allocation failed is empty, so that a caller that tries again,
or asks whether the buffer is long enough, never takes a null pointer for memory."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "flexiblefmm.jl_b200", "csrc")
MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "common.cuh"
using namespace fmmb;
static bool full = false;
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { if (full) return cudaErrorMemoryAllocation; *p = malloc(n); return cudaSuccess; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "out of memory"; }
}
static int failed(DBuf<double>& b, size_t n) {
  full = true;
  int code = 0;
  try { b.alloc(n); } catch (const Error& e) { code = e.code; }
  full = false;
  return code;
}
int main() {
  for (cudaStream_t s : {(cudaStream_t) nullptr, (cudaStream_t)8}) {
    g_alloc_stream = s;
    DBuf<double> a, b(10);
    if (failed(a, 5) != FMMB_ERR_MEMORY || a.p || a.n) return 1;     // a first allocation
    if (failed(b, 20) != FMMB_ERR_MEMORY || b.p || b.n) return 2;    // in place of a shorter one
    a.alloc(5);
    if (!a.p || a.n != 5) return 3;
  }
  return 0;
}
"""


def test_a_failed_allocation_leaves_an_empty_buffer(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I/usr/local/cuda/include", "-I" + CSRC, str(tmp_path / "main.cpp"),
                    "-o", str(tmp_path / "main")], check=True)
    assert subprocess.run([str(tmp_path / "main")]).returncode == 0
