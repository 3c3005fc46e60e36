"""Scratch memory of the engine's scans and rule chains (csrc/stream_memory.hpp) against
a fake allocator on the host: given back once on its own stream when its scope ends,
normally or by an exception, and nothing held or freed after a failed allocation."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "stream_memory.hpp"
#include <cstdio>
#include <cstdlib>
#include <map>
#include <stdexcept>
static std::map<void *, cudaStream_t> held;
static int left = 3, cleared = 0, wrong = 0;
extern "C" cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t st) {
  if (left-- <= 0) { *p = (void *)1; return cudaErrorMemoryAllocation; }
  *p = std::malloc(n);
  held[*p] = st;
  return cudaSuccess;
}
extern "C" cudaError_t cudaFreeAsync(void *p, cudaStream_t st) {
  wrong += !held.count(p) || held[p] != st;
  held.erase(p);
  return cudaSuccess;
}
extern "C" cudaError_t cudaGetLastError() { cleared++; return cudaSuccess; }
static int scan(cudaStream_t st) {
  mapb::StreamMemory a(st), b(st);
  if (a.alloc(64) != cudaSuccess) return 1;
  if (b.alloc(64) != cudaSuccess) throw std::runtime_error("second allocation");
  return a.ptr() && b.ptr() ? 0 : 2;
}
int main() {
  const cudaStream_t st = (cudaStream_t)0x40;
  if (scan(st) != 0 || !held.empty()) return 1;
  bool thrown = false;
  try { scan(st); } catch (const std::exception &) { thrown = true; }   // the pool is empty at the second
  if (!thrown || !held.empty()) return 2;
  if (scan(st) != 1 || !held.empty()) return 3;
  return wrong || cleared != 2 ? 4 : 0;
}
"""


def test_given_back_whichever_way_the_scope_ends(tmp_path):
    src = tmp_path / "scratch.cpp"
    src.write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "scratch")
    subprocess.run(["g++", "-std=c++17", "-O1", str(src), "-o", exe, "-I" + os.path.join(ROOT, "map_b200", "csrc"),
                    "-I" + os.path.join(cuda, "include")], check=True)
    assert subprocess.run([exe]).returncode == 0


def test_no_bare_pool_allocation_in_the_scans():
    # every scratch area of the scans goes through the class above
    text = open(os.path.join(ROOT, "map_b200", "csrc", "codegen_scan.cpp")).read()
    assert "cudaMallocAsync(" not in text and "cudaFreeAsync(" not in text
