"""Thread handling of the staged host copies (csrc/host_copy.cuh) on the CPU, with the CUDA calls replaced."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

from rcabeam_b200 import _build

# A copy during which the n-th allocation fails must still move every byte and return.
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include <new>
#include "host_copy.cuh"

static std::atomic<long> allowed{-1};  // allocations until one fails (-1: none does)
void* operator new(size_t n) {
  if (allowed >= 0 && allowed-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = cudaStream_t(1), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return *e = cudaEvent_t(1), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  return std::memcpy(d, s, n), cudaSuccess;
}
}

int main() {
  const size_t bytes = 20 * rcb::host::kChunk + 12, staging = 8 * 2 * rcb::host::kChunk;
  std::vector<unsigned char> from(bytes), to(bytes), pinned(staging);
  for (size_t i = 0; i < bytes; ++i) from[i] = (unsigned char)(i * 2654435761u >> 13);
  for (long fail = -1; fail < 12; ++fail) {
    for (bool upload : {true, false}) {
      std::fill(to.begin(), to.end(), 0);
      bool ok = false, thrown = false;
      allowed = fail;
      try {
        ok = upload ? rcb::host::copy(from.data(), to.data(), bytes, true, pinned.data(), staging)
                    : rcb::host::copy(to.data(), from.data(), bytes, false, pinned.data(), staging);
      } catch (const std::bad_alloc&) {
        thrown = true;  // before any thread runs: the C entry point returns an error
      }
      allowed = -1;
      if (!thrown && (!ok || to != from)) return std::printf("allocation %ld: wrong copy\n", fail), 1;
      if (thrown && fail > 1) return std::printf("allocation %ld: left with threads running\n", fail), 1;
    }
  }
  return 0;
}
"""


def test_copy_survives_failing_allocations(tmp_path):
    include = Path(_build.nvcc()).resolve().parent.parent / "include"
    if not shutil.which("g++") or not (include / "cuda_runtime.h").exists():
        pytest.skip("needs g++ and the CUDA headers")
    source, program = tmp_path / "copy.cpp", tmp_path / "copy"
    source.write_text("#include <atomic>\n" + PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-I{_build.CSRC}", f"-I{include}", "-x", "c++", str(source),
                    "-o", str(program)], check=True)
    done = subprocess.run([str(program)], capture_output=True, text=True, timeout=60)
    assert done.returncode == 0, done.stdout + done.stderr
