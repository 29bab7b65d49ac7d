"""The cache of device blocks (agdeblend_b200/csrc/device_pool.hpp), compiled for
the host against the CUDA headers and a fake of the runtime calls it makes
(addresses count up, each remembers its device): a block goes back to the
device it was allocated on; a table does not take the block of a large array;
a block that an exception releases is freed (cudaFree waits for the device)."""
import os
import shutil
import subprocess

import pytest

from agdeblend_b200 import build
from conftest import ROOT

FAKE = r"""
#include <cstdint>
#include <cstdlib>
#include <map>
#include "device_pool.hpp"

static int g_dev = 0, g_frees = 0;
static uintptr_t g_next = 1 << 20;
static std::map<void *, int> g_owner;
extern "C" {
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { g_dev = d; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *f = *t = size_t(1) << 30;
  return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
  *p = reinterpret_cast<void *>(g_next);
  g_next += n;
  g_owner[*p] = g_dev;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  g_frees += (int)g_owner.erase(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *, const void *, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
}
namespace agd {
bool injected_alloc_failure() { return false; }
}
using agd::DevArray;

static int device_of_a_block() {
  {  // made on device 0, released while device 1 is current
    DevArray<char> a;
    a.alloc(100000);
    g_dev = 1;
  }
  {
    DevArray<char> b;
    b.alloc(100000);
    if (g_owner.at(b.get()) != 1) return 1;
    g_dev = 0;
    DevArray<char> c;
    c.alloc(100000);
    if (g_owner.at(c.get()) != 0) return 2;
  }
  agd::DevicePool::release_all();
  return g_frees == 2 && g_dev == 0 ? 0 : 3;
}

static int large_blocks_are_left_to_large_arrays() {
  DevArray<char> big;
  big.alloc(1 << 20);
  void *block = big.get();
  big.release();
  DevArray<char> table, again;
  table.alloc(512);
  if (table.get() == block) return 1;
  again.alloc(900000);
  return again.get() == block ? 0 : 2;
}

static int exceptions_free_their_blocks() {
  try {
    DevArray<char> tmp;
    tmp.alloc(3000000);
    throw 1;
  } catch (int) {
  }
  return g_frees == 1 ? 0 : 1;
}

int main(int, char **argv) {
  int (*const cases[])() = {device_of_a_block, large_blocks_are_left_to_large_arrays, exceptions_free_their_blocks};
  return cases[std::atoi(argv[1])]();
}
"""
CASES = ["device_of_a_block",
         "large_blocks_are_left_to_large_arrays",
         "exceptions_free_their_blocks"]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    cxx = shutil.which("g++")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc()))),
                        "include")
    if cxx is None or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("no host compiler or CUDA headers")
    where = tmp_path_factory.mktemp("pool")
    src, exe = where / "pool.cpp", where / "pool"
    src.write_text(FAKE)
    subprocess.run([cxx, "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "agdeblend_b200", "csrc"), "-I", cuda, str(src), "-o",
                    str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("case", CASES)
def test_device_pool(program, case):
    env = {k: v for k, v in os.environ.items() if k != "AGD_GPU_CACHE"}
    assert subprocess.run([program, str(CASES.index(case))], env=env).returncode == 0
