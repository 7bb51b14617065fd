"""The block cache behind every call's device memory (csrc/device_memory.h), on the
CPU against a fake of the CUDA runtime calls that it makes."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

FAKE = r"""
#include <cassert>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <thread>
#include "device_memory.h"
using namespace pgsvt;

// ---- a device of kTotal bytes: addresses are numbers, nothing is stored
static const size_t MiB = (size_t)1 << 20, GiB = (size_t)1 << 30;
static size_t kTotal = 64 * GiB, live = 0, next_addr = 1 << 20;
static int mallocs = 0, frees = 0, bad_frees = 0, syncs = 0;
static unsigned long long device_ctx = 7;            // the primary context
static thread_local bool current = false;            // ... is current on this thread
static thread_local cudaError_t last = cudaSuccess;
static std::map<size_t, size_t> held;
static cudaError_t ret(cudaError_t e) { if (e != cudaSuccess) last = e; return e; }
namespace pgsvt { unsigned long long current_context_id() { return current ? device_ctx : 0; } }
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  current = true;
  ++mallocs;
  if (n > kTotal - live) return ret(cudaErrorMemoryAllocation);
  held[next_addr] = n;
  live += n;
  *p = (void*)next_addr;
  next_addr += (n + 511) / 512 * 512;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  current = true;
  if (!p) return cudaSuccess;
  auto it = held.find((size_t)p);
  if (it == held.end()) { ++bad_frees; return ret(cudaErrorInvalidValue); }
  live -= it->second;
  held.erase(it);
  ++frees;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { current = true; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { ++syncs; return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *f = kTotal - live; *t = kTotal; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)

static void call(std::initializer_list<size_t> sizes) {  // the arrays of one call
  DevMem mem;
  for (size_t n : sizes) mem.get(n);
}
"""

CASES = {
    # a repeated call allocates nothing; its arrays are aligned and do not overlap
    "reuse": r"""
  call({100, 3 * MiB, 20 * MiB, 5, 900 * MiB});
  const int m = mallocs;
  call({100, 3 * MiB, 20 * MiB, 5, 900 * MiB});
  CHECK(mallocs == m && frees == 0);
  std::srand(3);
  for (int round = 0; round < 200; ++round) {
    DevMem mem;
    std::map<size_t, size_t> arrays;
    for (int k = 0; k < 30; ++k) {
      const size_t n = (size_t)std::rand() % (1u << (std::rand() % 27)) + (round % 7 ? 1 : 0);
      const size_t p = (size_t)mem.get(n);
      CHECK(p % 256 == 0);
      auto up = arrays.lower_bound(p);
      CHECK(up == arrays.end() || p + n <= up->first);
      CHECK(up == arrays.begin() || std::prev(up)->first + std::prev(up)->second <= p);
      auto b = std::prev(held.upper_bound(p));
      CHECK(p >= b->first && p + n <= b->first + b->second);
      arrays[p] = n;
    }
  }
  block_cache().trim(0);
  CHECK(live == 0 && bad_frees == 0);
""",
    # at most kCacheBytes stay, the blocks longest unused go first
    "eviction": r"""
  for (int k = 0; k < 10; ++k) {
    DevMem mem;
    for (int q = 0; q <= k; ++q) mem.get(1 * GiB + q * MiB);
  }
  call({9 * GiB});
  CHECK(live <= kCacheBytes && live > kCacheBytes - 2 * GiB && block_cache().cached() == live);
  const int m = mallocs;
  call({9 * GiB});
  CHECK(mallocs == m);  // cached after the older ones went
  call({1 * GiB, 1 * GiB, 1 * GiB, 1 * GiB, 1 * GiB, 1 * GiB, 1 * GiB, 3 * GiB, 3 * GiB, 3 * GiB, 3 * GiB});
  CHECK(live <= kCacheBytes && block_cache().cached() == live && bad_frees == 0);
""",
    # an allocation that fails empties the cache and is tried again
    "retry": r"""
  kTotal = 10 * GiB;
  { DevMem a; a.get(4 * GiB); DevMem b; b.get(2 * GiB); }
  CHECK(live == 6 * GiB);
  call({9 * GiB});  // no room beside the cached blocks, no block to reuse
  CHECK(bad_frees == 0 && live <= 9 * GiB);
""",
    # a call that cannot have its memory fails; nothing of it is lost, the next one runs
    "failure": r"""
  kTotal = 10 * GiB;
  for (int k = 0; k < 3; ++k) {
    int code = 0;
    try {
      call({2 * GiB, 3 * GiB, 11 * GiB});
    } catch (const Fail& f) {
      code = f.code;
    }
    CHECK(code == PGSVT_ERR_OOM && syncs == k + 1);  // waited before its blocks were kept
    CHECK(live == block_cache().cached());
    call({2 * GiB, 3 * GiB});
  }
  block_cache().trim(0);
  CHECK(live == 0 && bad_frees == 0);
""",
    # emptied by a thread that has made no CUDA call yet
    "release": r"""
  call({100 * MiB, 7 * MiB});
  CHECK(live > 0);
  std::thread([] { block_cache().trim(0); }).join();
  CHECK(live == 0 && bad_frees == 0 && block_cache().cached() == 0);
  call({100 * MiB, 7 * MiB});  // and used again
  CHECK(live > 0);
""",
    # every call from a new thread: its first array too comes from the cache
    "threads": r"""
  call({30 * MiB, 7 * MiB, 50 * MiB});
  const int m = mallocs;
  for (int k = 0; k < 5; ++k) std::thread([] { call({30 * MiB, 7 * MiB, 50 * MiB}); }).join();
  CHECK(mallocs == m && block_cache().cached() == live);
""",
    # blocks of a context that a device reset destroyed are neither reused nor freed
    "reset": r"""
  call({100 * MiB});
  device_ctx = 8;
  held.clear();
  live = 0;
  const int m = mallocs;
  call({100 * MiB});
  CHECK(mallocs == m + 1 && frees == 0 && bad_frees == 0);
  block_cache().trim(0);
  CHECK(live == 0 && bad_frees == 0);
""",
    # arrays that fit the device one by one, after calls that left larger blocks: the
    # reused blocks take what is missing, so the call starts again without them
    "tight": r"""
  kTotal = 10 * GiB;
  call({3 * GiB, 3 * GiB});
  int tries = 0;
  try {
    call({1600 * MiB, 1600 * MiB, 5 * GiB});
    CHECK(!"fits without a second try");
  } catch (const Fail&) {
    cudaGetLastError();
  }
  with_retry([&] { ++tries; call({1600 * MiB, 1600 * MiB, 5 * GiB}); });
  CHECK(tries == 2 && bad_frees == 0 && cudaGetLastError() == cudaSuccess);
  tries = 0;
  try {
    with_retry([&] { ++tries; call({11 * GiB}); });
  } catch (const Fail& f) {
    CHECK(f.code == PGSVT_ERR_OOM);
  }
  CHECK(tries == 2);
  tries = 0;
  try {  // other failures are not tried again
    with_retry([&] { ++tries; throw Fail(PGSVT_ERR_OOM, "not from an allocation"); });
  } catch (const Fail&) {
  }
  CHECK(tries == 1);
""",
    # little memory left on the device: a finished call keeps nothing
    "scarce": r"""
  kTotal = 10 * GiB;
  call({5 * GiB});
  CHECK(live == 5 * GiB);
  call({9 * GiB});
  CHECK(live == 0 && bad_frees == 0);
""",
}


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("device_memory")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    body = "".join('  if (!std::strcmp(argv[1], "%s")) {%s  return 0; }\n' % kv for kv in CASES.items())
    src = d / "cache.cpp"
    src.write_text(FAKE + "int main(int, char** argv) {\n" + body + "  return 2;\n}\n")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-pthread", "-I", cuda,
                    "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "pgure-svt_gb300", "csrc"), str(src),
                    "-o", str(d / "cache")], check=True)
    return str(d / "cache")


@pytest.mark.parametrize("case", sorted(CASES))
def test_block_cache(program, case):
    r = subprocess.run([program, case], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
