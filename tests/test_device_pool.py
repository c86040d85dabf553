"""The allocation behind every device buffer (csrc/pool.cu), built for the host
against a fake runtime: a device of 100 bytes whose pools keep what is freed, as
the driver does (a block counts as free once its stream has been synchronised
after the free, and goes back to the device when the pool is trimmed)."""
import os
import shutil
import subprocess

import pytest

from getdp_gb300 import build as B

FAKE = r"""
#include "pool.h"
#include <cstdio>
#include <cstdint>
#include <map>
#include <vector>
using namespace gb;

static size_t device_free = 100;
static cudaError_t last = cudaSuccess;
struct Block { size_t n; cudaStream_t stream; bool pending; };
struct FakePool { std::vector<Block> idle; bool open = true; };
struct Alloc { size_t n; FakePool *pool; };
static std::map<void *, Alloc> live;
static uintptr_t next_p = 4096;

static cudaError_t fail(cudaError_t e) { return last = e; }
static void *put(size_t n, FakePool *p)
{
  void *q = (void *)(next_p += 4096);
  live[q] = {n, p};
  return q;
}
extern "C" {
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n)
{
  if(n > device_free) return fail(cudaErrorMemoryAllocation);
  device_free -= n;
  *p = put(n, nullptr);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *)
{
  *p = (cudaMemPool_t) new FakePool;
  return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { ((FakePool *)p)->open = false; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
static std::vector<FakePool *> all;
cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
  for(FakePool *p : all)
    for(Block &b : p->idle)
      if(b.stream == s) b.pending = false;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t q, size_t)
{
  FakePool *p = (FakePool *)q;
  std::vector<Block> keep;
  for(Block &b : p->idle)
    if(b.pending)
      keep.push_back(b);
    else
      device_free += b.n;
  p->idle = keep;
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **q, size_t n, cudaMemPool_t m, cudaStream_t)
{
  FakePool *p = (FakePool *)m;
  for(size_t i = 0; i < p->idle.size(); i++)
    if(p->idle[i].n == n) {  // (another size does not fit: fragments)
      p->idle.erase(p->idle.begin() + i);
      *q = put(n, p);
      return cudaSuccess;
    }
  if(n > device_free) return fail(cudaErrorMemoryAllocation);
  device_free -= n;
  *q = put(n, p);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *q, cudaStream_t s)
{
  Alloc a = live[q];
  live.erase(q);
  a.pool->idle.push_back({a.n, s, true});
  return cudaSuccess;
}
}
#define CHECK(x) do { if(!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while(0)

int main()
{
  cudaStream_t s1 = (cudaStream_t)0x10, s2 = (cudaStream_t)0x20, from = nullptr;
  MemPool m1, m2, other;
  pool_open(&m1, 0, s1);
  pool_open(&m2, 0, s2);
  pool_open(&other, 1, (cudaStream_t)0x30);  // another device: left alone
  all = {(FakePool *)m1.pool, (FakePool *)m2.pool, (FakePool *)other.pool};
  ((FakePool *)other.pool)->idle.push_back({7, (cudaStream_t)0x30, false});
  void *a, *b, *c, *d;
  // without a pool in force: cudaMalloc, to be freed by cudaFree
  CHECK(device_alloc(&a, 10, &from) == cudaSuccess && !from && !live[a].pool);
  // scratch of two contexts, given back to their pools
  t_pool = &m1;
  CHECK(device_alloc(&b, 50, &from) == cudaSuccess && from == s1);
  t_pool = &m2;
  CHECK(device_alloc(&c, 30, &from) == cudaSuccess && from == s2);
  cudaFreeAsync(b, s1);
  cudaFreeAsync(c, s2);
  CHECK(device_free == 10);
  // a buffer outside any pool takes what both hold
  t_pool = nullptr;
  CHECK(device_alloc(&d, 80, &from) == cudaSuccess && !from && device_free == 10);
  CHECK(last == cudaSuccess);
  // so does an explicit device allocation, and one context's scratch takes another's
  device_free += live[d].n;
  live.erase(d);
  t_pool = &m1;
  CHECK(device_alloc(&b, 85, &from) == cudaSuccess);
  cudaFreeAsync(b, s1);
  CHECK(device_malloc(&d, 20) == cudaSuccess && !live[d].pool);
  CHECK(device_alloc(&b, 60, &from) == cudaSuccess);
  cudaFreeAsync(b, s1);
  t_pool = &m2;
  CHECK(device_alloc(&c, 55, &from) == cudaSuccess && from == s2);
  // what does not fit is refused and leaves no error behind
  t_pool = nullptr;
  CHECK(device_alloc(&b, 500, &from) == cudaErrorMemoryAllocation && last == cudaSuccess);
  t_pool = &m1;
  CHECK(device_alloc(&b, 500, &from) == cudaErrorMemoryAllocation && last == cudaSuccess && !from);
  // a closed pool is not touched any more, and its context falls back to cudaMalloc
  cudaFreeAsync(c, s2);
  pool_close(&m2);
  CHECK(!all[1]->open);
  t_pool = &m2;
  CHECK(device_alloc(&b, 5, &from) == cudaSuccess && !from);
  CHECK(device_alloc(&b, 500, &from) == cudaErrorMemoryAllocation);
  CHECK(all[1]->idle.size() == 1 && all[2]->idle.size() == 1);
  // the lock keeps give-back and captures apart
  auto held = hold_capture();
  CHECK(held.owns_lock());
  held.unlock();
  printf("ok\n");
  return 0;
}
"""


def test_memory_held_by_pools_is_given_back(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no g++")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(B.nvcc()))), "include")
    src = tmp_path / "fake.cpp"
    src.write_text(FAKE)
    exe = tmp_path / "fake"
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", inc, "-I", B.CSRC, str(src), "-x", "c++",
                    os.path.join(B.CSRC, "pool.cu"), "-o", str(exe), "-pthread"], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_every_device_buffer_goes_through_it():
    """No other file allocates device memory or begins a capture unheld."""
    for f in os.listdir(B.CSRC):
        if not f.endswith((".cu", ".cuh", ".h")) or f.startswith("pool."):
            continue
        text = open(os.path.join(B.CSRC, f)).read()
        for call in ("cudaMalloc(", "cudaMallocAsync(", "cudaMallocFromPoolAsync("):
            assert call not in text, (f, call)
        assert text.count("cudaStreamBeginCapture(") == text.count("= hold_capture();"), f
