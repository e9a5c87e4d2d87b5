"""The device-memory pool of a context (dev_pool.h) compiled against a stand-in
allocator of fixed capacity: ranges join, blocks that hold nothing go back, and a
larger deck loads after a smaller one wherever it alone would fit."""
import os
import subprocess

from conftest import PKG

STUB = r"""
#pragma once
#include <cstddef>
#include <map>
using cudaError_t = int;
using cudaStream_t = struct CUstream_st*;
constexpr int cudaSuccess = 0, cudaErrorMemoryAllocation = 2;
#define cudaStreamLegacy ((cudaStream_t)1)
extern size_t g_capacity, g_used;
extern std::map<char*, size_t> g_live;
inline cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_used + n > g_capacity) return cudaErrorMemoryAllocation;
  static char* next = (char*)0x10000000000;
  *p = next;
  g_live[next] = n;
  next += (n + 4095) / 4096 * 4096;
  g_used += n;
  return 0;
}
inline cudaError_t cudaFree(void* p) {
  g_used -= g_live.at((char*)p);
  g_live.erase((char*)p);
  return 0;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return 0; }
inline cudaError_t cudaGetLastError() { return 0; }
"""

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "dev_pool.h"
size_t g_capacity = 0, g_used = 0;
std::map<char*, size_t> g_live;
constexpr size_t MB = size_t(1) << 20, GB = size_t(1) << 30;
#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::exit(1); } } while (0)
std::vector<size_t> deck(double gb) {  // a few large buffers, many small ones
  std::vector<size_t> v;
  for (double f : {0.30, 0.15, 0.15, 0.08, 0.08, 0.05, 0.05, 0.04, 0.03, 0.02, 0.02, 0.01, 0.01})
    v.push_back((size_t)(f * gb * GB));
  for (int k = 0; k < 80; k++) v.push_back((size_t)(k % 7 + 1) * 100000);
  return v;
}
using cfd::DevPool;
std::vector<void*> load(DevPool& p, const std::vector<size_t>& d) {
  std::vector<void*> b(d.size());
  for (size_t k = 0; k < d.size(); k++) CHECK(p.get(d[k], &b[k]) == 0);
  return b;
}
int main() {
  g_capacity = 100 * GB;
  {  // one deck after another, as a context loads them
    DevPool p;
    for (double gb : {1.0, 60.0, 70.0, 95.0, 2.0, 95.0}) {
      auto b = load(p, deck(gb));
      CHECK(g_used == p.held() && p.held() <= (size_t)(1.02 * gb * GB) + 512 * MB);
      // no two live ranges overlap
      std::map<char*, size_t> r;
      auto d = deck(gb);
      for (size_t k = 0; k < b.size(); k++) r[(char*)b[k]] = d[k];
      char* end = nullptr;
      for (auto& [q, n] : r) { CHECK(q >= end); end = q + n; }
      for (size_t k = 0; k < b.size(); k++) p.put(b[(k * 37 + 5) % b.size()]);
      p.trim();
      CHECK(p.held() == 0 && g_used == 0);
    }
  }
  CHECK(g_live.empty());
  {  // a large buffer replaced by a larger one that needs the first one's memory
    DevPool p;
    void *a, *b, *c;
    CHECK(p.get(30 * GB, &a) == 0 && p.get(30 * GB, &b) == 0);
    p.put(a);
    CHECK(p.get(60 * GB, &c) == 0);
    p.put(b);
    CHECK(p.get(101 * GB, &a) == cudaErrorMemoryAllocation);
    CHECK(g_used == 60 * GB);
  }
  {  // neighbouring ranges join, whatever the order they come back in
    DevPool p;
    void* v[8];
    for (auto& q : v) CHECK(p.get(2 * MB, &q) == 0);
    const size_t held = p.held();
    for (int k : {3, 1, 2, 5, 4}) p.put(v[k]);
    void* w;
    CHECK(p.get(10 * MB, &w) == 0 && w == v[1] && p.held() == held);
  }
  std::puts("ok");
}
"""


def test_pool_bookkeeping(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(STUB)
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "pool"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-fsanitize=undefined", "-fno-sanitize-recover", "-I",
                        str(tmp_path), "-I", os.path.join(PKG, "csrc"), str(tmp_path / "main.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
