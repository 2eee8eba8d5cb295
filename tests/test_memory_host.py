"""The memory that renders keep between calls (renderx_gb300/csrc/rx_memory.h) on a counterfeit
device of a given size: bounded over any number of contexts, given back when an allocation
finds no memory, on request and with the last context, never held by two renders at once,
and kept by an outer render while a nested one ends."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <random>
#include <thread>
#include "rx_memory.h"
using namespace rx;
#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); exit(1); } } while (0)
static std::mutex g_m;
static std::map<char*, size_t> g_live;
static size_t g_used = 0, g_size = 0, g_mallocs = 0;
static std::atomic<int> g_last{0};
static char* g_next = reinterpret_cast<char*>(1ull << 40);
extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) {
  std::lock_guard<std::mutex> l(g_m);
  if (g_used + n > g_size) { g_last = cudaErrorMemoryAllocation; return cudaErrorMemoryAllocation; }
  g_used += n;
  g_mallocs++;
  *p = g_next;
  g_live[g_next] = n;
  g_next += (n + 511) & ~(size_t)511;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::lock_guard<std::mutex> l(g_m);
  auto i = g_live.find(static_cast<char*>(p));
  CHECK(i != g_live.end());
  g_used -= i->second;
  g_live.erase(i);
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return (cudaError_t)g_last.exchange(0); }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
}
const size_t GB = (size_t)1 << 30, MB = (size_t)1 << 20;
struct Context {
  WorkspaceHold ws;
  Context() { WorkspacePool::of(0).add_context(); }
  ~Context() { WorkspacePool::of(0).drop_context(); }
  cudaError_t render(size_t buffer, int n) {
    WorkspaceHold::Frame frame(ws);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < n && e == cudaSuccess; k++) { WsBuf b; e = b.alloc(ws, buffer); }
    return e;
  }
};
int main() {
  g_size = 64 * GB;
  {  // sixty contexts that render 3 GB each, one after another
    std::vector<std::unique_ptr<Context>> c;
    for (int k = 0; k < 60; k++) {
      c.emplace_back(new Context);
      CHECK(c.back()->render(512 * MB, 6) == cudaSuccess);
      CHECK(g_used <= WorkspacePool::kKeep);
    }
    size_t m = g_mallocs;
    for (auto& i : c) CHECK(i->render(512 * MB, 6) == cudaSuccess);
    CHECK(g_mallocs == m);  // they share what is kept
    DevBuf other, most;       // another allocation of the library gets the memory that is idle
    CHECK(other.alloc(g_size - 4 * GB) == cudaSuccess);
    CHECK(most.alloc(4 * GB) == cudaSuccess && g_used == g_size);
    CHECK(most.alloc(4 * GB + 1) == cudaErrorMemoryAllocation && cudaGetLastError() == cudaSuccess);
    other.release();
    CHECK(g_used == 0);
    // and so does a render whose workspace is not the idle one
    Context a, b;
    WorkspaceHold::Frame fa(a.ws);
    CHECK(b.render(7 * GB, 1) == cudaSuccess && g_used == 7 * GB);
    void* p;
    CHECK(a.ws.alloc(60 * GB, &p) == cudaSuccess && g_used == 60 * GB);
  }
  CHECK(g_used == 0);  // the last context is gone
  {  // at most kKeep stays, of one render or of several at once
    Context a, b, c;
    CHECK(a.render(20 * GB, 1) == cudaSuccess && g_used <= WorkspacePool::kKeep);
    {
      WorkspaceHold::Frame fa(a.ws), fb(b.ws), fc(c.ws);
      void* p;
      for (auto* w : {&a.ws, &b.ws, &c.ws}) CHECK(w->alloc(5 * GB, &p) == cudaSuccess);
      CHECK(g_used == 15 * GB);
    }
    CHECK(g_used <= WorkspacePool::kKeep && g_used > 0);
    WorkspacePool::of(0).drain();
    CHECK(g_used == 0);
    CHECK(a.render(GB, 3) == cudaSuccess && g_used > 0);
    // a nested render gives back its own only, another context's takes other memory
    WorkspaceHold::Frame outer(a.ws);
    char *p, *q, *r;
    CHECK(a.ws.alloc(GB, (void**)&p) == cudaSuccess);
    {
      WorkspaceHold::Frame inner(a.ws);
      CHECK(a.ws.alloc(GB, (void**)&q) == cudaSuccess && (q >= p + GB || p >= q + GB));
      WorkspaceHold::Frame fb(b.ws);
      CHECK(b.ws.alloc(GB, (void**)&r) == cudaSuccess && (r >= p + GB || p >= r + GB) && (r >= q + GB || q >= r + GB));
    }
    CHECK(a.ws.alloc(GB, (void**)&r) == cudaSuccess && r == q);
  }
  CHECK(g_used == 0);
  {  // kept blocks that a larger render takes nothing from are given back wherever they lie
    Context a;
    {
      WorkspaceHold::Frame f(a.ws);
      void* p;
      for (size_t n : {GB, 2 * GB, 4 * GB}) CHECK(a.ws.alloc(n, &p) == cudaSuccess);
      CHECK(g_used == 7 * GB);
    }
    WorkspaceHold::Frame outer(a.ws);
    char *p, *q, *r;
    CHECK(a.ws.alloc(GB, (void**)&p) == cudaSuccess && a.ws.alloc(3 * GB, (void**)&q) == cudaSuccess);
    CHECK(g_used == 7 * GB);  // the blocks of 1 and 4 GB, with the one of 2 GB between them
    {
      WorkspaceHold::Frame inner(a.ws);
      CHECK(a.ws.alloc(g_size - 5 * GB, (void**)&r) == cudaSuccess && g_used == g_size);
    }
    CHECK(a.ws.alloc(g_size - 5 * GB, (void**)&p) == cudaSuccess && p == r && g_used == g_size);
  }
  CHECK(g_used == 0);
  // renders in several threads, too large to be kept and at times for the device: no two hold the same bytes
  g_size = 24 * GB;
  std::mutex held_m;
  std::map<char*, size_t> held;
  std::atomic<int> failed{0};
  std::vector<std::thread> t;
  for (int k = 0; k < 8; k++)
    t.emplace_back([&, k] {
      std::mt19937 rng(k);
      Context c;
      for (int i = 0; i < 400; i++) {
        WorkspaceHold::Frame f(c.ws);
        std::vector<char*> mine;
        for (int j = 0; j < 5; j++) {
          size_t n = rng() % (900 * MB) + 1;
          char* p;
          if (c.ws.alloc(n, (void**)&p) != cudaSuccess) { failed++; break; }
          std::lock_guard<std::mutex> l(held_m);
          auto after = held.lower_bound(p);
          CHECK(after == held.end() || p + n <= after->first);
          if (after != held.begin()) { auto before = std::prev(after); CHECK(before->first + before->second <= p); }
          held[p] = n;
          mine.push_back(p);
        }
        std::lock_guard<std::mutex> l(held_m);
        for (char* p : mine) held.erase(p);
      }
    });
  for (auto& i : t) i.join();
  CHECK(g_used == 0);
  printf("ok %zu %d\n", g_mallocs, failed.load());
}
"""


@pytest.mark.skipif(not os.path.exists("/usr/local/cuda/include/cuda_runtime.h"), reason="no CUDA headers")
def test_kept_memory_is_bounded_and_given_back(tmp_path):
    src, exe = tmp_path / "memory.cpp", tmp_path / "memory"
    src.write_text(SOURCE)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-O1", "-g", "-pthread", "-I", "/usr/local/cuda/include",
                    "-I", os.path.join(ROOT, "renderx_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
