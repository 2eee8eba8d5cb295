"""The mbarrier wait of the tensor-core kernels (mbar_wait in renderx_gb300/csrc/rx_tc.cuh) is
bounded by time: on a barrier that nothing arrives at it gives up after its limit, the
kernel ends and the context stays usable; on one that completes it reports so."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
LIMIT_NS = 50_000_000
SOURCE = r"""
#include <cstdio>
#include "rx_tc.cuh"
namespace tc = rx::tc;
__global__ void k_wait(int* out, unsigned long long* ns) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar, 1);
    tc::fence_mbar_init();
  }
  __syncthreads();
  const uint64_t t0 = tc::now_ns();
  const bool early = tc::mbar_wait(&bar, 0, LIMIT_NS);  // nothing arrives
  const uint64_t t1 = tc::now_ns();
  __syncthreads();
  if (threadIdx.x == 0) tc::mbar_expect_tx(&bar, 0);  // the one arrival
  const bool late = tc::mbar_wait(&bar, 0);
  out[threadIdx.x] = (early ? 2 : 0) | (late ? 1 : 0);
  ns[threadIdx.x] = t1 - t0;
}
int main() {
  int *d, h[128];
  unsigned long long *dn, hn[128], lo = ~0ull, hi = 0;
  cudaMalloc(&d, sizeof h);
  cudaMalloc(&dn, sizeof hn);
  k_wait<<<1, 128>>>(d, dn);
  if (cudaDeviceSynchronize() != cudaSuccess) return 1;
  cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost);
  cudaMemcpy(hn, dn, sizeof hn, cudaMemcpyDeviceToHost);
  for (int k = 0; k < 128; k++) {
    if (h[k] != 1) return 2;
    if (hn[k] < lo) lo = hn[k];
    if (hn[k] > hi) hi = hn[k];
  }
  printf("%llu %llu\n", lo, hi);
  return 0;
}
"""


def test_wait_gives_up_after_its_limit(tmp_path):
    src, exe = tmp_path / "wait.cu", tmp_path / "wait"
    src.write_text(SOURCE)
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_103a,code=sm_103a", f"-DLIMIT_NS={LIMIT_NS}",
                    "-I", os.path.join(ROOT, "renderx_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    lo, hi = map(int, r.stdout.split())
    # not before the limit; past it by at most the try that was under way (a second allows any
    # hardware limit of a try that is no longer than the default limit of the wait itself)
    assert LIMIT_NS <= lo and hi < LIMIT_NS + 1_000_000_000, (lo, hi)
