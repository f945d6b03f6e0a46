"""The grid barrier of the persistent step kernel (steps_sync in pliscuda_b200/csrc/engine_kernels.cuh), which a handle
always runs with its default limit: built here into a kernel of its own with a short one.  Barriers that every CTA
reaches let all of them through; where one CTA never comes, the others' waits run out, they leave, the control block
holds PLIS_ERR_TIMEOUT, and the context works on."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include <cstdio>
#include "engine_kernels.cuh"
using namespace plis;

__global__ void k_barriers(StepsRun R, Ctrl* K, int absent, int rounds, int* passed) {
  if ((int)blockIdx.x == absent) return;
  unsigned target = 0;
  for (int i = 0; i < rounds; ++i) {
    if (!steps_sync(R, K, target)) return;
    if (threadIdx.x == 0) passed[blockIdx.x] = i + 1;
  }
}

static int run(int ctas, int threads, int absent, int rounds, unsigned long long limit) {
  unsigned* bar;
  Ctrl* K;
  int* passed;
  cudaMallocManaged(&bar, sizeof *bar);
  cudaMallocManaged(&K, sizeof *K);
  cudaMallocManaged(&passed, ctas * sizeof *passed);
  *bar = 0;
  memset(K, 0, sizeof *K);
  for (int i = 0; i < ctas; ++i) passed[i] = 0;
  StepsRun R{bar, nullptr, limit, 1u};
  void* args[] = {&R, &K, &absent, &rounds, &passed};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_barriers, dim3(ctas), dim3(threads), args, 0, 0);
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return printf("%s\n", cudaGetErrorString(e)), 1;
  for (int i = 0; i < ctas; ++i)
    if (passed[i] != (absent >= 0 ? 0 : rounds)) return printf("CTA %d passed %d barriers\n", i, passed[i]), 2;
  if ((int)K->status != (absent >= 0 ? PLIS_ERR_TIMEOUT : PLIS_OK)) return printf("status %d\n", (int)K->status), 3;
  cudaFree(bar);
  cudaFree(K);
  cudaFree(passed);
  return 0;
}

int main() {
  const int ctas[] = {2, 5, 148, 296}, threads[] = {32, 64, 256};
  for (int c : ctas)
    for (int t : threads) {
      if (int rc = run(c, t, -1, 50, 1ull << 22)) return rc;
      if (int rc = run(c, t, c / 2, 3, 2000)) return rc;
      if (int rc = run(c, t, -1, 50, 1ull << 22)) return rc;
    }
  return 0;
}
"""


def test_waits_run_out_with_a_status(tmp_path):
    from pliscuda_b200 import build
    if not shutil.which(build.NVCC) and not os.path.exists(build.NVCC):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "barrier.cu", tmp_path / "barrier"
    src.write_text(SOURCE)
    subprocess.run([build.NVCC] + build.NVCC_FLAGS + ["-I" + os.path.join(ROOT, "pliscuda_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
