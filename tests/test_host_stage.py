"""Transfers through pinned slices (pliscuda_b200/csrc/host_stage.h), host code compiled here against a stand-in for the
CUDA runtime: rows arrive whole at every size around a slice's, with one worker and with several; and where the pinned
memory or an event cannot be had, the copies go through the driver and no error is left behind."""
import os
import shutil
import subprocess

import pytest

from helpers import ROOT

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include "host_stage.h"

static int fail_malloc = 0, fail_event = -1, events = 0, live_events = 0, live_bufs = 0, driver = 0;
static cudaError_t last = cudaSuccess;
static std::mutex mu;
static cudaError_t fail() { return last = cudaErrorMemoryAllocation; }
extern "C" {
cudaError_t cudaMallocHost(void** p, size_t n) { if (fail_malloc) return fail(); ++live_bufs; *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { --live_bufs; std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  if (events++ == fail_event) return fail();
  ++live_events;
  *e = (cudaEvent_t)&events;
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { --live_events; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return e ? cudaSuccess : cudaErrorInvalidResourceHandle; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
  std::lock_guard<std::mutex> lock(mu);
  ++driver;
  for (size_t i = 0; i < h; ++i) std::memcpy((char*)d + i * dp, (const char*)s + i * sp, w);
  return cudaSuccess;
}
}

static int round_trip(plis::HostStage& st, size_t bytes, size_t rows) {
  const size_t pitch = (bytes + 127) / 128 * 128 + 128;
  std::vector<unsigned char> host(bytes * rows), dev(pitch * rows, 0xAB), back(bytes * rows);
  for (size_t i = 0; i < host.size(); ++i) host[i] = (unsigned char)(i * 2654435761u >> 13);
  if (st.upload(dev.data(), pitch, host.data(), bytes, bytes, rows, nullptr) != cudaSuccess) return 1;
  for (size_t r = 0; r < rows; ++r) {
    if (std::memcmp(&dev[r * pitch], &host[r * bytes], bytes)) return 2;
    for (size_t i = bytes; i < pitch; ++i)
      if (dev[r * pitch + i] != 0xAB) return 3;  // the padding of a row is not touched
  }
  if (st.download(back.data(), bytes, dev.data(), pitch, bytes, rows, nullptr) != cudaSuccess) return 4;
  return std::memcmp(back.data(), host.data(), host.size()) ? 5 : 0;
}

int main(int argc, char** argv) {
  const size_t bytes = std::strtoull(argv[1], nullptr, 10), rows = std::strtoull(argv[2], nullptr, 10);
  fail_malloc = std::atoi(argv[3]);
  fail_event = std::atoi(argv[4]);
  const bool ok = !fail_malloc && (fail_event < 0 || fail_event >= 8);
  {
    plis::HostStage st;
    st.init(0, bytes);
    if (st.on() != ok) return 10;
    if (last != cudaSuccess) return 11;
    if (!ok && (live_bufs || live_events)) return 12;
    const int rc = round_trip(st, bytes, rows);
    if (rc) return rc;
    if ((driver > 0) == ok) return 13;
  }
  return live_bufs || live_events ? 14 : 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    from pliscuda_b200 import build
    cxx = shutil.which(os.environ.get("CXX", "g++"))
    if not cxx or not os.path.exists(os.path.join(build.CUDA_HOME, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("stage")
    src = d / "stage.cpp"
    src.write_text(SOURCE)
    exe = d / "stage"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "pliscuda_b200", "csrc"),
                    "-I" + os.path.join(build.CUDA_HOME, "include"), str(src), "-o", str(exe)], check=True)
    return str(exe)


MB = 1 << 20


@pytest.mark.parametrize("size,rows", [(4, 1), (4, 5), (4096, 3), (4100, 7), (MB // 2 - 4, 2), (MB // 2, 1), (MB // 2 + 4, 3),
                                       (MB // 2 + 4, 4), (4 * MB - 4, 1), (4 * MB, 1), (5 * MB + 12, 3)])
@pytest.mark.parametrize("fail", [(0, -1), (1, -1), (0, 0), (0, 7)], ids=["pinned", "no_memory", "no_event", "no_last_event"])
def test_round_trip(program, size, rows, fail):
    r = subprocess.run([program, str(size), str(rows), str(fail[0]), str(fail[1])], timeout=120)
    assert r.returncode == 0, r.returncode
