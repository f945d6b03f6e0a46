// host_stage.h — copies between pageable host memory and the device through a handle's own pinned slices.
//
// A copy from pageable memory goes through the driver's staging on the calling thread, 4-5 GB/s on the
// measured host for states of tens of megabytes.  Here the bytes pass through pinned slices that belong
// to the handle (kSlices x 512 KB, freed with it), with kWorkers threads, each alternating between its
// own slices so that its memcpy overlaps its DMA (pages of a fresh result array are then touched by
// several threads too).  The slices are an optimisation: where they cannot be had, the copies go through
// the driver.
#ifndef PLIS_HOST_STAGE_H_
#define PLIS_HOST_STAGE_H_

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

namespace plis {

inline cudaMemoryType host_memory(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return cudaMemoryTypeUnregistered;
  }
  return a.type;
}
// true when the caller's buffer is pinned already: a plain asynchronous copy runs at DMA speed
inline bool host_pinned(const void* p) { return host_memory(p) == cudaMemoryTypeHost; }
// true for a buffer the CUDA runtime does not know
inline bool host_pageable(const void* p) { return host_memory(p) == cudaMemoryTypeUnregistered; }

// Runs f(0) .. f(n - 1), on threads of their own but for the first; inline where a thread cannot be had.
template <class F>
inline void run_workers(int n, F f) {
  std::vector<std::thread> t;
  std::vector<int> mine;
  for (int w = 1; w < n; ++w) {
    try {
      t.emplace_back(f, w);
    } catch (...) {
      mine.push_back(w);
    }
  }
  f(0);
  for (int w : mine) f(w);
  for (auto& x : t) x.join();
}

// every count below 2^30
inline bool counts_in_range(const uint32_t* c, size_t n) {
  constexpr size_t kPart = size_t(1) << 20;
  const int workers = (int)std::min<size_t>(4, 1 + n / kPart / 2);
  std::vector<uint32_t> any(workers, 0);
  run_workers(workers, [&](int w) {
    const size_t a = n * (size_t)w / workers, b = n * (size_t)(w + 1) / workers;
    uint32_t m = 0;
    for (size_t i = a; i < b; ++i) m |= c[i];
    any[w] = m;
  });
  uint32_t m = 0;
  for (uint32_t v : any) m |= v;
  return m < (1u << 30);
}

class HostStage {
 public:
  static constexpr int kSlices = 8, kWorkers = 4;
  ~HostStage() { release(); }

  // slices for pieces of up to `piece` bytes (a piece above 512 KB passes in parts)
  void init(int device, size_t piece) {
    device_ = device;
    slice_ = std::min<size_t>(size_t(512) << 10, (piece + 4095) / 4096 * 4096);
    if (slice_ == 0) slice_ = 4096;
    cudaError_t e = cudaMallocHost((void**)&buf_, slice_ * kSlices);
    if (e != cudaSuccess) buf_ = nullptr;
    for (auto& v : ev_)
      if (e == cudaSuccess && (e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming)) != cudaSuccess) v = nullptr;
    if (e != cudaSuccess) {
      release();
      cudaGetLastError();  // not the error of a later launch
    }
  }
  bool on() const { return buf_ != nullptr; }
  void release() {
    if (buf_) {
      for (auto& v : ev_)
        if (v) cudaEventSynchronize(v);
      cudaFreeHost(buf_);
    }
    buf_ = nullptr;
    for (auto& v : ev_)
      if (v) { cudaEventDestroy(v); v = nullptr; }
  }

  // `rows` rows of `bytes` each; dpitch / hpitch: distance of two rows on the device / host.  An upload
  // returns with the host buffer free and the copies enqueued on s; a download returns with the data.
  cudaError_t upload(void* dev, size_t dpitch, const void* host, size_t hpitch, size_t bytes, size_t rows, cudaStream_t s) {
    if (!on()) {
      const cudaError_t e = cudaMemcpy2DAsync(dev, dpitch, host, hpitch, bytes, rows, cudaMemcpyHostToDevice, s);
      return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    }
    return copy(true, (char*)dev, dpitch, (char*)const_cast<void*>(host), hpitch, bytes, rows, s);
  }
  cudaError_t download(void* host, size_t hpitch, const void* dev, size_t dpitch, size_t bytes, size_t rows, cudaStream_t s) {
    if (!on()) {
      const cudaError_t e = cudaMemcpy2DAsync(host, hpitch, dev, dpitch, bytes, rows, cudaMemcpyDeviceToHost, s);
      return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    }
    return copy(false, (char*)const_cast<void*>(dev), dpitch, (char*)host, hpitch, bytes, rows, s);
  }

 private:
  cudaError_t copy(bool up, char* dev, size_t dp, char* host, size_t hp, size_t bytes, size_t rows, cudaStream_t s) {
    const size_t parts = (bytes + slice_ - 1) / slice_, n = parts * rows;
    constexpr int workers = kWorkers, per = kSlices / workers;
    cudaError_t err[kWorkers] = {};
    // worker w moves parts w, w + workers, ... through its slices w * per .. + per - 1 in turn
    auto run = [&](int w) {
      cudaError_t e = cudaSetDevice(device_);
      size_t done = 0;  // downloads: parts of this worker taken out of its slices
      auto place = [&](size_t j, char*& d, char*& h, size_t& len) {
        const size_t i = w + j * workers, row = i / parts, off = i % parts * slice_;
        d = dev + row * dp + off;
        h = host + row * hp + off;
        len = std::min(slice_, bytes - off);
      };
      auto take = [&]() {
        char *d, *h;
        size_t len;
        place(done, d, h, len);
        const int k = w * per + (int)(done % per);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev_[k]);
        if (e == cudaSuccess) std::memcpy(h, buf_ + k * slice_, len);
        ++done;
      };
      size_t j = 0;
      for (; w + j * workers < n && e == cudaSuccess; ++j) {
        char *d, *h;
        size_t len;
        place(j, d, h, len);
        if (!up && j >= (size_t)per) take();
        const int k = w * per + (int)(j % per);
        char* b = buf_ + k * slice_;
        if (e == cudaSuccess) e = cudaEventSynchronize(ev_[k]);  // the slice's last copy
        if (e != cudaSuccess) break;
        if (up) std::memcpy(b, h, len);
        e = cudaMemcpyAsync(up ? d : b, up ? b : d, len, up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[k], s);
      }
      while (!up && done < j) take();
      err[w] = e;
    };
    run_workers(workers, run);
    for (cudaError_t e : err)
      if (e != cudaSuccess) return e;
    return cudaSuccess;
  }

  int device_ = 0;
  size_t slice_ = 0;
  char* buf_ = nullptr;
  cudaEvent_t ev_[kSlices] = {};
};

}  // namespace plis

#endif
