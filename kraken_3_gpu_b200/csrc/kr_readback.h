// kr_readback.h -- large device-to-host reads into a caller's pageable memory.
//
// The driver stages such a copy through one pinned buffer on one thread (about
// 3.5 GB/s into fresh memory, most of it page faults of the destination).
// Here up to kLanes threads each own a pinned buffer: a thread's chunk comes
// over the link while the others write theirs out.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <system_error>
#include <thread>
#include <vector>

namespace kr {

class Readback {
 public:
  static constexpr int kLanes = 4;
  static constexpr size_t kChunk = size_t(4) << 20;

  Readback() = default;
  Readback(const Readback &) = delete;
  Readback &operator=(const Readback &) = delete;
  ~Readback() { release(); }

  void release() {
    for (int i = 0; i < kLanes; i++) {
      if (pin_[i]) cudaFreeHost(pin_[i]);
      if (ev_[i]) cudaEventDestroy(ev_[i]);
      pin_[i] = nullptr;
      ev_[i] = nullptr;
    }
  }

  // `bytes` from device memory to host memory, ordered after the work on
  // `st`; returns when they have arrived.  From two chunks on by threads: a
  // 172 MB observation ring took 49 ms as one copy.  Below, or without pinned
  // memory, the plain copy.
  cudaError_t read(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    return read(static_cast<char *>(dst), bytes, st, kChunk,
                [src](int, size_t off, size_t, cudaStream_t) { return static_cast<const char *>(src) + off; });
  }

  // The same for data that a launch produces: produce(lane, off, n, st)
  // queues the production of bytes off .. off + n on st, into memory that
  // belongs to the lane, and returns where they will be.  chunk: bytes a call
  // may produce at most.
  template <class Produce>
  cudaError_t read(char *dst, size_t bytes, cudaStream_t st, size_t chunk, Produce produce) {
    const size_t n = (bytes + chunk - 1) / chunk;
    if (n < 2 || chunk > kChunk || !prepare()) {
      for (size_t c = 0; c < n; c++) {
        const size_t off = c * chunk, k = std::min(chunk, bytes - off);
        const char *src = produce(0, off, k, st);
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(dst + off, src, k, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
    int dev = 0;
    cudaError_t status[kLanes] = {cudaGetDevice(&dev)};
    if (status[0] != cudaSuccess) return status[0];
    const int lanes = (int)std::min<size_t>(kLanes, n);
    auto run = [&](int lane) {
      cudaError_t e = cudaSetDevice(dev);
      for (size_t c = lane; c < n && e == cudaSuccess; c += lanes) {
        const size_t off = c * chunk, k = std::min(chunk, bytes - off);
        const char *src = produce(lane, off, k, st);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(pin_[lane], src, k, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[lane], st);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev_[lane]);
        if (e == cudaSuccess) std::memcpy(dst + off, pin_[lane], k);
      }
      status[lane] = e;
    };
    std::vector<std::thread> th;
    std::vector<int> here;
    for (int lane = 1; lane < lanes; lane++) {
      status[lane] = cudaSuccess;
      try {
        th.emplace_back(run, lane);
      } catch (const std::system_error &) {
        here.push_back(lane);  // no more threads: this one takes the lane
      }
    }
    run(0);
    for (int lane : here) run(lane);
    for (auto &t : th) t.join();
    for (int lane = 0; lane < lanes; lane++)
      if (status[lane] != cudaSuccess) return status[lane];
    return cudaSuccess;
  }

 private:
  char *pin_[kLanes] = {nullptr};
  cudaEvent_t ev_[kLanes] = {nullptr};

  bool prepare() {
    for (int i = 0; i < kLanes; i++) {
      if (!ev_[i] && cudaEventCreateWithFlags(&ev_[i], cudaEventDisableTiming) != cudaSuccess) ev_[i] = nullptr;
      if (!pin_[i] && cudaMallocHost(reinterpret_cast<void **>(&pin_[i]), kChunk) != cudaSuccess) pin_[i] = nullptr;
      if (!ev_[i] || !pin_[i]) {
        cudaGetLastError();
        release();
        return false;
      }
    }
    return true;
  }
};

}  // namespace kr
