// kr_readback.h -- large device-to-host reads into a caller's pageable memory.
//
// The driver stages such a copy through one pinned buffer on one thread: 20
// GB/s into mapped pages, 2 GB/s into fresh memory, whose page faults take the
// rest.  Here up to kLanes threads each own a pinned chunk: a thread's chunk
// comes over the link while the others write theirs out.  172 MB into fresh
// memory: 85 ms as one copy, 23.5 with 4 chunks of 4 MB, 13 with 8 of 512 KB.
// The chunks are one allocation, since each takes the driver 1 to 3 ms
// whatever its size (four of 4 MB: 14 ms on an engine's first read).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <thread>

namespace kr {

// `device` is the calling thread's current device while this lives
class OnDevice {
 public:
  explicit OnDevice(int device) {
    if (cudaGetDevice(&before_) != cudaSuccess) before_ = device;
    if (before_ != device) cudaSetDevice(device);
    device_ = device;
  }
  ~OnDevice() {
    if (before_ != device_) cudaSetDevice(before_);
  }
  OnDevice(const OnDevice &) = delete;
  OnDevice &operator=(const OnDevice &) = delete;

 private:
  int before_ = 0, device_ = 0;
};

class Readback {
 public:
  int device = 0;  // of the streams and memory it reads from

  static constexpr int kLanes = 8;
  static constexpr size_t kChunk = size_t(512) << 10;
  static constexpr size_t kLeast = size_t(4) << 20;  // smaller reads are plain copies

  Readback() = default;
  Readback(const Readback &) = delete;
  Readback &operator=(const Readback &) = delete;
  ~Readback() { release(); }

  void release() {
    if (pin_) cudaFreeHost(pin_);
    pin_ = nullptr;
    for (cudaEvent_t &ev : ev_) {
      if (ev) cudaEventDestroy(ev);
      ev = nullptr;
    }
  }

  // `bytes` from device memory to host memory, ordered after the work on
  // `st`; returns when they have arrived.  Below kLeast, or without pinned
  // memory, the plain copy.
  cudaError_t read(void *dst, const void *src, size_t bytes, cudaStream_t st) {
    if (bytes < kLeast) {
      const cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
      return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }
    return read(static_cast<char *>(dst), bytes, st, kChunk,
                [src](int, size_t off, size_t, cudaStream_t) { return static_cast<const char *>(src) + off; });
  }

  // The same for data that a launch produces: produce(lane, off, n, st)
  // queues the production of bytes off .. off + n on st, into memory that
  // belongs to the lane, and returns where they will be.  chunk: bytes a call
  // may produce at most.  One read at a time: the lanes' memory is shared.
  template <class Produce>
  cudaError_t read(char *dst, size_t bytes, cudaStream_t st, size_t chunk, Produce produce) {
    std::lock_guard<std::mutex> lock(mu_);
    const OnDevice on(device);  // events and launches need it; copies on a stream do not
    const size_t n = (bytes + chunk - 1) / chunk;
    if (n < 2 || bytes < kLeast || chunk > kChunk || !prepare()) {
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
    cudaError_t status[kLanes] = {};
    // cudaStreamPerThread names another stream in every lane's thread, so the
    // lanes start when the work on the caller's has finished
    if (const cudaError_t e = cudaStreamSynchronize(st); e != cudaSuccess) return e;
    const int lanes = (int)std::min<size_t>(kLanes, n);
    auto run = [&](int lane) {
      cudaError_t e = cudaSetDevice(device);
      for (size_t c = lane; c < n && e == cudaSuccess; c += lanes) {
        const size_t off = c * chunk, k = std::min(chunk, bytes - off);
        const char *src = produce(lane, off, k, st);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(pin_ + lane * kChunk, src, k, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev_[lane], st);
        if (e == cudaSuccess) e = cudaEventSynchronize(ev_[lane]);
        if (e == cudaSuccess) std::memcpy(dst + off, pin_ + lane * kChunk, k);
      }
      status[lane] = e;
    };
    std::thread th[kLanes];
    int started = 1;
    try {
      for (; started < lanes; started++) th[started] = std::thread(run, started);
    } catch (...) {  // no more threads: this one takes the other lanes
    }
    run(0);
    for (int lane = started; lane < lanes; lane++) run(lane);
    for (std::thread &t : th)
      if (t.joinable()) t.join();
    for (int lane = 0; lane < lanes; lane++)
      if (status[lane] != cudaSuccess) return status[lane];
    return cudaSuccess;
  }

 private:
  std::mutex mu_;
  char *pin_ = nullptr;  // kLanes chunks
  cudaEvent_t ev_[kLanes] = {nullptr};

  bool prepare() {
    bool ok = pin_ || cudaMallocHost(reinterpret_cast<void **>(&pin_), kLanes * kChunk) == cudaSuccess;
    if (!ok) pin_ = nullptr;
    for (cudaEvent_t &ev : ev_)
      if (ok && !ev && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
        ev = nullptr;
        ok = false;
      }
    if (!ok) {
      cudaGetLastError();
      release();
    }
    return ok;
  }
};

}  // namespace kr
