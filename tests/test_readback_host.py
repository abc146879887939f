"""csrc/kr_readback.h over a fake of the CUDA runtime: which thread, stream and
device its copies run on, which a GPU alone would show only now and then.  The
fake's streams run nothing until they are waited for; cudaStreamPerThread names
another stream in every thread; an event can only be recorded on a stream of
the device that was current when it was made, and a launch needs its stream's
device current."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "kraken_3_gpu_b200", "csrc")
CUDA_INCLUDE = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")

FAKE = r'''
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <vector>
#include "kr_readback.h"

struct Queue {
  std::mutex mu;
  std::deque<std::function<void()>> ops;
  int device = 0;
  void drain() {
    std::lock_guard<std::mutex> l(mu);
    while (!ops.empty()) { ops.front()(); ops.pop_front(); }
  }
  void add(std::function<void()> f) {
    std::lock_guard<std::mutex> l(mu);
    ops.push_back(std::move(f));
  }
};
static thread_local int t_device = 0;
static Queue &per_thread() {
  static std::mutex mu;
  static std::map<std::thread::id, Queue *> all;  // a thread's stream outlives it
  std::lock_guard<std::mutex> l(mu);
  Queue *&q = all[std::this_thread::get_id()];
  if (!q) { q = new Queue; q->device = t_device; }
  return *q;
}
static Queue &of(cudaStream_t st) { return st == cudaStreamPerThread ? per_thread() : *reinterpret_cast<Queue *>(st); }
struct Event { int device; Queue *on = nullptr; };

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = t_device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { t_device = d; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) { *p = std::malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(new Event{t_device}); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event *>(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
  Event &ev = *reinterpret_cast<Event *>(e);
  if (ev.device != of(st).device) return cudaErrorInvalidResourceHandle;
  ev.on = &of(st);
  return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { reinterpret_cast<Event *>(e)->on->drain(); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { of(st).drain(); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  of(st).add([=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
}
'''


def _run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text(FAKE + body)
    exe = tmp_path / "t"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-pthread", "-I", CSRC, "-I", CUDA_INCLUDE, "-o",
                    str(exe), str(src)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.startswith("ok"), out.stdout + out.stderr


def test_reads_follow_the_work_on_a_per_thread_stream(tmp_path):
    """An engine on cudaStreamPerThread: its work is queued on the caller's
    stream, the readback's threads have streams of their own, and what they
    read must be what that work left."""
    _run(tmp_path, r'''
int main() {
  std::vector<char> src(size_t(9) << 20, 0), dst(src.size(), 1);
  for (int turn = 1; turn < 4; turn++) {
    kr::Readback rb;
    of(cudaStreamPerThread).add([&] { std::memset(src.data(), 6 + turn, src.size()); });
    if (rb.read(dst.data(), src.data(), src.size(), cudaStreamPerThread) != cudaSuccess) { std::printf("FAIL read\n"); return 1; }
    for (size_t i = 0; i < dst.size(); i++)
      if (dst[i] != 6 + turn) { std::printf("FAIL turn %d byte %zu: %d\n", turn, i, dst[i]); return 1; }
  }
  std::printf("ok\n");
  return 0;
}
''')


def test_reads_need_no_current_device(tmp_path):
    """An engine on device 1, read by threads whose current device is 0: every
    call that depends on the current device is made under the engine's, and
    the caller's is as it was afterwards."""
    _run(tmp_path, r'''
int main() {
  Queue q1;
  q1.device = 1;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(&q1);
  std::vector<char> src(size_t(9) << 20), dst(src.size());
  for (size_t i = 0; i < src.size(); i++) src[i] = (char)(i * 31);
  kr::Readback rb;
  rb.device = 1;
  bool wrong = false;
  auto reader = [&] {
    if (rb.read(dst.data(), src.data(), src.size(), st) != cudaSuccess || dst != src) wrong = true;
    for (size_t bytes : {size_t(1000), src.size()}) {
      std::fill(dst.begin(), dst.end(), 0);
      const cudaError_t e = rb.read(dst.data(), bytes, st, kr::Readback::kChunk,
                                    [&](int, size_t off, size_t, cudaStream_t s) {
                                      if (t_device != of(s).device) wrong = true;
                                      return (const char *)src.data() + off;
                                    });
      if (e != cudaSuccess || std::memcmp(dst.data(), src.data(), bytes)) wrong = true;
    }
    if (t_device != 0) wrong = true;
  };
  reader();
  std::thread(reader).join();
  std::printf(wrong ? "FAIL\n" : "ok\n");
  return wrong;
}
''')
