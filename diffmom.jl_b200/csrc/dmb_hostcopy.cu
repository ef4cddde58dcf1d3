// dmb_hostcopy.cu -- large results to the caller's (pageable) host memory.
//
// cudaMemcpy to pageable memory runs at 5 GB/s here: one thread copies out of
// the driver's bounce buffer and takes the page faults of freshly allocated
// memory (53 MB of impedance matrix: 11.2 of a call's 12 ms).  Results above
// HC_MIN bytes instead go through pinned chunks of the context's own, one per
// worker: each worker copies its chunk from the device on a stream of its own
// and from there to the destination, so the transfers of some overlap the
// copies and faults of others.
#include <algorithm>
#include <atomic>
#include <thread>
#include <vector>

#include "dmb_device.cuh"
#include "dmb_internal.h"

namespace {

constexpr int HC_WORKERS = 8;
constexpr size_t HC_CHUNK = (size_t)1 << 20;  // bytes of destination per chunk
constexpr size_t HC_MIN = (size_t)2 << 20;

__global__ void k_widen(int64_t count, const float2 *__restrict__ a, double2 *__restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) b[i] = make_double2(a[i].x, a[i].y);
}

}  // namespace

struct HostCopy {
  cudaStream_t stream[HC_WORKERS] = {};
  void *pin[HC_WORKERS] = {};
  void *dev[HC_WORKERS] = {};
  cudaEvent_t ready = nullptr;
  int workers = 0;  // with a stream and both chunks
};

namespace dmb {

void hostcopy_release(dmb_ctx *c) {
  if (!c->hostcopy) return;
  HostCopy &h = *c->hostcopy;
  for (int w = 0; w < HC_WORKERS; w++) {
    if (h.stream[w]) cudaStreamDestroy(h.stream[w]);
    if (h.pin[w]) cudaFreeHost(h.pin[w]);
    if (h.dev[w]) cudaFree(h.dev[w]);
  }
  if (h.ready) cudaEventDestroy(h.ready);
  delete c->hostcopy;
  c->hostcopy = nullptr;
}

// dst (complex128, host) <- src (device, complex64 when widen) after the work
// issued on the context's stream; returns when dst is written
void copy_out(dmb_ctx *c, void *dst, const void *src, int64_t count, bool widen) {
  const size_t bytes = sizeof(double2) * (size_t)count;
  if (!c->hostcopy && bytes >= HC_MIN) {
    c->hostcopy = new HostCopy();
    HostCopy &h = *c->hostcopy;
    bool ok = cudaEventCreateWithFlags(&h.ready, cudaEventDisableTiming) == cudaSuccess;
    for (int w = 0; ok && w < HC_WORKERS; w++) {
      ok = cudaStreamCreateWithFlags(&h.stream[w], cudaStreamNonBlocking) == cudaSuccess &&
           cudaHostAlloc(&h.pin[w], HC_CHUNK, cudaHostAllocDefault) == cudaSuccess &&
           cudaMalloc(&h.dev[w], HC_CHUNK) == cudaSuccess;
      if (ok) h.workers = w + 1;
    }
    if (!ok) (void)cudaGetLastError();
  }
  if (bytes < HC_MIN || c->hostcopy->workers == 0) {
    if (widen) {
      c->d_io[0].ensure(bytes);
      DMB_LAUNCH(c, k_widen, (unsigned)((count + 255) / 256), 256, 0, count, (const float2 *)src,
                 c->d_io[0].as<double2>());
      src = c->d_io[0].p;
    }
    DMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
    DMB_CUDA(cudaStreamSynchronize(c->stream));
    return;
  }
  HostCopy &h = *c->hostcopy;
  DMB_CUDA(cudaEventRecord(h.ready, c->stream));
  const int64_t per = HC_CHUNK / sizeof(double2), chunks = (count + per - 1) / per;
  std::atomic<int64_t> next{0};
  std::atomic<int> bad{(int)cudaSuccess};
  auto work = [&](int w) {
    auto check = [&](cudaError_t e) {
      if (e != cudaSuccess) bad = (int)e;
      return e == cudaSuccess;
    };
    if (!check(cudaSetDevice(c->device)) || !check(cudaStreamWaitEvent(h.stream[w], h.ready, 0))) return;
    for (int64_t i; (i = next++) < chunks && bad == (int)cudaSuccess;) {
      const int64_t n = std::min(per, count - i * per);
      const void *from = (const char *)src + i * per * (widen ? sizeof(float2) : sizeof(double2));
      if (widen) {
        k_widen<<<(unsigned)((n + 255) / 256), 256, 0, h.stream[w]>>>(n, (const float2 *)from, (double2 *)h.dev[w]);
        if (!check(cudaGetLastError())) return;
        from = h.dev[w];
      }
      if (!check(cudaMemcpyAsync(h.pin[w], from, sizeof(double2) * n, cudaMemcpyDeviceToHost, h.stream[w])) ||
          !check(cudaStreamSynchronize(h.stream[w])))
        return;
      memcpy((char *)dst + i * HC_CHUNK, h.pin[w], sizeof(double2) * n);
    }
  };
  const int nw = (int)std::min<int64_t>(h.workers, chunks);
  std::vector<std::thread> threads;
  threads.reserve(nw);
  try {
    for (int w = 1; w < nw; w++) threads.emplace_back(work, w);
  } catch (...) {  // fewer threads: those that started and this one do it all
  }
  work(0);
  for (auto &t : threads) t.join();
  if (widen) c->launches += chunks;
  DMB_CUDA((cudaError_t)bad.load());
  DMB_CUDA(cudaStreamSynchronize(c->stream));
}

}  // namespace dmb
