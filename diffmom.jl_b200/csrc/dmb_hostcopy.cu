// dmb_hostcopy.cu -- large results to the caller's (pageable) host memory.
//
// cudaMemcpy to pageable memory runs at 5 GB/s here: one thread copies out of
// the driver's bounce buffer and takes the page faults of freshly allocated
// memory (53 MB of impedance matrix: 11.2 of a call's 12 ms).  Results above
// HC_MIN bytes instead go through pinned chunks, one per worker: each worker
// copies its chunk from the device on a stream of its own and from there to the
// destination, so the transfers of some overlap the copies and faults of others.
//
// The chunks and streams belong to the device and are shared by its contexts.
// They take 4 ms to make and 1.5 to free (0.45 ms a pinned MB, 60 us a stream; a
// set of its own cost each context 8 to 14 ms), so they are made for a result
// whose plain copy takes longer than that, or once a context's plain copies
// have, and stay for the contexts that follow: programs that make a context a
// call find them there.  The first context that ends without having used them,
// with no other one using them, gives them back.  A context that finds them
// in use by another thread copies plainly.  (Chunks of 512 KB: 53 MB in 3.6 ms
// against 3.0; pieces copied in turn within a chunk gave nothing below 50 MB.)
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
constexpr size_t HC_MAKE = (size_t)24 << 20;  // 5 ms of plain copy

__global__ void k_widen(int64_t count, const float2 *__restrict__ a, double2 *__restrict__ b) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < count) b[i] = make_double2(a[i].x, a[i].y);
}

}  // namespace

struct HostCopy {
  int device;
  std::mutex mu;  // held by the one copy that uses it
  cudaStream_t stream[HC_WORKERS] = {};
  cudaEvent_t ready = nullptr;
  char *pin = nullptr;  // HC_WORKERS chunks, written by the device's copies and kernels
  std::atomic<bool> usable{false};
  explicit HostCopy(int d) : device(d) {
    bool ok = cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) == cudaSuccess &&
              cudaHostAlloc((void **)&pin, HC_WORKERS * HC_CHUNK, cudaHostAllocDefault) == cudaSuccess;
    for (int w = 0; ok && w < HC_WORKERS; w++)
      ok = cudaStreamCreateWithFlags(&stream[w], cudaStreamNonBlocking) == cudaSuccess;
    if (!ok) (void)cudaGetLastError();
    usable = ok;
  }
  HostCopy(const HostCopy &) = delete;
  HostCopy &operator=(const HostCopy &) = delete;
  ~HostCopy() {
    int now = -1;
    cudaGetDevice(&now);
    cudaSetDevice(device);
    for (cudaStream_t s : stream)
      if (s) cudaStreamDestroy(s);
    if (ready) cudaEventDestroy(ready);
    if (pin) cudaFreeHost(pin);
    if (now >= 0) cudaSetDevice(now);
    (void)cudaGetLastError();
  }
};

namespace {

std::mutex g_mu;
// never destroyed: at the end of the process the driver is gone before it
std::map<int, std::shared_ptr<HostCopy>> &chunks_of_devices() {
  static auto *all = new std::map<int, std::shared_ptr<HostCopy>>();
  return *all;
}

// the device's chunks if they are there or if `make`
std::shared_ptr<HostCopy> hostcopy_of(int device, bool make) {
  std::lock_guard<std::mutex> lk(g_mu);
  std::shared_ptr<HostCopy> &h = chunks_of_devices()[device];
  if (h && !h->usable) h.reset();
  if (!h && make) h = std::make_shared<HostCopy>(device);
  return h;
}

}  // namespace

namespace dmb {

void hostcopy_release(dmb_ctx *c) {
  std::shared_ptr<HostCopy> last;  // freed after the lock
  std::lock_guard<std::mutex> lk(g_mu);
  const bool used = c->hostcopy != nullptr;
  c->hostcopy.reset();
  std::shared_ptr<HostCopy> &h = chunks_of_devices()[c->device];
  if (!used && h.use_count() == 1) last.swap(h);
}

// by the device's chunks and workers; false on a failure (dst is then to be
// copied again)
static bool copy_staged(dmb_ctx *c, HostCopy &h, void *dst, const void *src, int64_t count, bool widen) {
  if (cudaEventRecord(h.ready, c->stream) != cudaSuccess) return false;
  const int64_t per = HC_CHUNK / sizeof(double2), chunks = (count + per - 1) / per;
  std::atomic<int64_t> next{0};
  std::atomic<bool> ok{true};
  auto work = [&](int w) {
    auto check = [&](cudaError_t e) {
      if (e != cudaSuccess) ok = false;
      return e == cudaSuccess;
    };
    char *pin = h.pin + w * HC_CHUNK;
    if (!check(cudaSetDevice(c->device)) || !check(cudaStreamWaitEvent(h.stream[w], h.ready, 0))) return;
    for (int64_t i; (i = next++) < chunks && ok;) {
      const int64_t n = std::min(per, count - i * per);
      if (widen) {
        k_widen<<<(unsigned)((n + 255) / 256), 256, 0, h.stream[w]>>>(n, (const float2 *)src + i * per, (double2 *)pin);
        check(cudaGetLastError());
      } else {
        check(cudaMemcpyAsync(pin, (const char *)src + i * HC_CHUNK, sizeof(double2) * n, cudaMemcpyDeviceToHost,
                              h.stream[w]));
      }
      if (!check(cudaStreamSynchronize(h.stream[w])) || !ok) return;
      memcpy((char *)dst + i * HC_CHUNK, pin, sizeof(double2) * n);
    }
  };
  const int nw = (int)std::min<int64_t>(HC_WORKERS, chunks);
  std::vector<std::thread> threads;
  threads.reserve(nw);
  try {
    for (int w = 1; w < nw; w++) threads.emplace_back(work, w);
  } catch (...) {  // fewer threads: those that started and this one do it all
  }
  work(0);
  for (auto &t : threads) t.join();
  if (widen) c->launches += chunks;
  return ok;
}

// memory of the caller's that the device does not reach by itself; pinned memory is
// copied to at the bus rate without a detour
static bool pageable(const void *dst) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, dst) == cudaSuccess) return a.type == cudaMemoryTypeUnregistered;
  (void)cudaGetLastError();
  return true;
}

// dst (complex128, host) <- src (device, complex64 when widen) after the work
// issued on the context's stream; returns when dst is written
void copy_out(dmb_ctx *c, void *dst, const void *src, int64_t count, bool widen) {
  const size_t bytes = sizeof(double2) * (size_t)count;
  if (bytes >= HC_MIN && pageable(dst)) {
    c->copied += bytes;
    const bool make = bytes >= HC_MAKE || c->copied >= 2 * HC_MAKE;
    if (!c->hostcopy || !c->hostcopy->usable) c->hostcopy = hostcopy_of(c->device, make);
    if (c->hostcopy) {
      HostCopy &h = *c->hostcopy;
      std::unique_lock<std::mutex> lk(h.mu, std::try_to_lock);
      if (lk.owns_lock() && h.usable) {
        if (copy_staged(c, h, dst, src, count, widen)) {
          DMB_CUDA(cudaStreamSynchronize(c->stream));
          return;
        }
        (void)cudaGetLastError();
        h.usable = false;  // its streams may be gone with the device's state: the plain copy says what is wrong
      }
    }
  }
  if (widen) {
    c->d_io[0].ensure(bytes);
    DMB_LAUNCH(c, k_widen, (unsigned)((count + 255) / 256), 256, 0, count, (const float2 *)src,
               c->d_io[0].as<double2>());
    src = c->d_io[0].p;
  }
  DMB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, c->stream));
  DMB_CUDA(cudaStreamSynchronize(c->stream));
}

}  // namespace dmb
