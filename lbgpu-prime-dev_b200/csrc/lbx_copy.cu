// lbx_copy.cu -- large copies between device memory and the caller's
// pageable host buffers.
//
// A plain copy into a freshly allocated pageable buffer runs at 5 GB/s here:
// the driver stages it on one thread, which also takes the buffer's page
// faults (the four macro-variable planes of 150 x 131 x 117 FP64 nodes, 74
// MB, took 14.6 ms of a 29 ms job; 2.4 ms staged).  Copies of 4 MB or more go
// through page-locked chunks instead, filled or emptied by several host
// threads while the next chunks cross the link; a smaller one is done about
// when the threads have started (0.1 ms).  Smaller copies, buffers the
// caller has page-locked, and any failure to set this up take the plain copy.
//
// The chunks (one set per device, 1 MB x 2 x threads, at most 16 MB) live
// while any domain or batch of the device does: made by the first large copy,
// given back when the last is destroyed.  One copy uses them at a time; a
// copy that finds them taken by another host thread is a plain one.
#include "lbx.h"
#include "lbx_internal.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

namespace {

constexpr size_t kChunk = 1 << 20;
constexpr size_t kStaged = 4 << 20;     // copies from this size on are staged
constexpr int kMaxWorkers = 8;

struct Worker {
  void* buf[2] = {nullptr, nullptr};
  cudaEvent_t ev[2] = {nullptr, nullptr};
  cudaStream_t stream = nullptr;
};

struct Stage {
  std::mutex busy;
  int users = 0;
  bool failed = false;                  // could not be set up: not tried again
  std::vector<Worker> workers;
  cudaEvent_t ready = nullptr;
};

std::mutex g_mu;                        // guards the map and `users`
std::map<int, Stage> g_stages;          // per device; nodes never move

void tear_down(Stage& s)
{
  for (Worker& w : s.workers) {
    for (int b = 0; b < 2; ++b) {
      if (w.buf[b]) cudaFreeHost(w.buf[b]);
      if (w.ev[b]) cudaEventDestroy(w.ev[b]);
    }
    if (w.stream) cudaStreamDestroy(w.stream);
  }
  s.workers.clear();
  if (s.ready) cudaEventDestroy(s.ready);
  s.ready = nullptr;
}

bool set_up(Stage& s)
{
  if (s.failed) return false;
  if (!s.workers.empty()) return true;
  const int n = std::min(kMaxWorkers, (int)std::thread::hardware_concurrency() / 2);
  bool ok = n >= 2 && cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming) == cudaSuccess;
  if (ok) s.workers.resize(n);
  for (Worker& w : s.workers) {
    ok = ok && cudaStreamCreateWithFlags(&w.stream, cudaStreamNonBlocking) == cudaSuccess;
    for (int b = 0; b < 2; ++b)
      ok = ok && cudaHostAlloc(&w.buf[b], kChunk, cudaHostAllocDefault) == cudaSuccess &&
           cudaEventCreateWithFlags(&w.ev[b], cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    tear_down(s);
    s.failed = true;
  }
  return ok;
}

// Worker w's chunks: w, w + n, w + 2n, ...
cudaError_t drain(Worker& w, int device, int first, int n, char* dst, const char* src, size_t bytes)
{
  cudaError_t e = cudaSetDevice(device);
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  auto length = [&](size_t k) { return std::min(kChunk, bytes - k * kChunk); };
  auto issue = [&](size_t k, int b) {
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(w.buf[b], src + k * kChunk, length(k), cudaMemcpyDeviceToHost, w.stream);
    if (e == cudaSuccess) e = cudaEventRecord(w.ev[b], w.stream);
  };
  int b = 0;
  if ((size_t)first < chunks) issue(first, 0);
  for (size_t k = first; k < chunks && e == cudaSuccess; k += n, b ^= 1) {
    if (k + n < chunks) issue(k + n, b ^ 1);
    if (e == cudaSuccess) e = cudaEventSynchronize(w.ev[b]);
    if (e == cudaSuccess) std::memcpy(dst + k * kChunk, w.buf[b], length(k));
  }
  return e;
}

cudaError_t fill(Worker& w, int device, int first, int n, char* dst, const char* src, size_t bytes)
{
  cudaError_t e = cudaSetDevice(device);
  const size_t chunks = (bytes + kChunk - 1) / kChunk;
  int b = 0;
  for (size_t k = first, i = 0; k < chunks && e == cudaSuccess; k += n, ++i, b ^= 1) {
    const size_t len = std::min(kChunk, bytes - k * kChunk);
    if (i >= 2) e = cudaEventSynchronize(w.ev[b]);     // the chunk's last copy has left
    if (e != cudaSuccess) break;
    std::memcpy(w.buf[b], src + k * kChunk, len);
    e = cudaMemcpyAsync(dst + k * kChunk, w.buf[b], len, cudaMemcpyHostToDevice, w.stream);
    if (e == cudaSuccess) e = cudaEventRecord(w.ev[b], w.stream);
  }
  return e;
}

bool pageable(const void* p)
{
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
  return a.type == cudaMemoryTypeUnregistered;
}

// The staged copy, waited for; false: not done (nothing was copied that a
// plain copy would not overwrite).
bool staged(int device, cudaStream_t stream, void* dst, const void* src, size_t bytes, bool out,
            cudaError_t* err)
{
  Stage* s = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    s = &g_stages[device];
  }
  std::unique_lock<std::mutex> lock(s->busy, std::try_to_lock);
  if (!lock.owns_lock()) return false;
  // streams and events belong to the current device: the domain's, and the
  // caller's again at the end
  struct Current {
    int dev = -1;
    explicit Current(int d) { if (cudaGetDevice(&dev) != cudaSuccess) dev = -1; cudaSetDevice(d); }
    ~Current() { if (dev >= 0) cudaSetDevice(dev); }
  } current(device);
  if (!set_up(*s)) return false;
  const int n = (int)s->workers.size();
  cudaError_t e = cudaEventRecord(s->ready, stream);
  for (Worker& w : s->workers)
    if (e == cudaSuccess) e = cudaStreamWaitEvent(w.stream, s->ready, 0);
  std::vector<cudaError_t> res(n, e);
  std::vector<std::thread> threads;
  auto work = [&](int w) {
    res[w] = out ? drain(s->workers[w], device, w, n, (char*)dst, (const char*)src, bytes)
                 : fill(s->workers[w], device, w, n, (char*)dst, (const char*)src, bytes);
  };
  if (e == cudaSuccess) {
    threads.reserve(n - 1);
    int started = 0;
    try {
      for (int w = 1; w < n; ++w, ++started) threads.emplace_back(work, w);
    } catch (...) {}
    work(0);
    for (int w = started + 1; w < n; ++w) work(w);      // threads that could not start
    for (std::thread& t : threads) t.join();
  }
  for (Worker& w : s->workers) {
    const cudaError_t f = cudaStreamSynchronize(w.stream);
    if (e == cudaSuccess) e = f;
  }
  for (cudaError_t r : res)
    if (e == cudaSuccess) e = r;
  *err = e;
  return true;
}

cudaError_t copy(int device, cudaStream_t stream, void* dst, const void* src, size_t bytes, bool out)
{
  // (in a caller's capture the event below would draw the workers' streams in)
  if (bytes >= kStaged && pageable(out ? dst : src) && !lbx_internal_capturing(stream)) {
    try {
      cudaError_t e = cudaSuccess;
      if (staged(device, stream, dst, src, bytes, out, &e)) return e;
    } catch (...) {}
  }
  return cudaMemcpyAsync(dst, src, bytes, out ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice,
                         stream);
}

}  // namespace

bool lbx_internal_capturing(cudaStream_t stream)
{
  if (!stream) return false;            // the default stream cannot be captured
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &status) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return status != cudaStreamCaptureStatusNone;
}

void lbx_internal_copy_user(int device, int add)
{
  try {
    std::lock_guard<std::mutex> lock(g_mu);
    Stage& s = g_stages[device];
    s.users += add;
    if (s.users > 0) return;
    // no domain or batch is left on the device, so no copy is under way
    tear_down(s);
    s.failed = false;
  } catch (...) {}
}

cudaError_t lbx_internal_copy_out(int device, cudaStream_t stream, void* dst, const void* src,
                                  size_t bytes)
{
  return copy(device, stream, dst, src, bytes, true);
}

cudaError_t lbx_internal_copy_planes_out(int device, cudaStream_t stream, void* const* dst,
                                         int count, const void* src, size_t plane)
{
  for (int c = 0, n = 1; c < count; c += n, n = 1) {
    if (!dst[c]) continue;
    if (count * plane >= kStaged)
      while (c + n < count && dst[c + n] == (char*)dst[c] + n * plane && pageable(dst[c]) &&
             pageable(dst[c + n]))
        ++n;
    const cudaError_t e =
        copy(device, stream, dst[c], (const char*)src + c * plane, n * plane, true);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t lbx_internal_copy_in(int device, cudaStream_t stream, void* dst, const void* src,
                                 size_t bytes)
{
  return copy(device, stream, dst, src, bytes, false);
}
