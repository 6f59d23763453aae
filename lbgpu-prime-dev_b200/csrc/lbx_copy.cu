// lbx_copy.cu -- large copies between device memory and the caller's
// pageable host buffers.
//
// A plain copy into a freshly allocated pageable buffer is slow: the driver
// stages it on one thread, which also takes the buffer's page faults (74 MB,
// the four macro-variable planes of 150 x 131 x 117 FP64 nodes: 15 to 34 ms,
// the host's state decides).  Copies of 4 MB or more go through page-locked
// chunks instead, one for each of several host threads: while one thread
// empties or fills its chunk the others' cross the link (74 MB to the host:
// 3.5 ms; as fast with two chunks a thread; chunks of 512 KB 4.5, of 256 KB
// 5.0).  A smaller copy is done about when the threads have started (0.1 ms).
// From the host there is less to gain: 18 MB take 0.85 ms, plain 1.0 out of
// the caches and 2 out of memory.  Smaller copies, buffers the caller has
// page-locked, and any failure to set this up take the plain copy.
//
// Page-locking costs about 1 ms per MB, so it has to have been earned: the
// chunks are made when copies that would have gained about as much by them
// went before (kEarned).  A program that makes a domain, sets its fields and
// runs does not pay for what it does not use: with the chunks made by the
// first large copy, that took 20 ms longer.
//
// The chunks (one set per device, at most 8 MB) live while any domain or
// batch of the device does, and are given back when the last is destroyed.
// One copy uses them at a time; a copy that finds them taken by another host
// thread is a plain one.
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
// Bytes copied before the chunks are made, those from the host counted an
// eighth: what the chunks' 8 MB cost in time, plain copies of 16 MB into
// fresh pages lose against staged ones.
constexpr size_t kEarned = 16 << 20;
constexpr int kMaxWorkers = 8;

struct Worker {
  char* buf = nullptr;                  // its part of Stage::chunks
  cudaEvent_t ev = nullptr;             // its last copy is done
};

struct Stage {
  std::mutex busy;
  int users = 0;
  bool failed = false;                  // could not be set up: not tried again
  size_t earned = 0;
  void* chunks = nullptr;
  std::vector<Worker> workers;
  cudaStream_t stream = nullptr;        // all chunks': the link carries one after another
  cudaEvent_t ready = nullptr;
};

std::mutex g_mu;                        // guards the map and `users`
std::map<int, Stage> g_stages;          // per device; nodes never move

void tear_down(Stage& s)
{
  for (Worker& w : s.workers)
    if (w.ev) cudaEventDestroy(w.ev);
  s.workers.clear();
  if (s.chunks) cudaFreeHost(s.chunks);
  if (s.stream) cudaStreamDestroy(s.stream);
  if (s.ready) cudaEventDestroy(s.ready);
  s.chunks = nullptr;
  s.stream = nullptr;
  s.ready = nullptr;
}

bool set_up(Stage& s)
{
  if (s.failed || s.earned < kEarned) return false;
  if (!s.workers.empty()) return true;
  const int n = std::min(kMaxWorkers, (int)std::thread::hardware_concurrency() / 2);
  bool ok = n >= 2 && cudaEventCreateWithFlags(&s.ready, cudaEventDisableTiming) == cudaSuccess &&
            cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking) == cudaSuccess &&
            cudaHostAlloc(&s.chunks, n * kChunk, cudaHostAllocDefault) == cudaSuccess;
  if (ok) s.workers.resize(n);
  for (size_t w = 0; w < s.workers.size(); ++w) {
    s.workers[w].buf = (char*)s.chunks + w * kChunk;
    ok = ok && cudaEventCreateWithFlags(&s.workers[w].ev, cudaEventDisableTiming) == cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    tear_down(s);
    s.failed = true;
  }
  return ok;
}

// One worker's chunks of the copy: first, first + n, first + 2n, ...
cudaError_t move(Stage& s, int device, int first, int n, char* dst, const char* src, size_t bytes,
                 bool out)
{
  const Worker& w = s.workers[first];
  cudaError_t e = cudaSetDevice(device);
  for (size_t at = first * kChunk; at < bytes && e == cudaSuccess; at += n * kChunk) {
    const size_t len = std::min(kChunk, bytes - at);
    if (!out) std::memcpy(w.buf, src + at, len);
    e = out ? cudaMemcpyAsync(w.buf, src + at, len, cudaMemcpyDeviceToHost, s.stream)
            : cudaMemcpyAsync(dst + at, w.buf, len, cudaMemcpyHostToDevice, s.stream);
    if (e == cudaSuccess) e = cudaEventRecord(w.ev, s.stream);
    if (e == cudaSuccess) e = cudaEventSynchronize(w.ev);
    if (out && e == cudaSuccess) std::memcpy(dst + at, w.buf, len);
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
  s->earned += out ? bytes : bytes / 8;
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
  if (e == cudaSuccess) e = cudaStreamWaitEvent(s->stream, s->ready, 0);
  std::vector<cudaError_t> res(n, e);
  std::vector<std::thread> threads;
  auto work = [&](int w) {
    res[w] = move(*s, device, w, n, (char*)dst, (const char*)src, bytes, out);
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
  const cudaError_t f = cudaStreamSynchronize(s->stream);
  if (e == cudaSuccess) e = f;
  for (cudaError_t r : res)
    if (e == cudaSuccess) e = r;
  *err = e;
  return true;
}

cudaError_t copy(int device, cudaStream_t stream, void* dst, const void* src, size_t bytes, bool out)
{
  // (in a caller's capture the event would draw the chunks' stream in)
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
    s.earned = 0;
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
