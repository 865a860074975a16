// fr_host.cu -- results into pageable host memory.
//
// A fresh array of a map's size is not mapped yet, so a plain copy into it
// faults its pages in on one thread (67 MB: 7.6 ms) and goes through the
// driver's staging buffers (4 ms more); the same bytes leave the device in
// 1.3 ms.  Here several threads each take pieces of the result through two
// pinned buffers of their own: while one piece crosses the bus, the one before
// is copied out, and the page faults are spread over the threads.
//
// The threads queue their copies on a stream of the pool, which waits for an
// event that the calling thread records: the caller's stream handle may name
// another stream in another thread (cudaStreamPerThread does).
#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <exception>
#include <thread>
#include <vector>

#include "fr_handle.h"

namespace fr {
namespace {

constexpr size_t kPiece = 2u << 20;
constexpr int kThreads = 8;
constexpr size_t kLeast = 4u << 20;   // smaller results: a plain copy

// The pinned buffers: two pieces per thread, 32 MiB in all, one set for the
// process, with the copies' stream and event on the device of the last copy.
// A copy that finds them taken by another thread's goes the plain way; they
// are freed with the last handle.
struct Pool {
  std::mutex use;
  unsigned char *p = nullptr;
  int dev = -1;
  cudaStream_t st = nullptr;
  cudaEvent_t ready = nullptr;

  void drop_stream() {
    if (st) cudaStreamDestroy(st);
    if (ready) cudaEventDestroy(ready);
    st = nullptr;
    ready = nullptr;
    dev = -1;
  }
  // Lets the pool's stream go on from where `user` is now.
  bool follow(cudaStream_t user, int device) {
    if (dev != device) {
      drop_stream();
      if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess ||
          cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess) {
        drop_stream();
        return false;
      }
      dev = device;
    }
    return cudaEventRecord(ready, user) == cudaSuccess &&
           cudaStreamWaitEvent(st, ready, 0) == cudaSuccess;
  }
} g_pool;
std::atomic<int> g_handles{0};

bool one_thread(unsigned char *pinned, unsigned char *dst, const unsigned char *src, size_t bytes,
                int t, int threads, int dev, cudaStream_t st) {
  if (cudaSetDevice(dev) != cudaSuccess) return false;
  cudaEvent_t ev[2] = {nullptr, nullptr};
  bool ok = true;
  for (auto &e : ev) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  const size_t step = kPiece * threads;
  auto size = [&](size_t off) { return std::min(kPiece, bytes - off); };
  auto fetch = [&](size_t off, int b) {
    ok = ok && cudaMemcpyAsync(pinned + b * kPiece, src + off, size(off), cudaMemcpyDeviceToHost,
                               st) == cudaSuccess;
    ok = ok && cudaEventRecord(ev[b], st) == cudaSuccess;
  };
  size_t off = t * kPiece;
  if (off < bytes) fetch(off, 0);
  for (int b = 0; ok && off < bytes; off += step, b ^= 1) {
    if (off + step < bytes) fetch(off + step, b ^ 1);
    ok = ok && cudaEventSynchronize(ev[b]) == cudaSuccess;
    if (ok) memcpy(dst + off, pinned + b * kPiece, size(off));
  }
  for (auto &e : ev)
    if (e) {
      cudaEventSynchronize(e);   // the buffer is free for the next copy
      cudaEventDestroy(e);
    }
  return ok;
}

}  // namespace

void host_pool_enter() { g_handles++; }
void host_pool_leave() {
  if (--g_handles > 0) return;
  workspace_leave();
  std::lock_guard<std::mutex> lk(g_pool.use);
  if (g_handles > 0 || !g_pool.p) return;
  cudaFreeHost(g_pool.p);
  g_pool.p = nullptr;
  g_pool.drop_stream();
}

// Copies device memory to pageable host memory, after the work queued on st,
// and waits.  false: nothing was copied for certain, take the plain way.
bool copy_to_pageable(void *dst, const void *dsrc, size_t bytes, cudaStream_t st) {
  if (bytes < kLeast) return false;
  std::unique_lock<std::mutex> lk(g_pool.use, std::try_to_lock);
  if (!lk.owns_lock()) return false;
  if (!g_pool.p &&
      cudaHostAlloc((void **)&g_pool.p, 2 * kThreads * kPiece, cudaHostAllocPortable) != cudaSuccess) {
    cudaGetLastError();
    g_pool.p = nullptr;
    return false;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  if (!g_pool.follow(st, dev)) {
    cudaGetLastError();
    return false;
  }
  const int threads = (int)std::min<size_t>(
      std::min<unsigned>(kThreads, std::max(1u, std::thread::hardware_concurrency())),
      (bytes + kPiece - 1) / kPiece);
  std::atomic<bool> ok{true};
  auto work = [&](int t) {
    if (!one_thread(g_pool.p + 2 * t * kPiece, static_cast<unsigned char *>(dst),
                    static_cast<const unsigned char *>(dsrc), bytes, t, threads, dev, g_pool.st))
      ok = false;
  };
  std::vector<std::thread> others;
  int started = 1;
  try {
    others.reserve(threads);
    for (; started < threads; started++) others.emplace_back(work, started);
  } catch (const std::exception &) {   // no more threads: their pieces are done here
  }
  work(0);
  for (int t = started; t < threads; t++) work(t);
  for (auto &o : others) o.join();
  return ok;
}

}  // namespace fr
