// fr_workspace.cu -- the partial volume that large plane-column insertions add
// to (fr_plane.cu): one a device, whatever number of handles insert into it.
//
// At 16 bytes a cell it is larger than a job's accumulators (12), and a call
// needs it only between its first launch and its merge, which leaves it zero
// again.  So calls borrow it one after another, each stream waiting for the
// call before; it grows to the largest volume asked for while that leaves a
// quarter of the free memory, goes back to the device when an allocation of
// the library finds no room (device_malloc), and with the last handle.
#include <condition_variable>
#include <mutex>

#include "fr_handle.h"

namespace fr {
namespace {

struct Shared {
  std::mutex mu;
  std::condition_variable back;
  bool lent = false;
  void *p = nullptr;
  size_t cap = 0;
  cudaEvent_t done = nullptr;   // after the last borrower's work

  void drop() {
    if (p) {
      cudaEventSynchronize(done);
      cudaFree(p);
    }
    p = nullptr;
    cap = 0;
  }
};
constexpr int kDevices = 64;
Shared g_shared[kDevices];

Shared *of_current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= kDevices) return nullptr;
  return &g_shared[dev];
}

// Room for `bytes`, more than there was, zeroed on st; false: not to be had (a
// smaller volume stays where it is clear beforehand).
bool grow(Shared &s, size_t bytes, cudaStream_t st) {
  size_t free = 0, total = 0;
  if (cudaMemGetInfo(&free, &total) != cudaSuccess || bytes > (free + s.cap) / 4 * 3) {
    cudaGetLastError();
    return false;
  }
  s.drop();
  if (cudaMalloc(&s.p, bytes) == cudaSuccess) {
    s.cap = bytes;
    if (cudaMemsetAsync(s.p, 0, bytes, st) == cudaSuccess) return true;
  } else {
    s.p = nullptr;
  }
  cudaGetLastError();
  s.drop();
  return false;
}

}  // namespace

PlaneLease::PlaneLease(size_t bytes, cudaStream_t st) : st_(st) {
  if (bytes == 0) return;
  Shared *s = of_current_device();
  if (!s) return;
  std::unique_lock<std::mutex> lk(s->mu);
  s->back.wait(lk, [&] { return !s->lent; });
  if (!s->done && cudaEventCreateWithFlags(&s->done, cudaEventDisableTiming) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (bytes > s->cap) {
    if (!grow(*s, bytes, st)) return;
  } else if (cudaStreamWaitEvent(st, s->done, 0) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  s->lent = true;
  shared_ = s;
  quad_ = static_cast<float4 *>(s->p);
}

int PlaneLease::done() {
  if (!shared_) return FR_OK;
  Shared &s = *static_cast<Shared *>(shared_);
  const cudaError_t e = cudaEventRecord(s.done, st_);
  if (e != cudaSuccess) return fail(FR_ECUDA, "cudaEventRecord: %s", cudaGetErrorString(e));
  give_back(true);
  return FR_OK;
}

// not done(): a launch failed, and what it left behind is not zero
PlaneLease::~PlaneLease() {
  if (shared_) give_back(false);
}

void PlaneLease::give_back(bool clean) {
  Shared &s = *static_cast<Shared *>(shared_);
  {
    std::lock_guard<std::mutex> lk(s.mu);
    if (!clean) {
      cudaStreamSynchronize(st_);
      s.drop();
    }
    s.lent = false;
  }
  s.back.notify_one();
  shared_ = nullptr;
  quad_ = nullptr;
}

static bool drop_idle(Shared &s) {
  std::lock_guard<std::mutex> lk(s.mu);
  if (s.lent || !s.p) return false;
  s.drop();
  return true;
}

bool reclaim_device_memory() {
  Shared *s = of_current_device();
  return s && drop_idle(*s);
}

void workspace_leave() {
  for (Shared &s : g_shared) drop_idle(s);
}

cudaError_t device_malloc(void **p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation && reclaim_device_memory()) {
    cudaGetLastError();
    e = cudaMalloc(p, bytes);
  }
  if (e != cudaSuccess) *p = nullptr;
  return e;
}

}  // namespace fr
