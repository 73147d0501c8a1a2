// hostcopy.cu -- large copies between a caller's pageable buffers and the device.
//
// The drop-in calls take host buffers of the reference's program (Ne's state
// is 9 MB each way).  cudaMemcpyAsync on pageable memory runs one host thread
// through the driver's staging buffer, 7 to 10 GB/s, and fresh output pages are
// faulted in by that one thread.  Here the copy goes through a ring of pinned
// slots: several host threads fill (or empty) a slot in parallel while the
// slot before it crosses the bus.
//
// The ring and its threads belong to the process: four slots of 2 MB, made by
// the first large copy and given back by host_copy_release (with the last
// context).  Ne's right-hand side from host buffers: 2825 -> 1493 us (the RHS itself 490).
// From 512 KB on: a host call of 5 orbitals, us through the ring and on the plain path,
// by the state's size: 75 KB 149 and 137, 249 KB 161 and 156, 412 KB 177 and 182, 749 KB
// 200 and 233, 1.5 MB 280 to 320 and 335 to 355.  Page-locked (or managed) buffers cross the bus as they are, and a
// copy that finds the ring in use by another thread, a forked child, a second device, or a failed allocation takes
// the plain path too.
#include <pthread.h>
#include <sched.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>

#include "common.cuh"
#include "hostcopy.cuh"

namespace td1c {

namespace {

constexpr size_t HC_SLOT = 2u << 20, HC_MIN = 512u << 10, HC_PIECE = 128u << 10;
constexpr int HC_SLOTS = 4, HC_WORKERS = 7;

// threads that copy, the caller's included: at most one per core the process may run on, or TD1C_HOST_THREADS
int copy_threads() {
  int n = HC_WORKERS + 1;
  cpu_set_t set;
  if (sched_getaffinity(0, sizeof(set), &set) == 0) n = std::min(n, CPU_COUNT(&set));
  const char* v = getenv("TD1C_HOST_THREADS");
  if (v && atoi(v) > 0) n = std::min(HC_WORKERS + 1, atoi(v));
  return n;
}

// memcpy by several threads: the caller and the workers take pieces in turn
class CopyTeam {
 public:
  void copy(char* dst, const char* src, size_t n) {
    if (!start()) { memcpy(dst, src, n); return; }
    {
      std::unique_lock<std::mutex> l(m_);
      idle_.wait(l, [&] { return busy_ == 0; });  // a worker that woke late has left the job before
      dst_ = dst; src_ = src; n_ = n;
      next_.store(0); left_.store((int)((n + HC_PIECE - 1) / HC_PIECE));
      ++job_;
    }
    cv_.notify_all();
    work();
    while (left_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
  }

 private:
  bool start() {
    if (started_) return pid_ == getpid();
    started_ = true;
    pid_ = getpid();
    const int n = copy_threads() - 1;
    try {
      for (int k = 0; k < n; ++k) std::thread([this] { loop(); }).detach();
    } catch (...) {  // fewer workers: the caller takes their pieces
    }
    return true;
  }
  void loop() {
    unsigned long seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> l(m_);
        cv_.wait(l, [&] { return job_ != seen; });
        seen = job_;
        ++busy_;
      }
      work();
      std::lock_guard<std::mutex> l(m_);
      if (--busy_ == 0) idle_.notify_all();
    }
  }
  void work() {
    for (;;) {
      const size_t o = next_.fetch_add(1) * HC_PIECE;
      if (o >= n_) return;
      memcpy(dst_ + o, src_ + o, std::min(HC_PIECE, n_ - o));
      left_.fetch_sub(1, std::memory_order_release);
    }
  }
  std::mutex m_;
  std::condition_variable cv_, idle_;
  std::atomic<size_t> next_{0};
  std::atomic<int> left_{0};
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t n_ = 0;
  unsigned long job_ = 0;
  int busy_ = 0;
  bool started_ = false;
  pid_t pid_ = 0;
};

struct Ring {
  std::mutex m;
  CopyTeam* team = nullptr;  // lives as long as its threads, the process
  char* slot[HC_SLOTS] = {};
  cudaEvent_t ev[HC_SLOTS] = {};
  int dev = -1;
  pid_t pid = 0;

  bool ready() {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) return false;
    if (slot[0]) return d == dev && pid == getpid();
    if (team && pid != getpid()) return false;
    char* base = nullptr;
    if (cudaHostAlloc((void**)&base, HC_SLOT * HC_SLOTS, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    for (int k = 0; k < HC_SLOTS; ++k)
      if (cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) != cudaSuccess) {
        for (int q = 0; q < k; ++q) cudaEventDestroy(ev[q]);
        cudaFreeHost(base);
        cudaGetLastError();
        return false;
      }
    if (!team) team = new CopyTeam();
    for (int k = 0; k < HC_SLOTS; ++k) slot[k] = base + k * HC_SLOT;
    dev = d;
    pid = getpid();
    return true;
  }
};
Ring& ring() {
  static Ring* r = new Ring();
  return *r;
}

// whether a copy of n bytes goes through the ring: large, and of pageable memory
bool staged(const void* host, size_t n) {
  if (n < HC_MIN) return false;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return at.type == cudaMemoryTypeUnregistered;
}

}  // namespace

// queue the copy of n host bytes to the device on st; a pageable host buffer is free on return, a page-locked one
// when st is synchronised
cudaError_t host_to_device(void* dst, const void* src, size_t n, cudaStream_t st) {
  if (staged(src, n)) {
    Ring& r = ring();
    std::unique_lock<std::mutex> l(r.m, std::try_to_lock);
    if (l.owns_lock() && r.ready()) {
      int k = 0;
      for (size_t o = 0; o < n; o += HC_SLOT, k = (k + 1) % HC_SLOTS) {
        const size_t b = std::min(HC_SLOT, n - o);
        cudaError_t e = cudaEventSynchronize(r.ev[k]);  // the slot's last copy (of any call) has left it
        if (e != cudaSuccess) return e;
        r.team->copy(r.slot[k], (const char*)src + o, b);
        e = cudaMemcpyAsync((char*)dst + o, r.slot[k], b, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(r.ev[k], st);
        if (e != cudaSuccess) return e;
      }
      return cudaSuccess;
    }
  }
  return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
}

// copy n device bytes to the host after the work queued on st; complete on return where the ring was used,
// else when st is synchronised
cudaError_t device_to_host(void* dst, const void* src, size_t n, cudaStream_t st) {
  if (staged(dst, n)) {
    Ring& r = ring();
    std::unique_lock<std::mutex> l(r.m, std::try_to_lock);
    if (l.owns_lock() && r.ready()) {
      const int parts = (int)((n + HC_SLOT - 1) / HC_SLOT);
      cudaError_t e = cudaSuccess;
      auto issue = [&](int p) {
        const int k = p % HC_SLOTS;
        const size_t o = (size_t)p * HC_SLOT;
        e = cudaEventSynchronize(r.ev[k]);
        if (e == cudaSuccess) e = cudaMemcpyAsync(r.slot[k], (const char*)src + o, std::min(HC_SLOT, n - o), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(r.ev[k], st);
      };
      for (int p = 0; p < std::min(parts, HC_SLOTS) && e == cudaSuccess; ++p) issue(p);
      for (int p = 0; p < parts && e == cudaSuccess; ++p) {
        const int k = p % HC_SLOTS;
        const size_t o = (size_t)p * HC_SLOT;
        e = cudaEventSynchronize(r.ev[k]);
        if (e != cudaSuccess) break;
        r.team->copy((char*)dst + o, r.slot[k], std::min(HC_SLOT, n - o));
        if (p + HC_SLOTS < parts) issue(p + HC_SLOTS);
      }
      return e;
    }
  }
  return cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
}

// give the pinned slots back (their last copies are waited for)
void host_copy_release() {
  Ring& r = ring();
  std::lock_guard<std::mutex> l(r.m);
  if (!r.slot[0] || r.pid != getpid()) return;
  for (int k = 0; k < HC_SLOTS; ++k) {
    cudaEventSynchronize(r.ev[k]);
    cudaEventDestroy(r.ev[k]);
    r.ev[k] = nullptr;
  }
  cudaFreeHost(r.slot[0]);
  for (int k = 0; k < HC_SLOTS; ++k) r.slot[k] = nullptr;
  r.dev = -1;
}

}  // namespace td1c
