// rg_stage.cpp - large copies between the caller's pageable memory and the device.
//
// A cudaMemcpy from or to pageable memory goes through one driver thread: a
// 33 MB image into a fresh array takes 8.7 ms, most of it the first touch of the
// array's pages and the copy out of the driver's buffer, against 0.7 ms on the
// link.  Here a few host threads, each with two page-locked slots and a stream
// of its own, take chunks in turn: while one slot is on the link, the other is
// copied.  Page-locked callers, small copies and images into pages that are already
// there keep the direct copy.
//
// The page-locked slots, streams and threads are pooled (at most kKept sets of 8 MB
// per device) while any renderer, denoiser or server exists, and freed with the last.
// Every set is used by one copy at a time, and no set is made that would not be
// kept: copies beyond the sets are direct.
#include <cuda_runtime.h>

#include <sched.h>
#include <signal.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <utility>

#include "rg_host.h"

namespace rg {

namespace {

constexpr int kWorkers = 8;  // of a copy, and at most half of the cores
// Fewer cores than this: the copies go directly (on one core a staged copy of 28 MB took 2.5 ms
// against 1.8).
constexpr int kLeastCores = 3;
constexpr size_t kChunk = size_t(512) << 10;
// Direct / staged copies on 16 host cores, ms.  To the device: 3 MB 0.30 / 0.19, 8 MB 0.77 / 0.37,
// 33 MB 3.13 / 1.34, 128 MB 11.7 / 5.4.  To untouched pages: 3 MB 1.48 / 0.47, 8 MB 3.92 / 0.56,
// 33 MB 13.9 / 2.1.  To touched pages: 8 MB 0.41 / 0.43, 33 MB 1.65 / 1.66, 64 MB 3.17 / 2.61.
constexpr size_t kStagedBytes = size_t(3) << 20, kStagedTouched = size_t(48) << 20;
// A set takes 1 - 1.6 ms to make, which a staged copy earns at about 0.05 ms per MB to the device and
// six times that to untouched pages: copies stay direct until those that could have been staged
// would nearly have paid for it (the first 1M shadow rays, 28 MB: 2.7 ms with a set made for them,
// 4.0 without).
constexpr size_t kSetCost = size_t(16) << 20;
constexpr int kUntouchedGain = 6;
constexpr int kKept = 2, kDevices = 64;
// The slots are page-locked where they lie, in huge pages: a first copy waits 1.2 ms for them,
// and 3.3 - 6.3 ms for the 2048 small pages of a cudaHostAlloc.
constexpr size_t kHugePage = size_t(2) << 20, kSlotBytes = kWorkers * 2 * kChunk,
                 kMapBytes = kSlotBytes + kHugePage;
static_assert(kSlotBytes % kHugePage == 0, "whole huge pages");

// Host cores that this thread may use: its affinity, within the control group's quota.
int usableCores() {
  cpu_set_t set;
  int cores = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : (int)std::thread::hardware_concurrency();
  if (FILE* f = std::fopen("/sys/fs/cgroup/cpu.max", "r")) {
    long long quota = 0, period = 0;
    if (std::fscanf(f, "%lld %lld", &quota, &period) == 2 && quota > 0 && period > 0)
      cores = (int)std::min<long long>(cores, std::max<long long>(1, quota / period));
    std::fclose(f);
  }
  return cores;
}

// One copy at a time, its chunks taken off a common counter by the caller and by helper threads
// that sleep between copies.  A helper that the host does not run in time is not waited for: the
// others take its chunks.  With threads started and joined for each copy, on 16 cores that 16
// other processes kept busy, 28 MB of shadow rays took 10 - 12 ms, a 720p image and its guides
// through the learned denoiser 20; now 2.2 - 4.8 and 8.5 (direct copies 4 and 8), and on an idle
// host 1.49 and 2.77 instead of 1.6 and 3.1.  Waits that sleep (cudaEventBlockingSync) instead of
// spinning cost more than the copies: 4.1 - 4.7 and 5.8 - 7.0.
struct Stage {
  const pid_t owner = getpid();
  int device = 0;
  unsigned char* slots = nullptr;  // [kWorkers][2][kChunk], page-locked
  void* map = nullptr;
  bool registered = false;
  cudaStream_t stream[kWorkers] = {};
  cudaEvent_t done[kWorkers][2] = {};
  cudaEvent_t start = nullptr;
  // the copy under way
  bool toHost = false;
  unsigned char *host = nullptr, *dev = nullptr;
  size_t bytes = 0;
  std::atomic<size_t> next{0};
  // helpers; guarded by mu
  std::mutex mu;
  std::condition_variable wake, finished;
  std::thread helpers[kWorkers];  // [0] stays empty: the caller
  int number = 0, workers = 0, active = 0;
  bool open = false, stop = false;
  cudaError_t failed = cudaSuccess;

  ~Stage() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
    }
    wake.notify_all();
    for (auto& h : helpers)
      if (h.joinable()) h.join();
    for (int w = 0; w < kWorkers; ++w) {
      for (auto e : done[w])
        if (e) cudaEventDestroy(e);
      if (stream[w]) cudaStreamDestroy(stream[w]);
    }
    if (start) cudaEventDestroy(start);
    if (registered) cudaHostUnregister(slots);
    if (map) munmap(map, kMapBytes);
  }
  bool init(int onDevice, int cores) {
    device = onDevice;
    map = mmap(nullptr, kMapBytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (map == MAP_FAILED) map = nullptr;
    if (map) {
      slots = reinterpret_cast<unsigned char*>(((uintptr_t)map + kHugePage - 1) & ~(uintptr_t)(kHugePage - 1));
      madvise(slots, kSlotBytes, MADV_HUGEPAGE);
      madvise(slots, kSlotBytes, MADV_DONTFORK);  // a forked child must not turn the locked pages copy-on-write
    }
    registered = slots && cudaHostRegister(slots, kSlotBytes, cudaHostRegisterPortable) == cudaSuccess;
    bool ok = registered && cudaEventCreateWithFlags(&start, cudaEventDisableTiming) == cudaSuccess;
    for (int w = 0; ok && w < kWorkers; ++w) {
      ok = cudaStreamCreateWithFlags(&stream[w], cudaStreamNonBlocking) == cudaSuccess;
      for (int s = 0; ok && s < 2; ++s) ok = cudaEventCreateWithFlags(&done[w][s], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
      cudaGetLastError();
      return false;
    }
    workers = 1;
    sigset_t all, before;  // the process's signals are not for the helpers
    sigfillset(&all);
    pthread_sigmask(SIG_SETMASK, &all, &before);
    try {
      for (; workers < std::min(kWorkers, cores / 2); ++workers) {
        const int w = workers;
        helpers[w] = std::thread([this, w] { help(w); });
      }
    } catch (...) {  // no more threads to be had: those there are will do
    }
    pthread_sigmask(SIG_SETMASK, &before, nullptr);
    return true;
  }
  void help(int w) {
    pthread_setname_np(pthread_self(), "rg_copy");
    cudaSetDevice(device);
    std::unique_lock<std::mutex> lk(mu);
    for (int last = 0;;) {
      wake.wait(lk, [&] { return stop || (open && number != last); });
      if (stop) return;
      last = number;
      active++;
      lk.unlock();
      const cudaError_t e = work(w);
      lk.lock();
      if (failed == cudaSuccess) failed = e;
      if (--active == 0) finished.notify_one();
    }
  }
  cudaError_t copy(bool dir, void* hostBytes, void* devBytes, size_t count, cudaStream_t after) {
    cudaError_t err = cudaEventRecord(start, after);
    if (err != cudaSuccess) return err;
    const bool alone = workers == 1 || count <= 2 * kChunk;
    {
      std::lock_guard<std::mutex> lk(mu);
      toHost = dir;
      host = (unsigned char*)hostBytes;
      dev = (unsigned char*)devBytes;
      bytes = count;
      next = 0;
      failed = cudaSuccess;
      number++;
      open = !alone;
    }
    if (!alone) wake.notify_all();
    err = work(0);
    std::unique_lock<std::mutex> lk(mu);
    open = false;  // every chunk is taken: a helper that comes now has nothing to do
    finished.wait(lk, [&] { return active == 0; });
    return err == cudaSuccess ? failed : err;
  }
  // One worker's share: chunks off the common counter, two in flight.
  cudaError_t work(int w) {
    unsigned char* slot[2] = {slots + (size_t)(2 * w) * kChunk, slots + (size_t)(2 * w + 1) * kChunk};
    size_t at[2] = {0, 0}, len[2] = {0, 0};
    auto finish = [&](int k) -> cudaError_t {  // the slot's copy is over; toHost: hand its bytes to the caller
      if (!len[k]) return cudaSuccess;
      const cudaError_t e = cudaEventSynchronize(done[w][k]);
      if (e == cudaSuccess && toHost) std::memcpy(host + at[k], slot[k], len[k]);
      len[k] = 0;
      return e;
    };
    cudaError_t err = cudaStreamWaitEvent(stream[w], start, 0);
    for (int k = 0; err == cudaSuccess; k ^= 1) {
      if ((err = finish(k)) != cudaSuccess) break;
      const size_t o = next.fetch_add(kChunk);
      if (o >= bytes) break;
      at[k] = o;
      len[k] = std::min(kChunk, bytes - o);
      if (!toHost) std::memcpy(slot[k], host + o, len[k]);
      err = toHost ? cudaMemcpyAsync(slot[k], dev + o, len[k], cudaMemcpyDeviceToHost, stream[w])
                   : cudaMemcpyAsync(dev + o, slot[k], len[k], cudaMemcpyHostToDevice, stream[w]);
      if (err == cudaSuccess) err = cudaEventRecord(done[w][k], stream[w]);
    }
    for (int k = 0; k < 2; ++k) {
      const cudaError_t e = finish(k);
      if (err == cudaSuccess) err = e;
    }
    // nothing of this copy is in flight when the slots go back to the pool
    const cudaError_t e = cudaStreamSynchronize(stream[w]);
    return err == cudaSuccess ? e : err;
  }
};

// A forked child has no helpers to join and no CUDA: the set stays as it is.
void destroy(Stage* s) {
  if (s && s->owner == getpid()) delete s;
}

std::mutex g_mu;
int g_users = 0;
struct Pool {
  Stage* idle[kKept] = {};
  int made = 0;       // sets of this device, idle and in use
  size_t missed = 0;  // gain of the copies made directly for want of a set
} g_pool[kDevices];

Stage* acquire(int dev, size_t gain) {
  if (dev >= kDevices) return nullptr;
  Pool& pool = g_pool[dev];
  int cores = 0;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (g_users == 0) return nullptr;  // nothing would keep the set: not worth its allocation
    for (auto& s : pool.idle)
      if (s) return std::exchange(s, nullptr);
    if (pool.made == kKept) return nullptr;  // all in use
    cores = usableCores();
    if (cores < kLeastCores) return nullptr;
    if (gain < kSetCost - pool.missed) {
      pool.missed += gain;
      return nullptr;
    }
    pool.missed = 0;
    pool.made++;
  }
  Stage* s = new (std::nothrow) Stage();
  if (s && s->init(dev, cores)) return s;
  destroy(s);
  std::lock_guard<std::mutex> lk(g_mu);
  pool.made--;
  return nullptr;
}

void release(Stage* s) {
  {
    std::lock_guard<std::mutex> lk(g_mu);
    Pool& pool = g_pool[s->device];
    if (g_users > 0) {
      for (auto& place : pool.idle)
        if (!place) {
          place = s;
          return;
        }
    }
    pool.made--;
  }
  destroy(s);
}

cudaMemoryType typeOf(const void* p, int* device = nullptr) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return cudaMemoryTypeManaged;  // neither pageable nor a device's own: copied directly
  }
  if (device) *device = a.device;
  return a.type;
}

// Whether the bytes lie in pages that are already there (looked up at 16 of them).
bool touched(const unsigned char* p, size_t bytes) {
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = (uintptr_t)p;
  for (int k = 0; k < 16; ++k) {
    unsigned char in = 0;
    const uintptr_t at = (a + (bytes - 1) / 15 * k) & ~(page - 1);
    if (mincore((void*)at, 1, &in) != 0 || !(in & 1)) return false;
  }
  return true;
}

// The staged copy; false: not done (no staging to be had), copy directly.
bool staged(bool toHost, void* host, void* dev, size_t bytes, cudaStream_t after, cudaError_t& err) {
  if (bytes < kStagedBytes || typeOf(host) != cudaMemoryTypeUnregistered) return false;
  // a set's streams and events belong to the device that is current here; a thread may copy from
  // another one's memory
  int current = 0, device = 0;
  if (cudaGetDevice(&current) != cudaSuccess || typeOf(dev, &device) != cudaMemoryTypeDevice || device != current) return false;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(after, &cap) != cudaSuccess) {
    cudaGetLastError();  // the launch after a direct copy must not find this query's error
    return false;
  }
  if (cap != cudaStreamCaptureStatusNone) return false;
  if (toHost && bytes < kStagedTouched && touched((const unsigned char*)host, bytes)) return false;
  Stage* s = acquire(device, toHost ? bytes * kUntouchedGain : bytes);
  if (!s) return false;
  err = s->copy(toHost, host, dev, bytes, after);
  release(s);
  return true;
}

}  // namespace

StageUser::StageUser() {
  std::lock_guard<std::mutex> lk(g_mu);
  g_users++;
}

StageUser::~StageUser() {
  Stage* old[kDevices][kKept] = {};
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_users > 0) return;
    for (int d = 0; d < kDevices; ++d) {
      g_pool[d].missed = 0;
      for (int i = 0; i < kKept; ++i)
        if ((old[d][i] = std::exchange(g_pool[d].idle[i], nullptr))) g_pool[d].made--;
    }
  }
  for (auto& sets : old)
    for (auto* s : sets) destroy(s);
}

cudaError_t copyToHost(void* dst, const void* devSrc, size_t bytes, cudaStream_t after) {
  cudaError_t err = cudaSuccess;
  if (staged(true, dst, const_cast<void*>(devSrc), bytes, after, err)) return err;
  err = cudaMemcpyAsync(dst, devSrc, bytes, cudaMemcpyDeviceToHost, after);
  return err == cudaSuccess ? cudaStreamSynchronize(after) : err;
}

cudaError_t copyToDevice(void* devDst, const void* src, size_t bytes, cudaStream_t after) {
  cudaError_t err = cudaSuccess;
  if (staged(false, const_cast<void*>(src), devDst, bytes, after, err)) return err;
  return cudaMemcpyAsync(devDst, src, bytes, cudaMemcpyHostToDevice, after);
}

}  // namespace rg
