// Pageable copies of large walker sets.  A plain cudaMemcpy from or to pageable memory is
// one host thread's memcpy through the driver's staging buffer (10.5 GB/s measured, 4.4 GB/s
// into a fresh array, whose pages that thread also faults in).  Here several host threads
// move the chunks of a four-slot pinned ring while the copy engine fills or drains the
// others: 65.5 MB set 6.2 -> 2.2 ms, get 15 -> 3.2 ms with 8 threads.
#include "host_copy.h"

#include <atomic>
#include <cstring>
#include <new>
#include <thread>

namespace afq {

namespace {
constexpr int kSlots = 4;
constexpr size_t kChunk = 2u << 20;   // 8 MB of pinned memory per handle (pinning: 0.9 ms / MB)
constexpr size_t kLeast = 8u << 20;   // below: one plain copy (thread start-up ~0.1 ms)
constexpr int kMaxThreads = 8;
}  // namespace

struct HostRing {
  char* slot[kSlots] = {};
  cudaEvent_t ev[kSlots] = {};
};

void host_ring_destroy(HostRing* r) {
  if (!r) return;
  for (char* p : r->slot)
    if (p) cudaFreeHost(p);
  for (cudaEvent_t e : r->ev)
    if (e) cudaEventDestroy(e);
  delete r;
}

namespace {

bool ring_ready(HostRing** ring) {
  if (*ring) return true;
  HostRing* r = new (std::nothrow) HostRing();
  bool ok = r != nullptr;
  for (int i = 0; ok && i < kSlots; i++)
    ok = cudaMallocHost(&r->slot[i], kChunk) == cudaSuccess &&
         cudaEventCreateWithFlags(&r->ev[i], cudaEventDisableTiming) == cudaSuccess;
  if (!ok) {   // no pinned memory to spare: plain copies
    cudaGetLastError();
    host_ring_destroy(r);
    return false;
  }
  *ring = r;
  return true;
}

// Host threads that each copy their share of every chunk once it is ready.
struct Crew {
  std::atomic<long> ready{0};   // chunks whose source data is in place
  std::atomic<bool> stop{false};
  std::atomic<int> done[kSlots];
  std::thread t[kMaxThreads];
  int n = 0;

  template <class F>
  bool start(long chunks, const F& body) {
    for (auto& d : done) d.store(0);
    const unsigned hc = std::thread::hardware_concurrency();
    const int want = hc >= 4 ? (int)(hc / 2 < (unsigned)kMaxThreads ? hc / 2 : kMaxThreads) : 1;
    try {
      for (; n < want; n++)
        t[n] = std::thread([this, chunks, want, body, i = n] {
          for (long c = 0; c < chunks; c++) {
            while (ready.load(std::memory_order_acquire) <= c) {
              if (stop.load(std::memory_order_relaxed)) return;
              std::this_thread::yield();
            }
            body(c, i, want);
            done[c % kSlots].fetch_add(1, std::memory_order_release);
          }
        });
    } catch (...) {   // fewer threads than shares: none runs
      stop.store(true);
      join();
      return false;
    }
    return true;
  }
  // every thread has finished chunk c (chunks finish in order per slot)
  void wait(long c) {
    const int want = (int)(c / kSlots + 1) * n;
    while (done[c % kSlots].load(std::memory_order_acquire) < want) std::this_thread::yield();
  }
  void join() {
    for (int i = 0; i < n; i++)
      if (t[i].joinable()) t[i].join();
  }
};

// Thread i of n: its share of a chunk of `bytes`, in whole 4 KB pages.
void share(char* dst, const char* src, size_t bytes, int i, int n) {
  const size_t per = ((bytes + n - 1) / n + 4095) / 4096 * 4096;
  const size_t a = per * i < bytes ? per * i : bytes, b = a + per < bytes ? a + per : bytes;
  if (b > a) memcpy(dst + a, src + a, b - a);
}

}  // namespace

cudaError_t copy_to_host(HostRing** ring, void* dst, const void* src, size_t bytes,
                         cudaStream_t st) {
  if (bytes < kLeast) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
  Crew crew;
  const long chunks = (long)((bytes + kChunk - 1) / kChunk);
  auto len = [=](long c) { return c + 1 < chunks ? kChunk : bytes - (size_t)c * kChunk; };
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  bool crewed = ring_ready(ring);
  if (crewed) {
    HostRing* r = *ring;
    crewed = crew.start(chunks, [=](long c, int i, int n) {
      share(d + (size_t)c * kChunk, r->slot[c % kSlots], len(c), i, n);
    });
  }
  if (!crewed) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
  HostRing* r = *ring;
  cudaError_t e = cudaSuccess;
  auto issue = [&](long c) {
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(r->slot[c % kSlots], s + (size_t)c * kChunk, len(c),
                          cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaEventRecord(r->ev[c % kSlots], st);
  };
  for (long c = 0; c < chunks && c < kSlots; c++) issue(c);
  for (long c = 0; c < chunks && e == cudaSuccess; c++) {
    e = cudaEventSynchronize(r->ev[c % kSlots]);
    if (e != cudaSuccess) break;
    crew.ready.store(c + 1, std::memory_order_release);
    if (c > 0 && c - 1 + kSlots < chunks) {   // refill the slot drained before this one
      crew.wait(c - 1);
      issue(c - 1 + kSlots);
    }
  }
  if (e != cudaSuccess) crew.stop.store(true);
  crew.join();
  if (e != cudaSuccess) cudaStreamSynchronize(st);   // no copy into the ring stays in flight
  return e;
}

cudaError_t copy_to_device(HostRing** ring, void* dst, const void* src, size_t bytes,
                           cudaStream_t st) {
  if (bytes < kLeast) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  Crew crew;
  const long chunks = (long)((bytes + kChunk - 1) / kChunk);
  auto len = [=](long c) { return c + 1 < chunks ? kChunk : bytes - (size_t)c * kChunk; };
  char* d = static_cast<char*>(dst);
  const char* s = static_cast<const char*>(src);
  bool crewed = ring_ready(ring);
  if (crewed) {
    HostRing* r = *ring;
    crewed = crew.start(chunks, [=](long c, int i, int n) {
      share(r->slot[c % kSlots], s + (size_t)c * kChunk, len(c), i, n);
    });
  }
  if (!crewed) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  HostRing* r = *ring;
  cudaError_t e = cudaSuccess;
  crew.ready.store(chunks < kSlots ? chunks : kSlots, std::memory_order_release);
  for (long c = 0; c < chunks && e == cudaSuccess; c++) {
    crew.wait(c);
    e = cudaMemcpyAsync(d + (size_t)c * kChunk, r->slot[c % kSlots], len(c),
                        cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaEventRecord(r->ev[c % kSlots], st);
    if (c > 0 && c - 1 + kSlots < chunks && e == cudaSuccess) {   // the slot of c - 1 is free
      e = cudaEventSynchronize(r->ev[(c - 1) % kSlots]);
      if (e == cudaSuccess) crew.ready.store(c - 1 + kSlots + 1, std::memory_order_release);
    }
  }
  if (e != cudaSuccess) crew.stop.store(true);
  crew.join();
  const cudaError_t e2 = cudaStreamSynchronize(st);
  return e == cudaSuccess ? e2 : e;
}

}  // namespace afq
