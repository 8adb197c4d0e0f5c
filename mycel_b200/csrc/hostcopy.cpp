// Copies between a caller's pageable arrays and the device.
//
// The driver moves pageable memory through one staging buffer by one thread: about 14 GB/s into the device, and a few
// GB/s out of it into freshly allocated arrays, whose pages the same thread faults in one by one. Here large copies go
// in chunks through pinned slots of the context, and a few threads fill or empty the slots (and touch the caller's
// pages) while the copy engine runs. 16-core host, 192x96x96: a static solve that returns 58 MB in fresh arrays 37.3 ->
// 23.6 ms, creating its problem (25 MB in) 5.3 -> 2.8 ms; a product K x of 44 MB either way 13.0 -> 3.3 ms, of 5.6 MB
// 1.12 -> 1.00 ms.
// What the threads touch costs more to unmap afterwards (every core that ran one is interrupted): a caller that makes
// and drops an array for each call loses what the copy gains, up to 0.2 ms at 2 MB and 0.9 ms at 14 MB. So the mesh
// entry points, whose arrays are often made for the call, leave their copies to the driver.
//
// The threads and slots belong to the device, at most kMaxCopiers sets of them: made at the first large copies, borrowed by
// one copy at a time, given back with the device's last context. (A set for each context made contexts that come and go
// expensive: making and freeing 12 MB of pinned memory each, and a free waits for the device and holds up the other
// contexts' launches. Four contexts of 12 problems each took 58 ms to set up instead of 35 to 42 (22 without any), and where one ended
// before the others these stood still for up to 0.7 s.) Memory the driver already knows (pinned, managed, device) and short
// copies take cudaMemcpyAsync, as does everything where the threads or slots cannot be had.
#include <cuda_runtime.h>
#include <string.h>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "internal.h"

namespace mycel {

namespace {

constexpr size_t kStagedMin = 1 << 20;   // shorter copies: waking the threads costs more than they save
constexpr size_t kSlot = 1 << 20;        // bytes of a pinned slot, the largest chunk
constexpr size_t kMinChunk = 128 << 10;
constexpr int kMaxThreads = 6;           // the caller's thread and up to five more
constexpr int kMaxCopiers = 2;           // of a device: copies that find none idle are the driver's

// Into a slot (16-byte aligned), past the caches: from lines that six cores' caches hold the copy engine read at a third
// of the speed, and copies of 3 to 16 MB took longer than the driver's (us, driver / cached stores / these: 2 MB 143 /
// 145 / 110, 8 MB 485 / 693 / 288, 16 MB 870 / 1,100 / 490, 32 MB 1,800 / 1,550 / 960).
void fill_slot(char* slot, const char* src, size_t n) {
#if defined(__SSE2__)
  size_t i = 0;
  for (; i + 64 <= n; i += 64) {
    const __m128i a = _mm_loadu_si128((const __m128i*)(src + i)), b = _mm_loadu_si128((const __m128i*)(src + i + 16));
    const __m128i c = _mm_loadu_si128((const __m128i*)(src + i + 32)), d = _mm_loadu_si128((const __m128i*)(src + i + 48));
    _mm_stream_si128((__m128i*)(slot + i), a);
    _mm_stream_si128((__m128i*)(slot + i + 16), b);
    _mm_stream_si128((__m128i*)(slot + i + 32), c);
    _mm_stream_si128((__m128i*)(slot + i + 48), d);
  }
  memcpy(slot + i, src + i, n - i);
  _mm_sfence();
#else
  memcpy(slot, src, n);
#endif
}

}  // namespace

struct HostCopy {
  int device = 0;
  int parts = 0;                   // threads of a copy, the caller's among them
  char* pinned = nullptr;          // two slots per thread
  std::vector<cudaEvent_t> ev;     // per slot: its latest copy
  std::vector<char> used;
  std::vector<std::thread> threads;

  std::mutex mu;
  std::condition_variable wake;
  std::atomic<uint64_t> job_no{0};
  std::atomic<int> left{0};        // threads that have not finished the present job
  bool stop = false;

  bool to_host = false;
  char* host = nullptr;
  char* dev = nullptr;
  size_t bytes = 0, chunk = 0, chunks = 0;
  cudaStream_t stream = nullptr;
  std::atomic<size_t> next{0};
  std::atomic<int> err{0};

  void fail(cudaError_t e) {
    int none = 0;
    if (e != cudaSuccess) err.compare_exchange_strong(none, (int)e);
  }
  size_t len(size_t c) const { return std::min(chunk, bytes - c * chunk); }

  // the slot's previous copy has read or written it
  bool slot_ready(int s) {
    if (used[(size_t)s]) fail(cudaEventSynchronize(ev[(size_t)s]));
    return err.load() == 0;
  }
  bool issue(size_t c, int s) {
    char* slot = pinned + (size_t)s * kSlot;
    char* d = dev + c * chunk;
    cudaError_t e = to_host ? cudaMemcpyAsync(slot, d, len(c), cudaMemcpyDeviceToHost, stream)
                            : cudaMemcpyAsync(d, slot, len(c), cudaMemcpyHostToDevice, stream);
    if (e == cudaSuccess) {
      used[(size_t)s] = 1;
      e = cudaEventRecord(ev[(size_t)s], stream);
    }
    fail(e);
    return e == cudaSuccess;
  }
  // thread w's share: chunks as it comes to them, through its two slots in turn
  void work(int w) {
    int s = 2 * w;
    if (!to_host) {
      for (size_t c; (c = next.fetch_add(1)) < chunks; s ^= 1) {
        if (!slot_ready(s)) return;
        fill_slot(pinned + (size_t)s * kSlot, host + c * chunk, len(c));
        if (!issue(c, s)) return;
      }
      return;
    }
    size_t c = next.fetch_add(1);
    if (c >= chunks || !slot_ready(s) || !issue(c, s)) return;
    for (;;) {
      const size_t n = next.fetch_add(1);  // the next chunk is on its way while this one is stored
      const bool more = n < chunks && slot_ready(s ^ 1) && issue(n, s ^ 1);
      if (!slot_ready(s)) return;
      memcpy(host + c * chunk, pinned + (size_t)s * kSlot, len(c));
      if (!more) return;
      c = n;
      s ^= 1;
    }
  }
  void loop(int w) {
    cudaSetDevice(device);
    uint64_t seen = 0;
    for (;;) {
      // calls often copy several arrays in a row: look for the next one for a moment before sleeping
      for (int k = 0; k < 300 && job_no.load(std::memory_order_acquire) == seen; ++k) std::this_thread::yield();
      if (job_no.load(std::memory_order_acquire) == seen) {
        std::unique_lock<std::mutex> l(mu);
        wake.wait(l, [&] { return stop || job_no.load() != seen; });
        if (stop) return;
      }
      seen = job_no.load(std::memory_order_acquire);
      work(w);
      left.fetch_sub(1, std::memory_order_release);
    }
  }
  bool start(int dev_no) {
    device = dev_no;
    const int want = std::min(kMaxThreads, (int)std::thread::hardware_concurrency() / 2);
    if (want < 2) return false;
    if (cudaHostAlloc((void**)&pinned, 2 * (size_t)want * kSlot, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      pinned = nullptr;
      return false;
    }
    parts = 1;
    try {
      used.assign(2 * (size_t)want, 0);
      ev.reserve(2 * (size_t)want);
      for (int k = 0; k < 2 * want; ++k) {
        cudaEvent_t e;
        if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
          cudaGetLastError();
          return false;
        }
        ev.push_back(e);
      }
      for (int w = 1; w < want; ++w) {
        threads.emplace_back([this, w] { loop(w); });
        ++parts;
      }
    } catch (...) {  // no more memory or threads to be had: the threads there are
    }
    return parts >= 2;
  }
  ~HostCopy() {
    {
      std::lock_guard<std::mutex> l(mu);
      stop = true;
    }
    wake.notify_all();
    for (auto& t : threads) t.join();
    for (size_t k = 0; k < ev.size(); ++k) {
      if (used[k]) cudaEventSynchronize(ev[k]);
      cudaEventDestroy(ev[k]);
    }
    if (pinned) cudaFreeHost(pinned);
  }
  cudaError_t run(bool out, char* h, char* d, size_t n, cudaStream_t s) {
    to_host = out;
    host = h;
    dev = d;
    bytes = n;
    // two chunks a thread at least, as far as they are worth a copy of their own
    chunk = std::min(kSlot, std::max(kMinChunk, (n / (2 * (size_t)parts) + 4095) & ~(size_t)4095));
    chunks = (n + chunk - 1) / chunk;
    stream = s;
    next = 0;
    err = 0;
    left = parts - 1;
    {
      std::lock_guard<std::mutex> l(mu);
      job_no.fetch_add(1, std::memory_order_release);
    }
    wake.notify_all();
    work(0);
    while (left.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    return (cudaError_t)err.load();
  }
};

// The copiers of a device: contexts borrow one for the length of a copy. All are given back with the device's last
// context.
struct Pool {
  std::mutex mu;
  HostCopy* idle[kMaxCopiers] = {};
  int n_idle = 0, made = 0;
  int contexts = 0;
  bool failed = false;  // threads or slots could not be had: not tried again before the next first context
};
static Pool* pool_of(int device) {
  static Pool pools[64];
  return device >= 0 && device < 64 ? &pools[device] : nullptr;
}

void host_copy_attach(mycel_ctx* c) {
  if (Pool* p = pool_of(c->device)) {
    std::lock_guard<std::mutex> l(p->mu);
    ++p->contexts;
  }
}

void host_copy_release(mycel_ctx* c) {
  Pool* p = pool_of(c->device);
  if (!p) return;
  HostCopy* old[kMaxCopiers];
  int n = 0;
  {
    std::lock_guard<std::mutex> l(p->mu);
    if (--p->contexts > 0) return;
    while (p->n_idle > 0) old[n++] = p->idle[--p->n_idle];
    p->made = 0;
    p->failed = false;
  }
  while (n > 0) delete old[--n];
}

// one that is idle, a new one up to the bound, or none
static HostCopy* borrow(Pool* p, int device) {
  {
    std::lock_guard<std::mutex> l(p->mu);
    if (p->n_idle > 0) return p->idle[--p->n_idle];
    if (p->failed || p->made == kMaxCopiers || p->contexts == 0) return nullptr;
    ++p->made;
  }
  HostCopy* h = new (std::nothrow) HostCopy();
  if (h && h->start(device)) return h;
  delete h;
  std::lock_guard<std::mutex> l(p->mu);
  --p->made;
  p->failed = true;
  return nullptr;
}

static cudaError_t host_copy(mycel_ctx* c, bool out, void* h, void* d, size_t n) {
  const cudaMemcpyKind kind = out ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice;
  auto plain = [&] { return cudaMemcpyAsync(out ? h : d, out ? d : h, n, kind, c->stream); };
  if (n < kStagedMin) return plain();
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, h) != cudaSuccess) {
    cudaGetLastError();
    return plain();
  }
  if (a.type != cudaMemoryTypeUnregistered) return plain();
  Pool* p = pool_of(c->device);
  if (out) {  // wait for the producers here, not in every thread
    const cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return e;
  }
  HostCopy* k = p ? borrow(p, c->device) : nullptr;
  if (!k) return plain();
  const cudaError_t e = k->run(out, (char*)h, (char*)d, n, c->stream);
  std::lock_guard<std::mutex> l(p->mu);
  p->idle[p->n_idle++] = k;
  return e;
}

cudaError_t copy_in(mycel_ctx* c, void* d, const void* h, size_t n) {
  return host_copy(c, false, const_cast<void*>(h), d, n);
}
cudaError_t copy_out(mycel_ctx* c, void* h, const void* d, size_t n) {
  return host_copy(c, true, h, const_cast<void*>(d), n);
}

}  // namespace mycel
