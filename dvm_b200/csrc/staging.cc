// Copies between pageable host memory and the device through a ring of pinned chunks.
//
// What bounds it: a NumPy array is pageable, and the driver's own path for it runs one thread at about 17 GB/s (4 MB up in
// 242 us, a 64 KB array in 43 us) while the link carries 50 GB/s from pinned memory.  Here the calling thread and up to five
// workers copy into (or out of) pinned memory while the copy engine moves the chunk before (or after): the link and those
// threads' memcpy (42-55 GB/s together) run at the same time.  4 MB up take 120 us and down 124, of which the link needs 84.
//
// A transfer costs the calling thread about 10 us (the copy, its event, the look at it), so chunks are 1 MB: with 256 KB ones
// a call on two 4 MB arrays with a 4 MB result took 463 us, now 337.  The threads share a chunk in parts of 64 KB, so that the
// first one is ready after 25 us.
//
// The ring (8 MB per device used, in huge pages) is set up once the copies of a stretch without a pause of a minute have moved
// 32 MB by the driver's path, and given back after a minute without one: setting it up takes 2 to 4 ms, and up to 80 where the
// system has to make room for huge pages - a process that calls once, or now and then, would pay that for nothing
// (a call on two 4 MB arrays every eleven seconds took 2.8 to 84 ms with a ring set up at once and given back after ten
// seconds, 1.6 by the driver, 0.64 with a ring that is still there).  One copy uses the ring at a time; a copy that finds it taken, one on a capturing stream, a small one, one
// of pinned memory and any in a forked child goes to cudaMemcpyAsync as it is.
#include "staging.h"

#include <pthread.h>
#include <sched.h>
#include <sys/mman.h>
#ifdef __SSE2__
#include <emmintrin.h>
#endif

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>

namespace dvmb {
namespace {

constexpr size_t kChunk = 1024 * 1024;
constexpr uint32_t kSlots = 8;
constexpr size_t kPart = 64 * 1024;      // what one thread copies at a time: a chunk is ready when several have shared it
constexpr uint32_t kParts = kChunk / kPart;
constexpr size_t kSmall = 32 * 1024;   // (below this the driver's path is as fast: it sends small copies inside the command)
constexpr int kMaxDevices = 64;
constexpr uint32_t kMaxWorkers = 5;
constexpr auto kIdle = std::chrono::seconds(60);
constexpr size_t kWorth = 32 * 1024 * 1024;   // (about what the driver's path copies in the time that setting up takes)
// A worker looks for the next copy for this long before it sleeps: copies come in groups (two arguments and a result), and
// waking a thread takes 50 us and more, half the time of a 4 MB copy.
constexpr auto kLinger = std::chrono::microseconds(150);

// Into pinned memory past the caches: the copy engine reads lines that sit modified in a core's cache at a quarter of the
// link's rate (4 MB arrived 470 us after the call, the last byte having been copied after 97).
void CopyPastCache(char *dst, const char *src, size_t bytes) {
  size_t i = 0;
#ifdef __SSE2__
  if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
    for (; i + 64 <= bytes; i += 64) {
      const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i));
      const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 16));
      const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 32));
      const __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 48));
      _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i), a);
      _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 16), b);
      _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 32), c);
      _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 48), d);
    }
    _mm_sfence();
  }
#endif
  std::memcpy(dst + i, src + i, bytes - i);
}

// Pinned memory of a ring, in huge pages where the system has them: 8 MB in pages of 4 KB took cudaHostAlloc 7 to 10 ms, which
// the first call on a new process's arrays waited for; mapped in huge pages and registered they take 2 ms.
constexpr size_t kRingBytes = kChunk * kSlots, kHugePage = 2 * 1024 * 1024;
void *RingAlloc() {
  char *const map = static_cast<char *>(mmap(nullptr, kRingBytes + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
  if (map == MAP_FAILED) return nullptr;
  char *const at = map + (kHugePage - reinterpret_cast<uintptr_t>(map) % kHugePage) % kHugePage;
  if (at != map) munmap(map, at - map);
  if (map + kHugePage != at) munmap(at + kRingBytes, map + kHugePage - at);
  madvise(at, kRingBytes, MADV_HUGEPAGE);   // (refused: ordinary pages)
  madvise(at, kRingBytes, MADV_DONTFORK);   // (a child that wrote to its parent's memory here would take the pinned pages away)
  if (cudaHostRegister(at, kRingBytes, cudaHostRegisterPortable) == cudaSuccess) return at;
  munmap(at, kRingBytes);
  return nullptr;
}
void RingFree(void *p) {
  cudaHostUnregister(p);
  munmap(p, kRingBytes);
}

// While one of these lives, the thread's CUDA calls neither fail nor break a stream capture because somebody captures: polling
// an event counts as unsafe in the default mode, whatever stream the event belongs to and whichever thread captures.
class RelaxedCapture {
 public:
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
  RelaxedCapture(const RelaxedCapture &) = delete;

 private:
  cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

struct Ring {
  char *mem = nullptr;
  cudaEvent_t event[kSlots] = {nullptr};   // the last transfer that used the slot
  uint64_t issued = 0;                     // transfers ever issued; number i used slot i % kSlots
  size_t without = 0;                      // bytes that the copies of this stretch moved without a ring
};

struct Pool {
  std::mutex use;                          // one staged copy at a time
  Ring ring[kMaxDevices];
  std::chrono::steady_clock::time_point last_use;
  std::atomic<bool> dead{false};           // a forked child: its parent's workers do not exist here

  // the copy in progress
  char *host = nullptr;
  size_t bytes = 0;
  bool up = false;
  char *mem = nullptr;
  uint64_t first = 0;                      // number of the copy's first transfer
  uint32_t chunks = 0;
  uint32_t parts = 0;
  std::atomic<uint32_t> next{0}, limit{0}, done{0};   // in parts: the next to copy, those that may be copied, those copied
  std::atomic<uint32_t> copied[kSlots];    // parts copied into (out of) the slot
  std::atomic<uint32_t> inside{0};         // workers in the copy

  std::mutex m;
  std::condition_variable wake;
  std::atomic<uint64_t> generation{0};
  bool open = false;
  uint32_t workers = 0;
  bool started = false;

  size_t SizeOf(uint32_t c) const { return c + 1 == chunks ? bytes - static_cast<size_t>(c) * kChunk : kChunk; }
  char *SlotOf(uint32_t c) const { return mem + (first + c) % kSlots * kChunk; }
  uint32_t PartsOf(uint32_t c) const { return c + 1 == chunks ? parts - c * kParts : kParts; }
  // every part of chunk c has been copied (the chunks before it in its slot have, or it would not have begun)
  bool Copied(uint32_t c) const {
    return copied[(first + c) % kSlots].load(std::memory_order_acquire) >= c / kSlots * kParts + PartsOf(c);
  }

  // Copies one part if there is one to copy now.
  bool CopyOne() {
    uint32_t i = next.load(std::memory_order_relaxed);
    do {
      if (i >= parts || i >= limit.load(std::memory_order_acquire)) return false;
    } while (!next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
    const uint32_t c = i / kParts;
    const size_t at = static_cast<size_t>(i - c * kParts) * kPart, n = std::min(kPart, SizeOf(c) - at);
    char *const h = host + static_cast<size_t>(c) * kChunk + at;
    if (up) {
      CopyPastCache(SlotOf(c) + at, h, n);
    } else {
      std::memcpy(h, SlotOf(c) + at, n);
    }
    copied[(first + c) % kSlots].fetch_add(1, std::memory_order_release);
    done.fetch_add(1, std::memory_order_release);
    return true;
  }

  void Worker(bool keeper) {
    uint64_t seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lock(m);
        while (!open || generation.load() == seen) {
          if (!keeper) {
            wake.wait(lock);
          } else if (wake.wait_for(lock, kIdle) == std::cv_status::timeout) {
            lock.unlock();
            GiveBack();
            lock.lock();
          }
        }
        seen = generation.load();
        inside.fetch_add(1);
      }
      for (int idle = 0; next.load(std::memory_order_relaxed) < parts;) {
        if (CopyOne()) {
          idle = 0;
        } else if (++idle > 200) {
          std::this_thread::sleep_for(std::chrono::microseconds(20));   // (behind a long kernel or a slow link)
        } else {
          std::this_thread::yield();
        }
      }
      inside.fetch_sub(1);
      const auto until = std::chrono::steady_clock::now() + kLinger;
      while (generation.load(std::memory_order_relaxed) == seen && std::chrono::steady_clock::now() < until) std::this_thread::yield();
    }
  }

  // Frees rings when nothing has been copied for a while.
  void GiveBack() {
    std::unique_lock<std::mutex> lock(use, std::try_to_lock);
    if (!lock.owns_lock() || std::chrono::steady_clock::now() - last_use < kIdle) return;
    RelaxedCapture relaxed;
    for (int d = 0; d < kMaxDevices; ++d) {
      Ring &r = ring[d];
      if (r.mem == nullptr || cudaSetDevice(d) != cudaSuccess) continue;
      for (cudaEvent_t e : r.event) cudaEventSynchronize(e);
      for (cudaEvent_t &e : r.event) {
        cudaEventDestroy(e);
        e = nullptr;
      }
      RingFree(r.mem);
      r.mem = nullptr;
      r.issued = 0;
      r.without = 0;
    }
    cudaGetLastError();
  }

  // Whether the copy of `n` bytes goes through the ring, which is set up now if it has become worth it; `use` is held.
  bool Prepare(int dev, size_t n) {
    Ring &r = ring[dev];
    const auto now = std::chrono::steady_clock::now(), before = last_use;
    last_use = now;
    if (r.mem != nullptr) return true;
    if (now - before > kIdle) r.without = 0;
    r.without += n;
    if (r.without < kWorth) return false;
    r.without = 0;   // (should the system refuse: again after as many bytes)
    if (!started) {
      started = true;
      cpu_set_t set;
      const int cpus = sched_getaffinity(0, sizeof(set), &set) == 0 ? CPU_COUNT(&set) : 1;
      const uint32_t wanted = cpus < 2 ? 1 : std::min(static_cast<uint32_t>(cpus - 1), kMaxWorkers);
      try {
        for (; workers < wanted; ++workers) std::thread([this, keeper = workers == 0] { Worker(keeper); }).detach();
      } catch (const std::system_error &) {   // (as many as the system grants)
      }
      pthread_atfork(nullptr, nullptr, [] { Get()->dead = true; });
    }
    if (workers == 0) return false;   // (nobody would give the ring back)
    RelaxedCapture relaxed;
    void *p = RingAlloc();
    bool ok = p != nullptr;
    for (cudaEvent_t &e : r.event) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
      cudaGetLastError();
      for (cudaEvent_t &e : r.event) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
      }
      if (p) RingFree(p);
      return false;
    }
    r.mem = static_cast<char *>(p);
    return true;
  }

  static Pool *Get() {
    static Pool *const pool = new (std::nothrow) Pool();   // (never destroyed: its threads may outlive main)
    return pool;
  }

  // The copy itself; `use` is held.
  cudaError_t Run(int dev, char *device, cudaStream_t stream) {
    RelaxedCapture relaxed;
    Ring &r = ring[dev];
    mem = r.mem;
    first = r.issued;
    chunks = static_cast<uint32_t>((bytes + kChunk - 1) / kChunk);
    parts = static_cast<uint32_t>((bytes + kPart - 1) / kPart);
    next = 0;
    limit = 0;
    done = 0;
    for (auto &n : copied) n = 0;
    const bool share = parts > 1;
    if (share && up) Open();
    bool opened = share && up;
    cudaError_t err = cudaSuccess;
    uint32_t sent = 0, arrived = 0;   // transfers issued and known to be complete
    // a slot is free for chunk c when the transfer kSlots before it has completed (and, on the way down, has been copied out)
    auto complete = [&](uint64_t number) {
      const cudaError_t e = cudaEventQuery(r.event[number % kSlots]);
      if (e == cudaSuccess) return true;
      if (e != cudaErrorNotReady) err = e;
      return false;
    };
    uint32_t room = 0;   // up: chunks whose slot is free
    while (err == cudaSuccess && (up ? sent < chunks : done.load(std::memory_order_acquire) < parts)) {
      bool moved = false;
      if (up) {
        while (room < chunks && err == cudaSuccess) {
          const uint64_t number = first + room;
          if (number >= kSlots && (number - kSlots >= first + sent || !complete(number - kSlots))) break;
          ++room;
          limit.store(room * kParts, std::memory_order_release);
          moved = true;
        }
        while (sent < chunks && Copied(sent) && err == cudaSuccess) {
          err = Send(r, device, sent, stream);
          ++sent;
          moved = true;
        }
      } else {
        while (sent < chunks && err == cudaSuccess) {
          const uint64_t number = first + sent;
          if (sent >= kSlots) {
            if (!Copied(sent - kSlots)) break;
          } else if (number >= kSlots && !complete(number - kSlots)) {
            break;
          }
          err = Send(r, device, sent, stream);
          ++sent;
          moved = true;
        }
        while (arrived < sent && err == cudaSuccess && complete(first + arrived)) {
          ++arrived;
          limit.store(arrived * kParts, std::memory_order_release);
          moved = true;
        }
        if (share && !opened && arrived > 0) {   // (the workers rest until the first chunk is there)
          Open();
          opened = true;
        }
      }
      if (!CopyOne() && !moved) std::this_thread::yield();
    }
    r.issued = first + sent;
    next.store(parts);   // (after an error: nothing more to claim)
    if (opened) {
      {
        std::lock_guard<std::mutex> lock(m);
        open = false;
      }
      while (inside.load() != 0) std::this_thread::yield();
    }
    last_use = std::chrono::steady_clock::now();
    return err;
  }

  cudaError_t Send(Ring &r, char *device, uint32_t c, cudaStream_t stream) {
    char *const d = device + static_cast<size_t>(c) * kChunk;
    cudaError_t e = up ? cudaMemcpyAsync(d, SlotOf(c), SizeOf(c), cudaMemcpyHostToDevice, stream)
                       : cudaMemcpyAsync(SlotOf(c), d, SizeOf(c), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaEventRecord(r.event[(first + c) % kSlots], stream);
    return e;
  }

  void Open() {
    {
      std::lock_guard<std::mutex> lock(m);
      open = true;
      ++generation;
    }
    wake.notify_all();
  }
};

bool Pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t Copy(void *device, void *host, size_t bytes, bool up, cudaStream_t stream) {
  const auto plain = [&] {
    return up ? cudaMemcpyAsync(device, host, bytes, cudaMemcpyHostToDevice, stream)
              : cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, stream);
  };
  if (bytes < kSmall || !Pageable(host)) return plain();
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess || capturing != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return plain();
  }
  // (the ring and its events are the current device's: a stream of another one cannot record them)
  int dev = -1, stream_dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return plain();
  if (cudaStreamGetDevice(stream, &stream_dev) != cudaSuccess || stream_dev != dev) {
    cudaGetLastError();
    return plain();
  }
  Pool *const pool = Pool::Get();
  if (pool == nullptr || pool->dead.load()) return plain();
  Pool &p = *pool;
  std::unique_lock<std::mutex> lock(p.use, std::try_to_lock);   // (nothing here throws: this runs behind a C entry)
  if (!lock.owns_lock() || !p.Prepare(dev, bytes)) return plain();
  p.host = static_cast<char *>(host);
  p.bytes = bytes;
  p.up = up;
  return p.Run(dev, static_cast<char *>(device), stream);
}

}  // namespace

cudaError_t CopyToDevice(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
  return Copy(dst, const_cast<void *>(src), bytes, true, stream);
}
cudaError_t CopyToHost(void *dst, const void *src, size_t bytes, cudaStream_t stream) {
  return Copy(const_cast<void *>(src), dst, bytes, false, stream);
}

}  // namespace dvmb
