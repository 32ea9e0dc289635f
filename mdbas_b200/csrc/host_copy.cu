// host_copy.cu -- see host_copy.cuh.
//
// A cudaMemcpyAsync to pageable memory waits for the stream, and is copied by
// one thread through the driver's own page-locked buffer (about 12 GB/s where
// the link does 50), one array after the other.  Here the arrays of a result
// are cut into chunks with a page-locked slot each: all device copies are
// issued at once (as one where the arrays follow each other on the device)
// and waited for in order, and large results are unpacked by a few threads,
// any of which takes the next chunk, so that the caller never waits for a
// helper that is slow to wake up.  Results with more chunks than slots go
// round.  Host to device, the driver's way is as good (72 KB: 24 us against
// 44 through slots; 2.3 MB: 146 against 140) and stays.
//
// There is one set of slots, made after the first few results (kPlainFirst)
// and given back with the last engine.  A caller that finds it taken (another
// thread is copying) and arrays that are page-locked already use plain
// cudaMemcpyAsync.
//
// Measured (B200, 16-core virtual host), the caller's arrays touched before:
// 72 KB of forces 70 -> 39 us, 2.3 MB 240 -> 139 us; makelist and energy of
// 18,558 atoms (a 43 MB list) 5.5 -> 3.1 to 3.7 ms.  Helpers: one up to 8 MB (2.3 MB:
// 139 us, with two 154, with none 211), three beyond (five: no better); none
// for results that are added to the caller's arrays, whose pages are often
// new (every thread's page faults interrupt the others: an SPME call of
// 96,000 atoms 1.34 ms with three, 0.92 with none).  Slots of 256 KB and 1 MB
// measured 182 and 153 us for the 2.3 MB.
#include <string.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <exception>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

#include "host_copy.cuh"

namespace mdbas {
namespace {

constexpr size_t kSlotBytes = (size_t)512 << 10;
constexpr int kSlots = 32;    // 16 MB page-locked at most
// Results copied the plain way before the slots are made: page-locking costs
// about 0.7 ms a MB and 0.5 ms more (72 KB: 1 to 3 ms, 2.3 MB 4 ms), what 10 to
// 40 results gain, so that an engine that is asked a few times does not pay for
// it (the first result of a new engine of 3,000 atoms 1.7 -> 0.1 ms).
constexpr int kPlainFirst = 8;
constexpr int kHelpers = 3;
constexpr size_t kManyFrom = (size_t)8 << 20;     // smaller transfers: one helper
constexpr int kMaxSpans = 16;
constexpr size_t kLookFrom = (size_t)128 << 10;   // smaller arrays: staged even if page-locked

// Helper threads that run one job at a time; a job is a function every
// thread calls once, and returns from when nothing is left to take.  A job for
// `helpers` threads is always for the same ones: taken in turn by all of three,
// the lines of the caller's arrays move between their cores, and 2.3 MB took
// 380 us where one thread's 110 are.
class Helpers {
 public:
  void start(int helpers, void (*fn)(void *), void *arg) {
    {
      std::lock_guard<std::mutex> lk(m_);
      try {
        while ((int)threads_.size() < helpers)
          threads_.emplace_back([this, k = (int)threads_.size()] { loop(k); });
      } catch (const std::exception &) {  // no more threads: with those there are
      }
      fn_ = fn;
      arg_ = arg;
      helpers_ = helpers;
      ++job_;
    }
    for (int k = 0; k < helpers; ++k) cv_[k].notify_one();
  }
  // No helper enters the job any more, and those inside have left it.
  void finish() {
    std::unique_lock<std::mutex> lk(m_);
    fn_ = nullptr;
    idle_.wait(lk, [this] { return inside_ == 0; });
  }
  void stop() {
    {
      std::lock_guard<std::mutex> lk(m_);
      stop_ = true;
    }
    for (std::condition_variable &cv : cv_) cv.notify_one();
    for (std::thread &t : threads_) t.join();
    threads_.clear();
    stop_ = false;
  }

 private:
  void loop(int k) {
    std::unique_lock<std::mutex> lk(m_);
    for (unsigned long long done = job_ - 1;;) {
      cv_[k].wait(lk, [&] { return stop_ || (fn_ && k < helpers_ && done != job_); });
      if (stop_) return;
      done = job_;
      auto *fn = fn_;
      void *arg = arg_;
      ++inside_;
      lk.unlock();
      fn(arg);
      lk.lock();
      if (--inside_ == 0) idle_.notify_all();
    }
  }
  std::mutex m_;
  std::condition_variable cv_[kHelpers], idle_;  // cv_[k]: thread k's
  std::vector<std::thread> threads_;
  void (*fn_)(void *) = nullptr;
  void *arg_ = nullptr;
  int helpers_ = 0;             // threads that may enter the job
  unsigned long long job_ = 1;  // its number; each thread enters once
  int inside_ = 0;
  bool stop_ = false;
};

struct Pool {
  std::mutex busy;           // held for a whole transfer
  char *slot[kSlots] = {};
  cudaEvent_t ev[kSlots] = {};
  int device = -1;           // the events' device
  int plain = 0;             // results copied the plain way (up to kPlainFirst)
  std::mutex users_m;
  int users = 0;
  Helpers helpers;

  void free_slots() {
    for (int k = 0; k < kSlots; ++k) {
      if (ev[k]) cudaEventDestroy(ev[k]);
      if (slot[k]) cudaFreeHost(slot[k]);
      ev[k] = nullptr;
      slot[k] = nullptr;
    }
    device = -1;
    plain = 0;
  }
  // The first `n` slots and their events on the current device.
  bool ready(int n, int dev) {
    if (device != dev) {
      for (int k = 0; k < kSlots; ++k) {
        if (ev[k]) cudaEventDestroy(ev[k]);
        ev[k] = nullptr;
      }
      device = dev;
    }
    for (int k = 0; k < n; ++k) {
      if (!slot[k] && cudaHostAlloc(reinterpret_cast<void **>(&slot[k]), kSlotBytes,
                                    cudaHostAllocPortable) != cudaSuccess) {
        slot[k] = nullptr;
        cudaGetLastError();
        return false;
      }
      if (!ev[k] && cudaEventCreateWithFlags(&ev[k], cudaEventDisableTiming) != cudaSuccess) {
        ev[k] = nullptr;
        cudaGetLastError();
        return false;
      }
    }
    return true;
  }
};

Pool &pool() {
  static Pool *p = new Pool();  // outlives static destructors that still copy
  return *p;
}

// Page-locked (or managed) memory goes straight to the copy engine.
bool pageable(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// Pieces of spans; a chunk is a run of pieces that fits one slot.
struct Piece {
  char *host;
  char *dev;
  size_t bytes, at;  // at: offset in the slot
  bool add, joins;   // joins: one device array with the piece before
};
struct Chunk {
  int first, count;
};

struct Transfer {
  Pool *p;
  cudaStream_t s;
  int device;
  std::vector<Piece> pieces;
  std::vector<Chunk> chunks;
  std::vector<std::atomic<int>> issued;  // the chunk's device copies are on the stream
  std::atomic<int> next{0};
  std::atomic<int> err{0};
  explicit Transfer(size_t n) : issued(n) {}
};

void cut(const CopySpan *spans, int count, std::vector<Piece> &pieces,
         std::vector<Chunk> &chunks) {
  size_t used = kSlotBytes;  // no open chunk
  for (int k = 0; k < count; ++k) {
    char *h = static_cast<char *>(spans[k].host), *d = static_cast<char *>(spans[k].dev);
    bool joins = spans[k].joins;
    for (size_t left = spans[k].bytes; left > 0;) {
      if (used >= kSlotBytes) {
        chunks.push_back({(int)pieces.size(), 0});
        used = 0;
      }
      const size_t b = std::min(left, kSlotBytes - used);
      pieces.push_back({h, d, b, used, spans[k].add, joins});
      joins = true;
      ++chunks.back().count;
      used = (used + b + 15) & ~(size_t)15;
      h += b;
      d += b;
      left -= b;
    }
  }
}

void add(double *a, const double *b, size_t n) {
  for (size_t k = 0; k < n; ++k) a[k] += b[k];
}

// The device copies of a chunk; pieces of one device array that follow one
// another there and in the slot go as one.
cudaError_t issue(Transfer &t, int c) {
  const Chunk &ch = t.chunks[c];
  char *slot = t.p->slot[c % kSlots];
  for (int k = ch.first; k < ch.first + ch.count;) {
    Piece m = t.pieces[k++];
    while (k < ch.first + ch.count && t.pieces[k].joins &&
           t.pieces[k].dev == m.dev + m.bytes && t.pieces[k].at == m.at + m.bytes)
      m.bytes += t.pieces[k++].bytes;
    const cudaError_t e =
        cudaMemcpyAsync(slot + m.at, m.dev, m.bytes, cudaMemcpyDeviceToHost, t.s);
    if (e != cudaSuccess) return e;
  }
  return cudaEventRecord(t.p->ev[c % kSlots], t.s);
}

void issue_marked(Transfer &t, int c) {
  const cudaError_t e = issue(t, c);
  int none = 0;
  if (e != cudaSuccess) t.err.compare_exchange_strong(none, (int)e);
  t.issued[c].store(1, std::memory_order_release);
}

void run(void *arg) {
  Transfer &t = *static_cast<Transfer *>(arg);
  const int n = (int)t.chunks.size();
  bool device_set = false;
  for (;;) {
    const int c = t.next.fetch_add(1);
    if (c >= n) return;
    if (!device_set) {
      cudaSetDevice(t.device);
      device_set = true;
    }
    while (!t.issued[c].load(std::memory_order_acquire)) std::this_thread::yield();
    const cudaError_t e = cudaEventSynchronize(t.p->ev[c % kSlots]);
    int none = 0;
    if (e != cudaSuccess) t.err.compare_exchange_strong(none, (int)e);
    const char *slot = t.p->slot[c % kSlots];
    const Chunk &ch = t.chunks[c];
    if (e == cudaSuccess && !t.err.load())
      for (int k = ch.first; k < ch.first + ch.count; ++k) {
        const Piece &pc = t.pieces[k];
        if (pc.add)
          add(reinterpret_cast<double *>(pc.host), reinterpret_cast<const double *>(slot + pc.at),
              pc.bytes / sizeof(double));
        else
          memcpy(pc.host, slot + pc.at, pc.bytes);
      }
    if (c + kSlots < n) issue_marked(t, c + kSlots);  // the slot is free
  }
}

// The plain way; what is added is added once all of the spans are there.
cudaError_t plain(const CopySpan *spans, int count, cudaStream_t s) {
  std::vector<std::vector<double>> h(count);
  bool adds = false;
  for (int k = 0; k < count; ++k)
    if (spans[k].add) {
      h[k].resize(spans[k].bytes / sizeof(double));
      adds = true;
    }
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < count && e == cudaSuccess; ++k)
    e = cudaMemcpyAsync(spans[k].add ? h[k].data() : spans[k].host, spans[k].dev, spans[k].bytes,
                        cudaMemcpyDeviceToHost, s);
  if (!adds) return e;
  const cudaError_t w = cudaStreamSynchronize(s);  // before h goes, in any case
  if (e == cudaSuccess) e = w;
  for (int k = 0; k < count && e == cudaSuccess; ++k)
    if (spans[k].add) add(static_cast<double *>(spans[k].host), h[k].data(), h[k].size());
  return e;
}

}  // namespace

int copy_in(const CopySpan *spans, int count, cudaStream_t s) {
  for (int k = 0; k < count; ++k)
    if (spans[k].bytes > 0)
      MDB_CUDA(cudaMemcpyAsync(spans[k].dev, spans[k].host, spans[k].bytes,
                               cudaMemcpyHostToDevice, s));
  return MDBAS_NB_OK;
}

namespace {

// With the pool's slots, or without (p null).
int unpack(const CopySpan *spans, int count, cudaStream_t s, Pool *p) {
  CopySpan staged[kMaxSpans], direct[kMaxSpans];
  int ns = 0, nd = 0;
  size_t bytes = 0;
  bool adds = false;
  for (int k = 0; k < count; ++k) {
    if (spans[k].bytes == 0) continue;
    if (p && (spans[k].add || spans[k].bytes < kLookFrom || pageable(spans[k].host))) {
      adds |= spans[k].add;
      bytes += spans[k].bytes;
      staged[ns++] = spans[k];
    } else {
      direct[nd++] = spans[k];
    }
  }
  std::vector<Piece> pieces;
  std::vector<Chunk> chunks;
  cut(staged, ns, pieces, chunks);
  const int n = (int)chunks.size();
  int dev = 0;
  if (n > 0) MDB_CUDA(cudaGetDevice(&dev));
  if (n > 0 && !p->ready(std::min(n, kSlots), dev))  // no page-locked memory left
    return unpack(spans, count, s, nullptr);
  if (nd > 0) MDB_CUDA(plain(direct, nd, s));
  if (n > 0) {
    Transfer t(n);
    t.p = p;
    t.s = s;
    t.device = dev;
    t.pieces.swap(pieces);
    t.chunks.swap(chunks);
    for (int c = 0; c < std::min(n, kSlots); ++c) issue_marked(t, c);
    const int helpers = adds || n == 1 ? 0 : bytes < kManyFrom ? 1 : kHelpers;
    if (helpers > 0) p->helpers.start(helpers, run, &t);
    run(&t);
    if (helpers > 0) p->helpers.finish();
    if (const int e = t.err.load())
      return cuda_fail((cudaError_t)e, "copy_out", __FILE__, __LINE__);
  }
  MDB_CUDA(cudaStreamSynchronize(s));
  return MDBAS_NB_OK;
}

}  // namespace

int copy_out(const CopySpan *spans, int count, cudaStream_t s) {
  if (count > kMaxSpans) return MDBAS_NB_ERR_ARG;
  Pool &p = pool();
  std::unique_lock<std::mutex> lk(p.busy, std::try_to_lock);
  if (lk.owns_lock() && p.plain < kPlainFirst) {
    ++p.plain;
    lk.unlock();
  }
  int st;
  try {
    st = unpack(spans, count, s, lk.owns_lock() ? &p : nullptr);
  } catch (const std::bad_alloc &) {
    st = MDBAS_NB_ERR_ALLOC;
  }
  // copies on their way must not outlive the call, nor its hold on the slots
  if (st != MDBAS_NB_OK) cudaStreamSynchronize(s);
  return st;
}

void host_copy_enter() {
  std::lock_guard<std::mutex> lk(pool().users_m);
  ++pool().users;
}

void host_copy_leave() {
  Pool &p = pool();
  std::lock_guard<std::mutex> lk(p.users_m);
  if (--p.users > 0) return;
  std::lock_guard<std::mutex> busy(p.busy);
  p.helpers.stop();
  p.free_slots();
}

}  // namespace mdbas
