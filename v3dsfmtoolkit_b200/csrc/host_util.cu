// Host-side helpers shared by the entry points.
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>

#include <cudaTypedefs.h>

#include "common.cuh"

namespace v3dba {

bool all_finite(const double* p, size_t n) {
  constexpr uint64_t kExp = 0x7ff0000000000000ull;   // exponent all ones: Inf or NaN
  uint64_t bad = 0;
  for (size_t i = 0; i < n; ++i) {
    uint64_t b;
    std::memcpy(&b, p + i, sizeof(b));
    bad |= (uint64_t)((b & kExp) == kExp);
  }
  return bad == 0;
}

bool all_finite_f(const float* p, size_t n) {
  constexpr uint32_t kExp = 0x7f800000u;
  uint32_t bad = 0;
  for (size_t i = 0; i < n; ++i) {
    uint32_t b;
    std::memcpy(&b, p + i, sizeof(b));
    bad |= (uint32_t)((b & kExp) == kExp);
  }
  return bad == 0;
}

static double now_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

PhaseTrace::PhaseTrace(const char* env, const char* lbl) : on(std::getenv(env) != nullptr), label(lbl), t(now_ms()) {}

void PhaseTrace::mark(const char* phase, cudaStream_t st) {
  if (!on) return;
  if (st) cudaStreamSynchronize(st);
  const double n = now_ms();
  std::fprintf(stderr, "%s %-12s %8.3f ms\n", label, phase, n - t);
  t = n;
}

// -1: off; k >= 0: the allocation k requests from now reports out-of-memory (then off again)
static std::atomic<long long> g_alloc_countdown{-1};

bool injected_alloc_failure() {
  if (g_alloc_countdown.load(std::memory_order_relaxed) < 0) return false;
  long long c = g_alloc_countdown.load(std::memory_order_relaxed);
  while (c >= 0 && !g_alloc_countdown.compare_exchange_weak(c, c - 1, std::memory_order_relaxed)) {
  }
  return c == 0;
}

// ---- call resources and pinned rings kept between calls --------------------------------------------

namespace {

// Pinned slots for large copies in either direction, each with the event of its copy.
struct Ring {
  static constexpr int kSlots = 8;
  static constexpr size_t kSlot = (size_t)2 << 20;
  char* mem = nullptr;
  cudaEvent_t ev[kSlots] = {};
  uint64_t ctx = 0;
};
constexpr int kRingsKept = 2;
// All that is kept, whatever its context; what a device reset left of one is among it, never used again.
constexpr size_t kAllKept = 64;

// The driver's number of a context; it is not used again after the context has ended.  Each function is asked
// for in the version whose type is named: later ones of cuStreamGetCtx take another argument.
struct Driver {
  PFN_cuCtxGetId_v12000 id = nullptr;
  PFN_cuStreamGetCtx_v9020 of_stream = nullptr;
};
const Driver& driver() {
  static const Driver d = [] {
    Driver n;
    void* f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault) == cudaSuccess)
      n.id = reinterpret_cast<PFN_cuCtxGetId_v12000>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &f, 9020, cudaEnableDefault) == cudaSuccess)
      n.of_stream = reinterpret_cast<PFN_cuStreamGetCtx_v9020>(f);
    cudaGetLastError();
    return n;
  }();
  return d;
}
// The current context, made where there is none yet in this thread or it was reset (only then is the runtime
// asked: another thread may be capturing a graph), and a stream's; 0 where there is none.
uint64_t current_context(bool make = true) {
  unsigned long long id = 0;
  if (!driver().id) return 0;
  if (driver().id(nullptr, &id) == CUDA_SUCCESS) return id;
  if (!make || cudaFree(nullptr) != cudaSuccess) return 0;
  return driver().id(nullptr, &id) == CUDA_SUCCESS ? id : 0;
}
uint64_t stream_context(cudaStream_t st) {
  CUcontext c = nullptr;
  unsigned long long id = 0;
  return driver().id && driver().of_stream && driver().of_stream(st, &c) == CUDA_SUCCESS &&
                 driver().id(c, &id) == CUDA_SUCCESS
             ? id
             : 0;
}

void destroy(CallRes& r) {
  if (r.pinned) cudaFreeHost(r.pinned);
  if (r.ev0) cudaEventDestroy(r.ev0);
  if (r.ev1) cudaEventDestroy(r.ev1);
  if (r.st) cudaStreamDestroy(r.st);
  r = CallRes();
}
void destroy(Ring& r) {
  if (r.mem) cudaFreeHost(r.mem);
  for (cudaEvent_t& e : r.ev)
    if (e) cudaEventDestroy(e);
  r = Ring();
}

// Never destroyed itself (other threads may be in a call when the process ends); what it keeps of the
// context that is current then is destroyed by a handler that runs before the CUDA runtime's own, registered
// after its first use.
struct Kept {
  std::mutex m;
  std::vector<CallRes> res;
  std::vector<Ring> rings;
  bool closing = false;
};
Kept& kept() {
  static Kept* k = [] {
    auto* n = new Kept;
    cudaFree(nullptr);
    std::atexit([] {
      Kept& k2 = kept();
      std::lock_guard<std::mutex> lock(k2.m);
      k2.closing = true;
      const uint64_t ctx = current_context(false);
      for (CallRes& r : k2.res)
        if (r.ctx == ctx) destroy(r);
      for (Ring& r : k2.rings)
        if (r.ctx == ctx) destroy(r);
      k2.res.clear();
      k2.rings.clear();
    });
    return n;
  }();
  return *k;
}

template <typename T>
bool take(std::vector<T>& v, uint64_t ctx, T& out) {
  for (size_t i = v.size(); i-- > 0;)
    if (v[i].ctx == ctx) {
      out = v[i];
      v.erase(v.begin() + (long)i);
      return true;
    }
  return false;
}
// Keeps x if its context is known and has fewer than `most`; false: the caller destroys it.
template <typename T>
bool put(std::vector<T>& v, const T& x, int most) {
  if (x.ctx == 0 || v.size() >= kAllKept) return false;
  for (const T& y : v) most -= y.ctx == x.ctx;
  if (most <= 0) return false;
  v.push_back(x);
  return true;
}

// A ring of the current context.
int ring_acquire(Ring& r) {
  const uint64_t ctx = current_context();
  if (ctx) {
    Kept& k = kept();
    std::lock_guard<std::mutex> lock(k.m);
    if (take(k.rings, ctx, r)) return V3DBA_OK;
  }
  r.ctx = ctx;
  cudaError_t e = cudaMallocHost(reinterpret_cast<void**>(&r.mem), Ring::kSlots * Ring::kSlot);
  for (int t = 0; t < Ring::kSlots && e == cudaSuccess; ++t) e = cudaEventCreateWithFlags(&r.ev[t], cudaEventDisableTiming);
  if (e == cudaSuccess) return V3DBA_OK;
  cudaGetLastError();
  destroy(r);
  return V3DBA_ERR_OUT_OF_MEMORY;
}
void ring_release(Ring& r) {
  Kept& k = kept();
  std::lock_guard<std::mutex> lock(k.m);
  if (!k.closing && put(k.rings, r, kRingsKept)) r = Ring();
  else destroy(r);
}

}  // namespace

int CallRes::acquire() {
  ctx = current_context();
  if (ctx) {
    Kept& k = kept();
    std::lock_guard<std::mutex> lock(k.m);
    if (take(k.res, ctx, *this)) return V3DBA_OK;
  }
  cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&ev1);
  if (e == cudaSuccess) e = cudaMallocHost(reinterpret_cast<void**>(&pinned), kCallResDoubles * sizeof(double));
  if (e == cudaSuccess) return V3DBA_OK;
  cudaGetLastError();
  destroy(*this);
  return e == cudaErrorMemoryAllocation ? V3DBA_ERR_OUT_OF_MEMORY : V3DBA_ERR_CUDA;
}

void CallRes::release() {
  if (!st) return;
  const bool sound = cudaStreamSynchronize(st) == cudaSuccess;
  if (!sound) cudaGetLastError();
  Kept& k = kept();
  std::lock_guard<std::mutex> lock(k.m);
  if (sound && !k.closing && put(k.res, *this, kCallResKept)) *this = CallRes();
  else destroy(*this);
}

namespace {

// Memory that the DMA engine reads and writes itself: pinned, registered or managed.
bool direct(const void* host) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host) == cudaSuccess) return a.type != cudaMemoryTypeUnregistered;
  cudaGetLastError();
  return false;
}

// A list of copies, the large ones to and from pageable memory cut into pieces of at most a slot.  The pieces
// end where a 2 MB page of the caller's memory ends, so that no two threads fault one page.
struct Pieces {
  std::vector<HostCopy> p;
  bool staged = false;
  Ring ring;
  cudaError_t err = cudaSuccess;

  Pieces(const std::vector<HostCopy>& list, bool down, cudaStream_t st) {
    constexpr size_t kPieceMin = (size_t)256 << 10;
    const size_t least = down ? kRingDown : kRingUp;
    size_t large = 0;
    for (const HostCopy& c : list)
      if (c.bytes >= kPieceMin) large += c.bytes;
    std::vector<char> cut(list.size(), 0);
    if (large >= least)   // (the look at a pointer takes 3 us)
      for (size_t i = 0; i < list.size(); ++i) {
        if (list[i].bytes < kPieceMin) continue;
        cut[i] = !direct(down ? list[i].dst : list[i].src);
        if (!cut[i]) large -= list[i].bytes;
      }
    // (the slots' events are the current context's and cannot be recorded on another one's stream)
    staged = large >= least && stream_context(st) == current_context() && ring_acquire(ring) == V3DBA_OK;
    for (size_t i = 0; i < list.size(); ++i) {
      const HostCopy& c = list[i];
      if (!c.bytes) continue;
      if (!staged || !cut[i]) {
        if (err == cudaSuccess)
          err = cudaMemcpyAsync(c.dst, c.src, c.bytes, down ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, st);
        continue;
      }
      for (size_t at = 0; at < c.bytes;) {
        const uintptr_t host = reinterpret_cast<uintptr_t>(down ? c.dst : c.src) + at;
        const size_t n = std::min(c.bytes - at, Ring::kSlot - (host & (Ring::kSlot - 1)));
        p.push_back({static_cast<char*>(c.dst) + at, static_cast<const char*>(c.src) + at, n});
        at += n;
      }
    }
  }
  ~Pieces() {
    if (!staged) return;
    if (err == cudaSuccess) ring_release(ring);
    else destroy(ring);
  }
  char* slot(int i) const { return ring.mem + (size_t)(i % Ring::kSlots) * Ring::kSlot; }
  cudaEvent_t event(int i) const { return ring.ev[i % Ring::kSlots]; }
};

// Up to kThreads threads that help a call with its copies.  They are started when a call first asks for
// help (starting them for every call cost 1 ms and more), serve any number of calls at a time, and end
// when nobody has asked for kIdle.  Never destroyed (a thread may be asleep in it when the process ends).
struct Crew {
  static constexpr int kThreads = 7;
  static constexpr std::chrono::seconds kIdle{2};
  struct Job {
    std::function<void()> work;
    int wanted = 0, running = 0;
  };
  std::mutex m;
  std::condition_variable asked, left;
  std::deque<Job*> jobs;
  int threads = 0, idle = 0;

  static Crew& get() {
    static Crew* c = new Crew;
    return *c;
  }
  void thread() {
    std::unique_lock<std::mutex> lock(m);
    for (;;) {
      ++idle;
      const bool job = asked.wait_for(lock, kIdle, [&] { return !jobs.empty(); });
      --idle;
      if (!job) {
        --threads;
        return;
      }
      Job* j = jobs.front();
      if (--j->wanted == 0) jobs.pop_front();
      ++j->running;
      lock.unlock();
      j->work();
      lock.lock();
      if (--j->running == 0) left.notify_all();
    }
  }
  void ask(Job& j, int wanted) {
    std::lock_guard<std::mutex> lock(m);
    try {
      for (int more = std::min(wanted - idle, kThreads - threads); more > 0; --more) {
        std::thread([this] { thread(); }).detach();
        ++threads;
      }
    } catch (const std::system_error&) {   // fewer, or none
    }
    if (threads == 0) return;
    j.wanted = wanted;
    jobs.push_back(&j);
    asked.notify_all();
  }
  // Ends the job: who has not begun does not begin, who has is waited for.
  void end(Job& j) {
    std::unique_lock<std::mutex> lock(m);
    if (j.wanted > 0) {
      j.wanted = 0;
      jobs.erase(std::remove(jobs.begin(), jobs.end(), &j), jobs.end());
    }
    left.wait(lock, [&] { return j.running == 0; });
  }
};

// The helpers of one call: they run `work` until it returns, at most until the end of the scope.  They
// may come late or not at all (busy with other calls, or the system has no threads left): the calling
// thread takes pieces too whenever it has nothing else to do.
struct Helpers {
  Crew::Job job;
  template <typename F>
  Helpers(int pieces, F work) {
    job.work = work;
    Crew::get().ask(job, std::min({Crew::kThreads, pieces, std::max(1, (int)std::thread::hardware_concurrency() / 2)}));
  }
  ~Helpers() { Crew::get().end(job); }
};

}  // namespace

// In both directions the pieces are taken in order, `arrived` / `done` and the flags only move forward,
// and every wait ends with the copies before it or with `stop`.
int copy_down(const std::vector<HostCopy>& list, cudaStream_t st) {
  Pieces pc(list, true, st);
  const int n = (int)pc.p.size();
  cudaError_t& err = pc.err;
  if (n > 0 && err == cudaSuccess) {
    std::vector<std::atomic<char>> taken(n);
    for (auto& t : taken) t.store(0, std::memory_order_relaxed);
    std::atomic<int> next{0}, arrived{0};
    std::atomic<bool> stop{false};
    auto take = [&](int i) {
      std::memcpy(pc.p[i].dst, pc.slot(i), pc.p[i].bytes);
      taken[i].store(1, std::memory_order_release);
    };
    Helpers helpers(n, [&]() {
      for (int i; (i = next.fetch_add(1)) < n; take(i))
        while (arrived.load(std::memory_order_acquire) <= i) {
          if (stop.load()) return;
          std::this_thread::yield();
        }
    });
    int issued = 0, a = 0;   // a: arrived
    while (a < n && err == cudaSuccess) {
      while (issued < n && issued - a < Ring::kSlots && err == cudaSuccess &&
             (issued < Ring::kSlots || taken[issued - Ring::kSlots].load(std::memory_order_acquire))) {
        err = cudaMemcpyAsync(pc.slot(issued), pc.p[issued].src, pc.p[issued].bytes, cudaMemcpyDeviceToHost, st);
        if (err == cudaSuccess) err = cudaEventRecord(pc.event(issued), st);
        ++issued;
      }
      if (err != cudaSuccess) break;
      if (a == issued) {   // every slot waits to be taken out of
        int i = next.load();
        if (i < a && next.compare_exchange_strong(i, i + 1)) take(i);
        else std::this_thread::yield();
        continue;
      }
      if ((err = cudaEventSynchronize(pc.event(a))) != cudaSuccess) break;
      arrived.store(++a, std::memory_order_release);
    }
    // who is still at work ends with its piece; pieces that nobody has begun are this thread's
    if (err != cudaSuccess) stop.store(true);
    else
      for (int i; (i = next.fetch_add(1)) < n;) take(i);
  }
  if (err == cudaSuccess) err = cudaStreamSynchronize(st);
  V3DBA_CUDA_TRY(err);
  return V3DBA_OK;
}

int copy_up(const std::vector<HostCopy>& list, cudaStream_t st) {
  Pieces pc(list, false, st);
  const int n = (int)pc.p.size();
  cudaError_t& err = pc.err;
  if (n > 0 && err == cudaSuccess) {
    std::vector<std::atomic<char>> filled(n);
    for (auto& t : filled) t.store(0, std::memory_order_relaxed);
    std::atomic<int> next{0}, done{0};   // done: pieces that have left their slots
    std::atomic<bool> stop{false};
    auto fill = [&](int i) {
      std::memcpy(pc.slot(i), pc.p[i].src, pc.p[i].bytes);
      filled[i].store(1, std::memory_order_release);
    };
    Helpers helpers(n, [&]() {
      for (int i; (i = next.fetch_add(1)) < n; fill(i))
        while (done.load(std::memory_order_acquire) + Ring::kSlots <= i) {
          if (stop.load()) return;
          std::this_thread::yield();
        }
    });
    int issued = 0, d = 0;
    while (d < n && err == cudaSuccess) {
      bool moved = false;
      if (issued < n && filled[issued].load(std::memory_order_acquire)) {
        err = cudaMemcpyAsync(pc.p[issued].dst, pc.slot(issued), pc.p[issued].bytes, cudaMemcpyHostToDevice, st);
        if (err == cudaSuccess) err = cudaEventRecord(pc.event(issued), st);
        if (err != cudaSuccess) break;
        ++issued;
        moved = true;
      }
      if (d < issued) {
        const cudaError_t q = cudaEventQuery(pc.event(d));
        if (q == cudaSuccess) {
          done.store(++d, std::memory_order_release);
          moved = true;
        } else if (q != cudaErrorNotReady) {
          err = q;
        }
      }
      if (!moved) {
        int i = next.load();
        if (i < n && i < d + Ring::kSlots && next.compare_exchange_strong(i, i + 1)) fill(i);
        else std::this_thread::yield();
      }
    }
    if (err != cudaSuccess) stop.store(true);
  }
  V3DBA_CUDA_TRY(err);
  return V3DBA_OK;
}

int Arena::commit(cudaStream_t st) {
  size_t total = 0;
  for (const Req& r : req_) total += r.bytes;
  int rc = ensure_pool();
  if (rc) return rc;
  if (injected_alloc_failure()) return V3DBA_ERR_OUT_OF_MEMORY;
  void* q = nullptr;
  V3DBA_CUDA_TRY(cudaMallocAsync(&q, std::max<size_t>(total, 256), st));
  base = static_cast<char*>(q);
  size_t off = 0;
  for (const Req& r : req_) {
    *r.p = base + off;
    off += r.bytes;
  }
  return V3DBA_OK;
}

void Arena::release(cudaStream_t st) {
  if (base) cudaFreeAsync(base, st);
  base = nullptr;
}

int ensure_pool() {
  static std::atomic<uint64_t> done_mask{0};
  int dev = 0;
  V3DBA_CUDA_TRY(cudaGetDevice(&dev));
  const uint64_t bit = 1ull << (dev & 63);
  if (done_mask.load() & bit) return V3DBA_OK;
  cudaMemPool_t pool;
  V3DBA_CUDA_TRY(cudaDeviceGetDefaultMemPool(&pool, dev));
  uint64_t thr = UINT64_MAX;
  V3DBA_CUDA_TRY(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &thr));
  done_mask.fetch_or(bit);
  return V3DBA_OK;
}

}  // namespace v3dba

extern "C" int v3dba_debug_fail_allocation(long long k) {
  if (k < -1) return V3DBA_ERR_INVALID_ARGUMENT;
  v3dba::g_alloc_countdown.store(k);
  return V3DBA_OK;
}
