// Host resources an engine keeps between calls: its worker threads, and the
// page-locked buffers of target sets and row copies.
#pragma once

#include <cuda_runtime_api.h>
#include <sys/types.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <functional>
#include <list>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace sxe {

// ---- host workers ------------------------------------------------------------
// The engine's host threads, started with the first loop that needs them and
// joined with the engine: a search runs several short loops, and fresh threads
// for each cost it more than the work (15 threads: ~0.2 ms).  Loops of several
// threads may run at once (the engine thread's and the domain-definition
// driver's); every caller works on its own loop until it is done.  An exception
// of a body ends its loop and is thrown to the loop's caller.
// The threads belong to the process that started them.  In a child forked from
// it they do not exist, though the pool's state says so: there a loop runs on its
// caller alone, and the state is left behind rather than joined.
class WorkerPool {
 public:
  explicit WorkerPool(int threads) : most_(std::max(0, threads - 1)), st_(new State) {}
  ~WorkerPool() {
    if (foreign()) {
      (void)st_.release();
      return;
    }
    {
      std::lock_guard<std::mutex> g(st_->mu);
      st_->stop = true;
    }
    st_->wake.notify_all();
    for (auto& t : st_->th) t.join();
  }
  // f(i) for every i < n on at most `threads` threads, the caller among them.
  template <typename F>
  void run(size_t n, int threads, F&& f) {
    if (n == 0) return;
    const int helpers = (int)std::min<size_t>({(size_t)std::max(0, threads - 1), (size_t)most_, n - 1});
    if (helpers == 0 || foreign()) {
      for (size_t i = 0; i < n; i++) f(i);
      return;
    }
    Loop loop;
    loop.n = n;
    loop.room = helpers;
    loop.body = [&f](size_t i) { f(i); };
    State& st = *st_;
    {
      std::lock_guard<std::mutex> g(st.mu);
      try {
        while ((int)st.th.size() < most_) {
          owner_.store(getpid());
          st.th.emplace_back([&st] { work(st); });
        }
      } catch (const std::system_error&) {  // no more threads to be had: fewer help
      }
      st.open.push_back(&loop);
    }
    if (helpers == 1) st.wake.notify_one();
    else st.wake.notify_all();
    loop.drain();
    std::unique_lock<std::mutex> g(st.mu);
    st.open.remove(&loop);  // no helper joins any more
    st.idle.wait(g, [&] { return loop.inside == 0; });
    if (loop.error) std::rethrow_exception(loop.error);
  }

 private:
  struct Loop {
    size_t n = 0;
    int room = 0, inside = 0;  // helpers that may still join, helpers at work (under the pool's mutex)
    std::function<void(size_t)> body;
    std::atomic<size_t> next{0};
    std::mutex err_mu;
    std::exception_ptr error;
    void drain() {
      try {
        for (size_t i; (i = next.fetch_add(1)) < n;) body(i);
      } catch (...) {
        next.store(n);
        std::lock_guard<std::mutex> g(err_mu);
        if (!error) error = std::current_exception();
      }
    }
  };
  struct State {
    std::mutex mu;
    std::condition_variable wake, idle;
    std::list<Loop*> open;
    std::vector<std::thread> th;
    bool stop = false;
  };
  static void work(State& st) {
    std::unique_lock<std::mutex> g(st.mu);
    for (;;) {
      Loop* l = nullptr;
      st.wake.wait(g, [&] {
        for (Loop* o : st.open)
          if (o->room > 0 && o->next.load() < o->n) {
            l = o;
            return true;
          }
        return st.stop;
      });
      if (!l) return;
      l->room--;
      l->inside++;
      g.unlock();
      l->drain();
      g.lock();
      if (--l->inside == 0) st.idle.notify_all();
    }
  }
  bool foreign() const {
    const pid_t o = owner_.load();
    return o && o != getpid();
  }
  const int most_;
  std::unique_ptr<State> st_;
  std::atomic<pid_t> owner_{0};  // of the threads; 0 before the first
};

// ---- page-locked buffers -------------------------------------------------------
// Page-locked host memory for the packed residues of target sets, so their
// copy to the device runs at the bus's rate rather than through the driver's
// pageable staging; plain heap memory when the pinned allocation fails.
// Growing a vector leaves the new elements uninitialised (the packers write
// every byte).
template <typename T>
struct PinnedAlloc {
  using value_type = T;
  PinnedAlloc() = default;
  template <typename U>
  PinnedAlloc(const PinnedAlloc<U>&) {}
  // Each block starts with a 64-byte header recording how it was obtained,
  // so it is freed the same way even after the CUDA context is gone.
  static constexpr size_t kHead = 64;
  T* allocate(size_t n) {
    const size_t bytes = std::max<size_t>(n, 1) * sizeof(T) + kHead;
    void* p = nullptr;
    uint32_t pinned = 1;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocDefault) != cudaSuccess) {
      cudaGetLastError();
      pinned = 0;
      p = std::malloc(bytes);
      if (!p) throw std::bad_alloc();
    }
    std::memcpy(p, &pinned, sizeof pinned);
    return reinterpret_cast<T*>(static_cast<char*>(p) + kHead);
  }
  void deallocate(T* q, size_t) {
    void* p = reinterpret_cast<char*>(q) - kHead;
    uint32_t pinned = 0;
    std::memcpy(&pinned, p, sizeof pinned);
    if (pinned) {
      if (cudaFreeHost(p) != cudaSuccess) cudaGetLastError();
    } else {
      std::free(p);
    }
  }
  template <typename U>
  void construct(U* p) noexcept {}  // default-initialise: no fill
  template <typename U, typename... A>
  void construct(U* p, A&&... a) {
    ::new ((void*)p) U(std::forward<A>(a)...);
  }
  template <typename U>
  bool operator==(const PinnedAlloc<U>&) const { return true; }
  template <typename U>
  bool operator!=(const PinnedAlloc<U>&) const { return false; }
};
using HostBytes = std::vector<uint8_t, PinnedAlloc<uint8_t>>;

// Recycled page-locked buffers, the two largest that came back: a caller that
// streams batches of targets (or of row copies) writes into pages already locked
// and touched.  Locking 300 MB anew took 220 ms a batch, against 17 for packing
// and uploading it.
class HostBytePool {
 public:
  // Buffers above `most` bytes are not kept.
  explicit HostBytePool(size_t most = SIZE_MAX) : most_(most) {}
  HostBytes take(size_t bytes) {
    std::lock_guard<std::mutex> g(mu_);
    for (size_t i = 0; i < free_.size(); i++)
      if (free_[i].capacity() >= bytes) {
        HostBytes v = std::move(free_[i]);
        free_.erase(free_.begin() + (std::ptrdiff_t)i);
        v.clear();
        return v;
      }
    HostBytes v;
    // sizes vary from call to call: some room, so that buffers grow seldom
    v.reserve(bytes + std::min<size_t>(bytes / 4, 16u << 20));
    return v;
  }
  void give(HostBytes&& v) {
    if (!v.capacity()) return;
    if (v.capacity() > most_) {
      HostBytes().swap(v);
      return;
    }
    std::lock_guard<std::mutex> g(mu_);
    free_.push_back(std::move(v));
    if (free_.size() > 2)  // keep the two largest
      free_.erase(std::min_element(free_.begin(), free_.end(),
                                   [](const auto& x, const auto& y) { return x.capacity() < y.capacity(); }));
  }

 private:
  const size_t most_;
  std::mutex mu_;
  std::vector<HostBytes> free_;
};

}  // namespace sxe
