// Internal declarations shared by the engine's host translation units:
// device buffers, streams and slots, the engine / profile-set / target-set
// objects behind the C ABI handles, and the functions one file defines for
// another (packing: pack.cu; the search scheduler: scheduler.cu; device
// domain-definition passes: domain_passes.cu; C ABI: engine.cu, score.cu,
// static_entry.cu).
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <functional>
#include <memory>
#include <mutex>
#include <numeric>
#include <string>
#include <thread>
#include <unordered_map>
#include <vector>

#include "../../include/sxhmm.h"
#include "host_pools.hpp"
#include "internal.hpp"
#include "shapes.hpp"

using namespace sx;
using sxk::BinRegion;
using sxk::DevProfile;
using sxk::MsvTile;
using sxk::PairRec;
using sxk::Thresholds;

// defined with their kernels in long.cuh / plain.cuh
namespace sxk {
struct LongPair;
struct PlainProfile;
struct AdjPair;
}  // namespace sxk

namespace sxe {

// last error message of the calling thread (sx_last_error)
extern thread_local std::string g_err;

// Names the kernels of one entry-point call for profilers (a no-op unless a
// tool is attached), e.g. ncu --nvtx --nvtx-include "sx_search/".
struct NvtxRange {
  explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
};

// Wall-clock phases of one sx_search, printed to stderr when the environment
// variable SXHMM_PROFILE is set (a diagnostic for tuning placements; it adds
// clock reads only).
struct PhaseLog {
  bool on = std::getenv("SXHMM_PROFILE") != nullptr;
  std::mutex mu;  // entries may come from the host pool's thread
  std::vector<std::pair<std::string, double>> v;
  void add(const std::string& name, std::chrono::steady_clock::time_point t0) {
    if (!on) return;
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    std::lock_guard<std::mutex> g(mu);
    v.emplace_back(name, ms);
  }
  void print() {
    if (!on) return;
    std::lock_guard<std::mutex> g(mu);
    std::string o = "[sxhmm profile]";
    char buf[96];
    for (const auto& p : v) {
      snprintf(buf, sizeof buf, " %s=%.1fms", p.first.c_str(), p.second);
      o += buf;
    }
    fprintf(stderr, "%s\n", o.c_str());
  }
};
// Records msg as the calling thread's last error and returns code.
int fail(int code, const std::string& msg);


struct CudaError {
  int code;
  std::string msg;
};

#define CK(call)                                                                                      \
  do {                                                                                                \
    cudaError_t e_ = (call);                                                                          \
    if (e_ != cudaSuccess)                                                                            \
      throw CudaError{e_ == cudaErrorMemoryAllocation ? SX_ENOMEM : SX_ECUDA,                         \
                      std::string(#call) + ": " + cudaGetErrorString(e_)};                            \
  } while (0)

template <typename T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;
  bool owned = true;  // false: a view into memory someone else frees
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (p && owned) cudaFree(p);
    p = nullptr;
    n = 0;
    owned = true;
  }
  void view(void* at, size_t count) {
    release();
    p = static_cast<T*>(at);
    n = count;
    owned = false;
  }
  // Grow-only, contents undefined.  A buffer that must grow takes a quarter
  // more than asked: the scratch of a stream of searches (survivor lists,
  // envelope planes) varies from call to call, and each regrowth is a
  // cudaFree -- which waits for the whole device -- and a fresh cudaMalloc.
  void alloc(size_t count) {
    if (count <= n && p) return;
    release();
    const size_t want = std::max<size_t>(count, 1);
    const size_t ask = want + want / 4;
    if (cudaMalloc(&p, ask * sizeof(T)) == cudaSuccess) {
      n = ask;
      return;
    }
    cudaGetLastError();
    p = nullptr;
    CK(cudaMalloc(&p, want * sizeof(T)));
    n = want;
  }
  void upload(const T* src, size_t count, cudaStream_t s) {
    alloc(count);
    if (count) CK(cudaMemcpyAsync(p, src, count * sizeof(T), cudaMemcpyHostToDevice, s));
  }
};

// Page-locked host buffer (grow-only): device-to-host copies into it run at
// full link speed and never fault in fresh pages.
template <typename T>
struct PinnedBuf {
  T* p = nullptr;
  size_t n = 0;
  PinnedBuf() = default;
  PinnedBuf(const PinnedBuf&) = delete;
  PinnedBuf& operator=(const PinnedBuf&) = delete;
  ~PinnedBuf() { release(); }
  void release() {
    if (p) cudaFreeHost(p);
    p = nullptr;
    n = 0;
  }
  void alloc(size_t count) {
    if (count <= n && p) return;
    release();
    CK(cudaHostAlloc((void**)&p, std::max<size_t>(count, 1) * sizeof(T), cudaHostAllocDefault));
    n = std::max<size_t>(count, 1);
  }
};

// Launch tables of every kernel instantiation (filled once).
const KernelTables& kernels();

// Smallest f32 statistic s with pass(s) true, assuming pass is monotone
// (false below the boundary, true above); +inf if it never passes, -inf if it
// always passes on the finite range.
template <typename Pred>
float f32_boundary(Pred pass) {
  auto key = [](float f) {
    int32_t i;
    memcpy(&i, &f, 4);
    return i >= 0 ? i : (int32_t)(0x80000000u - (uint32_t)i) * -1;  // monotone int order
  };
  (void)key;
  // order-preserving map float <-> int64 over finite floats
  auto to_ord = [](float f) -> int64_t {
    uint32_t u;
    memcpy(&u, &f, 4);
    return (u & 0x80000000u) ? -(int64_t)(u & 0x7fffffffu) : (int64_t)u;
  };
  auto from_ord = [](int64_t o) -> float {
    uint32_t u = o < 0 ? (0x80000000u | (uint32_t)(-o)) : (uint32_t)o;
    float f;
    memcpy(&f, &u, 4);
    return f;
  };
  int64_t lo = to_ord(-3.0e38f), hi = to_ord(3.0e38f);
  if (pass(from_ord(lo))) return -INFINITY;
  if (!pass(from_ord(hi))) return INFINITY;
  while (hi - lo > 1) {  // invariant: !pass(lo), pass(hi)
    const int64_t mid = lo + (hi - lo) / 2;
    if (pass(from_ord(mid))) hi = mid;
    else lo = mid;
  }
  return from_ord(hi);
}

// Device blocks recycled between target sets, so that a caller streaming
// batches of targets through one engine does not pay a cudaMalloc/cudaFree
// pair (and the device-wide synchronisation of cudaFree) per batch.
class BlockPool {
 public:
  ~BlockPool() {
    for (auto& b : free_) cudaFree(b.first);
  }
  // A block of at least `bytes`; its size is returned in `got`.
  void* take(size_t bytes, size_t& got) {
    {
      std::lock_guard<std::mutex> g(mu_);
      size_t best = free_.size();
      for (size_t i = 0; i < free_.size(); i++)
        if (free_[i].second >= bytes && (best == free_.size() || free_[i].second < free_[best].second)) best = i;
      if (best < free_.size()) {
        auto b = free_[best];
        free_.erase(free_.begin() + (std::ptrdiff_t)best);
        got = b.second;
        return b.first;
      }
    }
    void* p = nullptr;
    CK(cudaMalloc(&p, std::max<size_t>(bytes, 256)));
    got = std::max<size_t>(bytes, 256);
    return p;
  }
  void give(void* p, size_t bytes) {
    std::lock_guard<std::mutex> g(mu_);
    free_.emplace_back(p, bytes);
    if (free_.size() > kKeep) {  // drop the smallest
      auto it = std::min_element(free_.begin(), free_.end(),
                                 [](const auto& a, const auto& b) { return a.second < b.second; });
      cudaFree(it->first);
      free_.erase(it);
    }
  }

 private:
  static constexpr size_t kKeep = 2;
  std::mutex mu_;
  std::vector<std::pair<void*, size_t>> free_;
};

// A main stream with auxiliary streams that fan out from it and join back
// into it, all of one scheduling priority.
struct Streams {
  static constexpr int kAux = 8;
  int naux = kAux;  // auxiliary streams in use
  cudaStream_t main = nullptr;
  cudaStream_t aux[kAux] = {};  // independent launches (shapes, bins) run side by side
  cudaEvent_t fork_ev = nullptr, join_ev[kAux] = {};
  void create(int priority, int n_aux) {
    naux = std::max(1, std::min(n_aux, kAux));
    CK(cudaStreamCreateWithPriority(&main, cudaStreamNonBlocking, priority));
    for (int a = 0; a < naux; a++) {
      CK(cudaStreamCreateWithPriority(&aux[a], cudaStreamNonBlocking, priority));
      CK(cudaEventCreateWithFlags(&join_ev[a], cudaEventDisableTiming));
    }
    CK(cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming));
  }
  void destroy() {
    if (main) cudaStreamSynchronize(main);
    for (int a = 0; a < naux; a++)
      if (aux[a]) cudaStreamSynchronize(aux[a]);
    for (int a = 0; a < naux; a++) {
      if (aux[a]) cudaStreamDestroy(aux[a]);
      if (join_ev[a]) cudaEventDestroy(join_ev[a]);
    }
    if (fork_ev) cudaEventDestroy(fork_ev);
    if (main) cudaStreamDestroy(main);
  }
};

// Set once a host job has copied a slot's row buffers out; the engine thread
// waits for it before it reuses those buffers for a later block.
struct RowsTicket {
  std::mutex mu;
  std::condition_variable cv;
  bool done = false;
  void set() {
    {
      std::lock_guard<std::mutex> g(mu);
      done = true;
    }
    cv.notify_all();
  }
  void wait() {
    std::unique_lock<std::mutex> g(mu);
    cv.wait(g, [&] { return done; });
  }
};

// Streams, events and survivor lists of one block of a search.  A search
// keeps two blocks in flight: block b+1's MSV runs on one slot while block
// b's later stages, row passes and host re-check use the other.  MSV goes to
// the low-priority streams, everything after it to the high-priority ones,
// so the short, latency-bound later stages of block b get SMs as soon as
// block b+1's MSV CTAs retire and MSV fills the rest of the GPU.
struct Slot {
  Streams hi, lo;
  cudaEvent_t ev[8] = {};
  cudaEvent_t msv_done = nullptr;
  // grow-only device scratch
  DevBuf<PairRec> lists[4];
  DevBuf<BinRegion> bins[4];
  DevBuf<unsigned> counts;  // 4 stages x kMaxBins
  DevBuf<unsigned> overflow;
  DevBuf<unsigned> cursor;  // kMaxBins pair cursors of the Viterbi launches
  DevBuf<double> cells;     // DP cells entering each stage (stats)
  DevBuf<MsvTile> tiles;
  DevBuf<sxk::PackedTile> ptiles;  // packed pre-screen tiles
  DevBuf<int32_t> rlist;           // pre-screen survivors: target indices, rcap per profile of the block
  DevBuf<unsigned> rcount;         // survivors per profile of the block
  cudaEvent_t pre_done = nullptr;  // pre-screen finished (its time, for the stats)
  // packed Viterbi pre-screen: the bias filter's survivors of pre-screened
  // profiles, vcap per profile of the block, and the pre-screen's tiles
  DevBuf<PairRec> vlist;
  DevBuf<unsigned> vcount;
  DevBuf<sxk::VitTile> vtiles;
  DevBuf<double> vstats;           // cells bounded, cells passed, pairs passed
  cudaEvent_t bias_done = nullptr, vpre_done = nullptr;
  // Forward/Backward row passes of the block's final pairs, in buffers of
  // their own: the engine thread queues them and moves on to the next block;
  // a host job waits for them, copies the rows out and releases the buffers.
  DevBuf<sxk::RowRec> rrecs;
  DevBuf<float> rows;
  cudaEvent_t rows_t0 = nullptr, rows_t1 = nullptr;
  cudaStream_t rows_copy = nullptr;  // device-to-host copies of the rows (host job)
  std::shared_ptr<RowsTicket> rows_busy;
  void create() {
    int least = 0, greatest = 0;
    CK(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    // 2 slots x (9 + 6) streams + 1 envelope stream = 31, within the 32
    // hardware work queues a process can have (CUDA_DEVICE_MAX_CONNECTIONS=32):
    // with fewer queues, streams share them and a high-priority launch can
    // wait behind queued MSV work
    hi.create(greatest, 8);
    lo.create(least, 5);
    for (auto& e : ev) CK(cudaEventCreate(&e));
    CK(cudaEventCreate(&pre_done));
    CK(cudaEventCreate(&bias_done));
    CK(cudaEventCreate(&vpre_done));
    CK(cudaEventCreate(&rows_t0));
    CK(cudaEventCreate(&rows_t1));
    CK(cudaStreamCreateWithFlags(&rows_copy, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&msv_done, cudaEventDisableTiming));
  }
  void destroy() {
    hi.destroy();
    lo.destroy();
    for (auto& e : ev)
      if (e) cudaEventDestroy(e);
    if (msv_done) cudaEventDestroy(msv_done);
    if (pre_done) cudaEventDestroy(pre_done);
    if (bias_done) cudaEventDestroy(bias_done);
    if (vpre_done) cudaEventDestroy(vpre_done);
    if (rows_busy) rows_busy->wait();
    if (rows_t0) cudaEventDestroy(rows_t0);
    if (rows_t1) cudaEventDestroy(rows_t1);
    if (rows_copy) {
      cudaStreamSynchronize(rows_copy);
      cudaStreamDestroy(rows_copy);
    }
  }
};

}  // namespace sxe

using namespace sxe;

// ---- engine objects ----------------------------------------------------------
struct sx_engine {
  int device = 0;
  int host_threads = 1;
  std::unique_ptr<WorkerPool> pool;
  uint32_t flags = 0;
  int64_t batch_bytes = 0;
  int num_sms = 148;
  static constexpr int kAux = Streams::kAux;
  Slot sl[2];
  // slot 0 under the names the single-batch entry points use
  cudaStream_t& stream = sl[0].hi.main;
  cudaStream_t (&aux)[kAux] = sl[0].hi.aux;
  cudaEvent_t& fork_ev = sl[0].hi.fork_ev;
  cudaEvent_t (&join_ev)[kAux] = sl[0].hi.join_ev;
  cudaEvent_t (&ev)[8] = sl[0].ev;
  DevBuf<PairRec> (&lists)[4] = sl[0].lists;
  DevBuf<BinRegion> (&bins)[4] = sl[0].bins;
  DevBuf<unsigned>& counts = sl[0].counts;
  DevBuf<unsigned>& overflow = sl[0].overflow;
  DevBuf<MsvTile>& tiles = sl[0].tiles;
  std::mutex mu;
  sx_search_stats stats{};
  int pipeline_blocks = 0;  // profile blocks per search; 0 = by workload size
  // kernel shape per profile length, set by a tuner (sx_set_shape_table):
  // [0] MSV, [1] Viterbi; empty or -1 = the built-in choice
  std::vector<int16_t> shape_table[2];
  int64_t mem_free = 0;     // device memory free when the engine was created
  // Lifetime: profile and target sets point at their engine.  sx_destroy
  // releases the engine's streams at once, but the engine object itself lives
  // until the last of its sets is freed, so a set freed after its engine (a
  // garbage-collected binding, say) never touches freed memory.
  std::mutex life_mu;
  int64_t live_sets = 0;
  bool destroyed = false;
  BlockPool target_blocks;  // device memory of freed target sets
  HostBytePool target_bytes;  // host residue buffers of freed target sets
  HostBytePool row_bytes{256u << 20};  // host copies of the row passes (a chunk, or one very long pair)
  // envelope passes of the host domain definition (used by the host pool's
  // driver thread, one batch at a time)
  cudaStream_t env_stream = nullptr;  // the passes' copies; their launches fan out over the slots' streams
  cudaEvent_t env_ev = nullptr;
  DevBuf<sxk::EnvRec> env_recs;
  DevBuf<float> env_planes, env_rows, env_aux, env_out;
  DevBuf<double> env_fac;
  DevBuf<sxk::TraceRec> trc_recs;  // stochastic-trace passes of multi-domain regions
  DevBuf<int32_t> trc_pool, trc_count, trc_status;
  DevBuf<float> trc_cols;
  DevBuf<sxk::LongPair> long_pairs;  // pairs of profiles longer than kMaxM
  DevBuf<float> long_scratch, long_out, long_rows_f, long_rows_b;
  DevBuf<int64_t> long_row_off;
  DevBuf<Thresholds> thr;
  DevBuf<float> scores;
  DevBuf<int32_t> slots, plist;
  DevBuf<sxk::AdjPair> adj_pairs;
  DevBuf<float> adj_f, adj_acc, adj_out;
  PinnedBuf<float> adj_host;  // staging of the adjoint's counts on their way to the caller
  PinnedBuf<double> adj_lnz_host;
  DevBuf<double> adj_d, adj_lnz;
};

struct sx_profiles {
  sx_engine* eng = nullptr;
  ProfileList h;
  std::vector<DevProfile> dp;
  std::vector<int64_t> plain_off;  // float offsets of the plain images
  std::vector<int> msv_shape;
  DevBuf<DevProfile> d_prof;
  DevBuf<sxk::PlainProfile> d_pprof;  // plain one-pair-per-block layout
  DevBuf<float> d_plain;
  DevBuf<float4> d_msv;
  DevBuf<uint2> d_qimg;  // quantized MSV images of the pre-screen (int16, 4 columns per uint2)
  DevBuf<float4> d_vit;  // Viterbi lane-group images
  DevBuf<uint4> d_qvimg;  // quantized Viterbi images of the packed pre-screen
  DevBuf<float> d_vfb;
  DevBuf<float> d_x;  // row images of the exact row passes
  DevBuf<double> d_bias;
  // the filter thresholds of the last search options seen (they depend on the
  // profiles' statistics and F1/F2/F3 alone): a stream of searches with one
  // configuration computes them once
  mutable std::mutex th_mu;
  mutable std::vector<Thresholds> th_cache;
  mutable double th_key[4] = {-1, -1, -1, -1};
};

struct sx_targets {
  sx_engine* eng = nullptr;
  std::vector<std::string> ids;  // caller's names (sx_targets_create); empty for digital sets
  HostBytes dsq;  // packed digital residues, each target 16-byte aligned (page-locked)
  std::vector<int64_t> off;
  std::vector<int32_t> len;
  std::vector<int32_t> order;  // indices sorted by length, longest first
  double residues = 0;
  DevBuf<uint8_t> d_res;
  DevBuf<int64_t> d_off;
  DevBuf<int32_t> d_len;
  DevBuf<float4> d_tpar;  // MSV tloop, tmove, null score
  DevBuf<float4> d_xsc;   // multihit loop, move (log), loop, move (prob)
  DevBuf<int32_t> d_order;
  void* block = nullptr;  // one device block holding all d_* arrays (engine pool)
  size_t block_bytes = 0;
  ~sx_targets() {
    if (block) eng->target_blocks.give(block, block_bytes);
    eng->target_bytes.give(std::move(dsq));
  }
};

struct sx_hits {
  std::vector<sx_hit> hits;
  std::vector<sx_domain> doms;
};

namespace sxe {

constexpr float kSlackBits = 1.0e-3f;  // device-log decisions: never reject what the reference keeps

struct FinalPair {
  int32_t p, t;
  float usc, filtersc, vsc;
  int32_t slot;
};

// Raw Forward/Backward special rows of a chunk of pairs: how the device passes
// are laid out (records sorted by shape, then longest first) and, once they
// are done, the rows' host copy.
struct RowsChunk {
  std::vector<sxk::RowRec> recs;
  std::vector<size_t> which;  // record q's index in the caller's list
  std::vector<int64_t> boff;  // offset of its Backward rows
  size_t first[kNumXShapes + 1] = {};  // records of shape s: first[s] .. first[s+1]
  int longest[kNumXShapes] = {};       // rows of the longest one
  int64_t floats = 0;
  // The copy goes to a page-locked buffer of the engine's pool: tens of MB of
  // rows arrive at the link's rate and no page of fresh memory is touched.
  HostBytePool* pool = nullptr;
  HostBytes rows;
  RowsChunk() = default;
  RowsChunk(RowsChunk&&) = default;
  RowsChunk& operator=(RowsChunk&&) = delete;
  ~RowsChunk() {
    if (pool) pool->give(std::move(rows));
  }
  const float* data() const { return reinterpret_cast<const float*>(rows.data()); }
  const float* fwd(size_t q) const { return data() + recs[q].row_off; }
  const float* bwd(size_t q) const { return data() + boff[q]; }
  void fetch(HostBytePool& from, const float* dev, cudaStream_t s) {
    const size_t bytes = sizeof(float) * (size_t)floats;
    pool = &from;
    rows = from.take(bytes);
    rows.resize(bytes);
    CK(cudaMemcpyAsync(rows.data(), dev, bytes, cudaMemcpyDeviceToHost, s));
    CK(cudaStreamSynchronize(s));
  }
};
// floats of one pair's rows, both directions
inline int64_t row_floats(int64_t l) { return 12 * (l + 1); }

// One batch's requests and the places for their results.
struct EnvSource {
  const DomainBatch* db;
  const std::vector<EnvRequest>* reqs;
  std::vector<EnvFactors>* F;
  std::vector<EnvDeviceOut>* D;
};

struct RegionSource {
  DomainBatch* db;
  const std::vector<RegionRequest>* regs;
};
struct RegionPassStats {
  int64_t launches = 0, device = 0, redone = 0;
  double cells = 0;
};

int vit_threads(int num_sms, int shape, unsigned n);
int vit_blocks(int num_sms, int shape, unsigned n, int threads);
unsigned scan_ctas(unsigned n);
std::vector<int16_t> default_shape_table(int kind);
int shape_for(const sx_engine* E, int kind, int m);
void pack_profiles(sx_profiles* P);
void pack_targets(sx_targets* T);
void append_target(sx_targets* T, const uint8_t* dig, size_t l);
std::vector<Thresholds> make_thresholds(const ProfileList& H, const SearchOpts& o);
std::vector<Thresholds> thresholds_of(const sx_profiles* P, const SearchOpts& o);
void combine_profiles(sx_profiles* P, const sx_profiles* const* sets, size_t n, const SearchOpts& o);
void allow_shared_memory();
void fork_aux(Streams& X);
void join_aux(Streams& X);
void note_free_memory(sx_engine* E);
int64_t scratch_budget(const sx_engine* E, int64_t want);
int report(const sx_profiles* P, const sx_targets* T, const sx_search_cfg* cfg,
           std::vector<std::vector<std::pair<int32_t, HitOut>>>& per_profile, sx_hits* out);
int check_cutoffs(const sx_profiles* P, int kind);
size_t msv_smem(int s);
void launch_msv(sx_engine* E, Slot& S, Streams& X, const sx_profiles* P, const sx_targets* T, const std::vector<std::vector<MsvTile>>& tiles,
                const int32_t* d_list, float* d_scores, const int32_t* d_slot, PairRec* surv, const BinRegion* bins,
                unsigned* counts, const unsigned* rcount = nullptr, unsigned rcap = 0, int p0 = 0);
double elapsed_ms(cudaEvent_t a, cudaEvent_t b);
int long_grid(const sx_engine* E, size_t n);
int64_t long_stride(const sx_profiles* P, const std::vector<sxk::LongPair>& v, size_t a, size_t b);
void long_scores(sx_engine* E, const sx_profiles* P, const sx_targets* T, const std::vector<sxk::LongPair>& v,
                 bool viterbi, std::vector<float>& out);  // v: any profiles of M > kMaxM
SearchOpts search_opts(const sx_search_cfg* cfg);
int run_search(sx_engine* E, const sx_profiles* P, const sx_targets* T, const sx_search_cfg* cfg, sx_hits* out);
int64_t envelope_passes(sx_engine* E, const sx_profiles* P, const sx_targets* T, std::vector<EnvSource>& srcs,
                        int nthr, PhaseLog* plog = nullptr);
RegionPassStats region_passes(sx_engine* E, const sx_profiles* P, const sx_targets* T,
                              std::vector<RegionSource>& srcs, int nthr);

// Device Forward and Backward with row output for `pairs`, in chunks bounded
// by the scratch budget; hands each chunk's host copy to consume(RowsChunk&&)
// as soon as it has arrived.
void rows_pass(sx_engine* E, Slot& S, const sx_profiles* P, const sx_targets* T, const std::vector<FinalPair>& pairs,
               const std::function<void(RowsChunk&&)>& consume);

// rows_pass with each chunk consumed on the calling thread: sink(i, fwd_rows,
// bwd_rows) for every pair, spread over the engine's host threads.
template <typename Sink>
void rows_pass_sync(sx_engine* E, const sx_profiles* P, const sx_targets* T, const std::vector<FinalPair>& pairs,
                    Sink&& sink) {
  rows_pass(E, E->sl[0], P, T, pairs, [&](RowsChunk&& c) {
    E->pool->run(c.which.size(), E->host_threads, [&](size_t q) { sink(c.which[q], c.fwd(q), c.bwd(q)); });
  });
}

// Raw Forward/Backward special rows of pairs of profiles past the exact row
// shapes, in chunks bounded by the scratch budget; consume(first, n, fwd, bwd,
// off) per chunk, pair first + q having its rows at fwd + off[q] and bwd + off[q].
using LongRowsSink = std::function<void(size_t, size_t, const float*, const float*, const std::vector<int64_t>&)>;
void long_rows(sx_engine* E, const sx_profiles* P, const sx_targets* T, const std::vector<sxk::LongPair>& v,
               const LongRowsSink& consume);

}  // namespace sxe
