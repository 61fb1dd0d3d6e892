// Forward and Backward in the reference's order of operations: the raw special
// rows of final pairs (src/hmmer/dp.rs:229-392) and, with the M and I matrices
// kept, the full-matrix passes of envelopes and multi-domain regions
// (dp.rs:442-601).
//
// A team -- one warp up to 256 columns, a CTA of several warps above -- runs
// one pair in one direction, thread t holding columns t*C+1 .. t*C+C.  What
// bounds a pass is the latency of one row, because the B state of a row needs
// the row's E (Forward) or B (Backward) sum, a sum the reference takes in
// column order.  Three parts of a row are sequential in the reference:
//   * the row sum.  Up to 512 columns it stays sequential, but as one chain of
//     adds over a row laid out in shared memory (4 cycles a term, loads 16
//     terms ahead), not as a baton handed from lane to lane.  Above, most of it
//     runs in parallel (team_sum_wide): while the running sum stays within one
//     binade an add changes it by the term rounded to the sum's ulp, whatever
//     the sum, except that a tie goes by the parity of its last bit;
//   * the D chain D[k] = a_k + p_k D[k-1].  Every lane runs its own columns
//     at once from a guessed carry, then takes the carry its left neighbour
//     computed and runs them again until no lane's carry changes.  A state
//     that no lane changes satisfies the sequential recurrence with every
//     rounding, so the result is the reference's bit for bit; after r rounds
//     the first r lanes are final, so 32 rounds always suffice.  A wrong
//     carry fades by the product of p_k, 0.4 a column in a typical model:
//     a scan of the lanes' transfers gives the first guess and two or three
//     rounds repair its last bits;
//   * the descending D chain of Backward, the same way from the other end.
// A thread's Forward chain starts from the D of its first column and ends with
// the D of its right neighbour's, so it needs no match value but its own.
// Between warps the carry goes through shared memory: each warp runs its D
// chain from carry 0, publishes its end, takes its neighbour's and repairs its
// first lanes; a warp whose own end that changed (its 256 columns did not
// absorb the carry) sets a flag and the CTA repeats the exchange.
//
// Measured on B200 against the lane-to-lane baton it replaced (device time of
// the row passes of one search): marker-set genome (242 pairs, M to 1,500)
// 45.5 -> 6.9 ms, one profile of M = 100 (50 pairs) 1.99 -> 0.45 ms, 64
// profiles of M 60-700 (60 pairs) 11.0 -> 2.0 ms.
//
// The images hold zeros past column M and where node M has no transition, so
// the padding columns need no tests: whatever finite value they hold is
// multiplied by a zero before it reaches a real column.
#pragma once
#include "kernels.cuh"

namespace sxk {

// Row image of a profile: kXRows rows of 32 * C * warps floats (its shape's
// width), column k at index k - 1.
enum : int {
  kXMo = 0,    // 25 rows: match odds mo[x][k]
  kXFwd = 25,  // p_bm[k], p_mm[k-1], p_im[k-1], p_dm[k-1], p_mi[k], p_ii[k], p_md[k-1], p_dd[k-1]
  kXBwd = 33,  // p_mm[k], p_mi[k], p_md[k], p_im[k], p_ii[k], p_dm[k], p_dd[k], p_bm[k]
  kXRows = 41
};
constexpr int kXMaxWarps = 16;

// One pass over a target: rows of 6 floats (N B E J C, rescale factor) go to
// row_off (Forward) and row_off + 6 (lr + 1) (Backward).
struct RowRec {
  int32_t p, t;
  int64_t row_off;
};

// team_sum_wide's exchange, by warp and by thread.
struct XSumShared {
  float total[kXMaxWarps];
  unsigned odd[kXMaxWarps];        // threads that need their exact start
  int inc[2][32 * kXMaxWarps];     // at the last thread of each run: what the run adds to an even / odd sum
};

struct XShared {  // exchange between the warps of a team
  float mv[kXMaxWarps];       // Backward: the first column's match term
  float end[kXMaxWarps];      // D at the warp's end of the chain
  float prev[3][kXMaxWarps];  // M, I, D of the last column
  int mx[kXMaxWarps];
  float sum;
  int flag;
};

template <bool MULTI>
__device__ __forceinline__ void team_sync() {
  if constexpr (MULTI) __syncthreads();
  else __syncwarp();
}

template <int C>
__device__ __forceinline__ void load_cols(const float* __restrict__ p, float (&v)[C]) {
#pragma unroll
  for (int q = 0; q < C / 4; q++) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(p) + q);
    v[4 * q] = x.x;
    v[4 * q + 1] = x.y;
    v[4 * q + 2] = x.z;
    v[4 * q + 3] = x.w;
  }
}
template <int C>
__device__ __forceinline__ void store_cols(float* p, const float (&v)[C]) {
#pragma unroll
  for (int q = 0; q < C / 4; q++)
    reinterpret_cast<float4*>(p)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
}

// Where a thread keeps its columns of the eight transition rows: registers, or
// (teams of more than eight warps have 128 registers a thread) shared memory,
// or the image itself when 8 rows of the team's width do not fit there.
enum TransIn { kTrReg, kTrShared, kTrGlobal };
template <int C>
struct ColVec {
  float v[C];
  __device__ __forceinline__ float operator[](int c) const { return v[c]; }
};
template <int C, TransIn IN, bool BWD>
struct TeamTrans {
  float r[IN == kTrReg ? 8 : 1][C];
  const float* p;
  int width;
  // Forward and optimal accuracy: bm, mm im dm into the column, mi ii, then md
  // dd out of it; Backward: mm mi md im ii dm dd bm
  static __device__ __forceinline__ int image_row(int q) { return BWD ? kXBwd + q : q < 6 ? kXFwd + q : q == 6 ? kXBwd + 2 : kXBwd + 6; }
  __device__ __forceinline__ void init(const float* __restrict__ img, int w, int k0, float* shared) {
    width = w;
    p = IN == kTrShared ? shared + k0 : img + k0;
    if constexpr (IN != kTrGlobal) {
#pragma unroll
      for (int q = 0; q < 8; q++) {
        if constexpr (IN == kTrReg) {
          load_cols<C>(img + image_row(q) * w + k0, r[q]);
        } else {  // every thread reads back its own columns only
          float v[C];
          load_cols<C>(img + image_row(q) * w + k0, v);
          store_cols<C>(shared + q * w + k0, v);
        }
      }
    }
  }
  __device__ __forceinline__ ColVec<C> row(int q) const {
    ColVec<C> o;
    if constexpr (IN == kTrReg) {
#pragma unroll
      for (int c = 0; c < C; c++) o.v[c] = r[q][c];
    } else if constexpr (IN == kTrShared) {
#pragma unroll
      for (int u = 0; u < C / 4; u++) {
        const float4 x = reinterpret_cast<const float4*>(p + q * width)[u];
        o.v[4 * u] = x.x; o.v[4 * u + 1] = x.y; o.v[4 * u + 2] = x.z; o.v[4 * u + 3] = x.w;
      }
    } else {
      load_cols<C>(p + image_row(q) * width, o.v);
    }
    return o;
  }
};

__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_int(a) == __float_as_int(b); }

// t[0] + t[1] + ... + t[n-1] in that order from 0 (n a positive multiple of
// 16); the loads of the next 16 terms overlap the adds of these.
__device__ __forceinline__ float ordered_sum(const float* t, int n) {
  const float4* p = reinterpret_cast<const float4*>(t);
  float4 a[4];
#pragma unroll
  for (int u = 0; u < 4; u++) a[u] = p[u];
  float s = 0.f;
  for (int q = 4; q < n / 4; q += 4) {
    float4 b[4];
#pragma unroll
    for (int u = 0; u < 4; u++) b[u] = p[q + u];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      s = fadd(fadd(fadd(fadd(s, a[u].x), a[u].y), a[u].z), a[u].w);
      a[u] = b[u];
    }
  }
#pragma unroll
  for (int u = 0; u < 4; u++) s = fadd(fadd(fadd(fadd(s, a[u].x), a[u].y), a[u].z), a[u].w);
  return s;
}
// The team's sum of its shared row (n terms), known to every thread; the row
// may be overwritten after the call.
template <bool MULTI>
__device__ __forceinline__ float team_sum(const float* t, int n, XShared& sh) {
  if constexpr (MULTI) {
    if (threadIdx.x < 32) {
      const float s = ordered_sum(t, n);
      if (threadIdx.x == 0) sh.sum = s;
    }
    __syncthreads();
    return sh.sum;
  } else {
    const float s = ordered_sum(t, n);
    __syncwarp();
    return s;
  }
}

// The team's sum of every thread's terms t[0..C), in thread order, bit for bit
// as one chain of adds from 0 would give it; T holds the terms (written by the
// caller, ordered by this function's barriers).
// An approximate prefix sum tells each thread the binades of the running sum at
// its first and after its last term, with a margin (2^-10) well above the
// difference between any two orders of adding 8192 non-negative terms.  Where
// both are one binade, the thread's effect on the sum's bit pattern is an
// integer that depends on the last bit of the sum alone: it runs its chain from
// the binade's first even and first odd value and takes the differences.  These
// compose across the lanes of a run of such threads in a scan.  The other
// threads, a dozen a row where the sum crosses a power of two (in the subnormal
// range there is one "binade", without rounding), are walked in order: the run
// before the thread, an integer, then the thread's own chain of C adds.
// A sum that is infinite or not a number is walked too.
// Measured at M = 1,500 (12 warps): the row passes of 1,800 targets 6.64 ->
// 4.57 ms, their envelope matrices 7.47 -> 5.32 ms; at M = 500 (4 warps) 3.29 ->
// 2.90 and 3.65 -> 2.95 ms.  With a run's two integers loaded beside the thread's
// terms, not after the sum's last bit is known, M = 2,100 to 2,500: 10.5 -> 9.5
// and 12.9 -> 11.7 ms (a software pipeline over the walk's steps: slower, 42
// against 37 ms for that search).
template <int C>
__device__ __forceinline__ float team_sum_wide(const float (&t)[C], const float* T, XShared& sh, XSumShared& ss) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  float own = t[0];
#pragma unroll
  for (int c = 1; c < C; c++) own = fadd(own, t[c]);
  float inc = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(kFull, inc, o);
    if (lane >= o) inc = fadd(inc, v);
  }
  if (lane == 31) ss.total[warp] = inc;
  __syncthreads();
  float before = 0.f;
  for (int q = 0; q < warp; q++) before = fadd(before, ss.total[q]);
  const float up = __shfl_up_sync(kFull, inc, 1);
  const float first = fadd(before, lane ? up : 0.f), last = fadd(before, inc);
  const int e0 = __float_as_int(fmul(first, 0.9990234375f)) >> 23, e1 = __float_as_int(fmul(last, 1.0009765625f)) >> 23;
  const bool odd = e0 != e1 || (unsigned)e1 >= 255u;
  const unsigned om = __ballot_sync(kFull, odd);
  int n0 = 0, n1 = 0;
  {
    const int s0 = e0 << 23, s1 = s0 + 1;
    float a = __int_as_float(s0), b = __int_as_float(s1);
#pragma unroll
    for (int c = 0; c < C; c++) {
      a = fadd(a, t[c]);
      b = fadd(b, t[c]);
    }
    n0 = __float_as_int(a) - s0;
    n1 = __float_as_int(b) - s1;
  }
  const unsigned upto = om & ((2u << lane) - 1u);
  const int head = upto ? 32 - __clz(upto) : 0;  // first lane of this lane's run
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {  // earlier lanes' effect, then this one's
    const int p0 = __shfl_up_sync(kFull, n0, o), p1 = __shfl_up_sync(kFull, n1, o);
    if (lane - o >= head) {
      const int m0 = p0 + (p0 & 1 ? n1 : n0), m1 = p1 + (p1 & 1 ? n0 : n1);
      n0 = m0;
      n1 = m1;
    }
  }
  ss.inc[0][threadIdx.x] = n0;
  ss.inc[1][threadIdx.x] = n1;
  if (lane == 0) ss.odd[warp] = om;
  __syncthreads();
  if (warp == 0) {
    // lane q: warp q's odd threads and the run up to its end
    const unsigned masks = lane < nw ? ss.odd[lane] : 0u;
    const int r0 = lane < nw ? ss.inc[0][32 * lane + 31] : 0, r1 = lane < nw ? ss.inc[1][32 * lane + 31] : 0;
    int s = 0;  // the sum's bits
    for (int q = 0; q < nw; q++) {
      unsigned m = __shfl_sync(kFull, masks, q);
      const int t0 = __shfl_sync(kFull, r0, q), t1 = __shfl_sync(kFull, r1, q);
      int at = 0;
      while (m) {
        const int jn = __ffs(m) - 1, id = 32 * q + jn;
        m &= m - 1;
        const float4* p = reinterpret_cast<const float4*>(T + id * C);
        float4 x[C / 4];
#pragma unroll
        for (int u = 0; u < C / 4; u++) x[u] = p[u];
        if (jn > at) {
          const int i0 = ss.inc[0][id - 1], i1 = ss.inc[1][id - 1];
          s += s & 1 ? i1 : i0;
        }
        float v = __int_as_float(s);
#pragma unroll
        for (int u = 0; u < C / 4; u++) v = fadd(fadd(fadd(fadd(v, x[u].x), x[u].y), x[u].z), x[u].w);
        s = __float_as_int(v);
        at = jn + 1;
      }
      if (at < 32) s += s & 1 ? t1 : t0;
    }
    if (lane == 0) sh.sum = __int_as_float(s);
  }
  __syncthreads();
  return sh.sum;
}
// Teams from kWideSumWarps on take it; two warps are faster with the chain, 4
// cycles a column (M = 300, 2,048 pairs: 6.8 ms, 7.7 in parallel).
constexpr int kWideSumWarps = 3;
template <int C, bool MULTI>
__device__ __forceinline__ float row_sum(const float (&t)[C], const float* T, int n, XShared& sh, XSumShared* ss) {
  if constexpr (MULTI) {
    if ((blockDim.x >> 5) >= kWideSumWarps) return team_sum_wide<C>(t, T, sh, *ss);
  }
  return team_sum<MULTI>(T, n, sh);
}

// Products of the lanes' p_dd for the guess scan: after the call bs[s] is the
// product over the 2^s lanes that end at this one (UP: ascending lanes) and
// `all` the product up to and including this lane; returns the number of scan
// steps whose factor is not negligible.
template <bool UP>
__device__ __forceinline__ int scan_factors(float b, int lane, float (&bs)[5], float& all) {
  int steps = 5;
#pragma unroll
  for (int s = 0; s < 5; s++) {
    const int o = 1 << s;
    bs[s] = b;
    if (steps == 5 && !__any_sync(kFull, b > 1.0e-9f)) steps = s;
    const float n = UP ? __shfl_up_sync(kFull, b, o) : __shfl_down_sync(kFull, b, o);
    if (UP ? lane >= o : lane + o < 32) b = b * n;
  }
  all = b;
  return steps;
}
template <bool UP>
__device__ __forceinline__ float scan_guess(float a, int lane, const float (&bs)[5], int steps) {
#pragma unroll
  for (int s = 0; s < 5; s++) {
    if (s >= steps) break;
    const int o = 1 << s;
    const float n = UP ? __shfl_up_sync(kFull, a, o) : __shfl_down_sync(kFull, a, o);
    if (UP ? lane >= o : lane + o < 32) a = fadd(a, fmul(bs[s], n));
  }
  return UP ? __shfl_up_sync(kFull, a, 1) : __shfl_down_sync(kFull, a, 1);
}

// Ascending D chain of a warp whose first column has D = `in`: rounds from the
// guessed carries `cin` until no carry changes.  a and p are the terms and
// factors out of each column; returns the D right of the lane's last column.
template <int C>
__device__ __forceinline__ float settle_up(float (&d)[C], const float (&a)[C], const ColVec<C>& p, float cin, float in,
                                           int lane) {
  float v = 0.f;
  for (int it = 0; it < 32; it++) {
    v = cin;
#pragma unroll
    for (int c = 0; c < C; c++) {
      d[c] = v;
      v = fadd(a[c], fmul(v, p[c]));
    }
    const float up = __shfl_up_sync(kFull, v, 1);
    const float nc = lane ? up : in;
    if (__all_sync(kFull, same_bits(nc, cin))) break;
    cin = nc;
  }
  return v;
}
// Descending: d[k] = ((a_k + p_k d[k+1]) + e) from `in` past its last column.
template <int C>
__device__ __forceinline__ void settle_down(float (&d)[C], const float (&a)[C], const ColVec<C>& p, float e, float cin,
                                            float in, int lane) {
  for (int it = 0; it < 32; it++) {
    float v = cin;
#pragma unroll
    for (int c = C - 1; c >= 0; c--) d[c] = v = fadd(fadd(a[c], fmul(v, p[c])), e);
    const float dn = __shfl_down_sync(kFull, v, 1);
    const float nc = lane < 31 ? dn : in;
    if (__all_sync(kFull, same_bits(nc, cin))) break;
    cin = nc;
  }
}

// What a pass keeps of the matrices: nothing, the M and I planes (rows 0..L of
// the team's width), or the M, I and D planes in the diagonal layout that the
// stochastic traceback reads.
enum Keep { kKeepNone, kKeepMI, kKeepDiag };

// Diagonal layout of a region's M/I/D planes for the stochastic traceback:
// cell (i, k), 1 <= i <= lr, 1 <= k <= M, at (i - k + M - 1) * M + (k - 1), so
// the cells of a run of match states, (i, k) -> (i-1, k-1), are adjacent.
__host__ __device__ __forceinline__ int64_t diag_at(int64_t i, int k, int M) {
  return (i - k + M - 1) * (int64_t)M + (k - 1);
}
__host__ __device__ __forceinline__ int64_t diag_plane(int64_t lr, int M) { return (lr + M - 1) * (int64_t)M; }

// Forward (dp.rs:229-298, 442-513).
template <int C, bool MULTI, TransIn IN, Keep KEEP>
__device__ __forceinline__ void exact_forward(const float* __restrict__ img, int M, const uint8_t* __restrict__ s, int L,
                                              float ploop, float pmove, float pe_loop, float pe_move, float* orow,
                                              float* planes, float* T, XShared& sh, XSumShared* ss) {
  const int lane = threadIdx.x & 31;
  const int warp = MULTI ? threadIdx.x >> 5 : 0;
  const int width = (MULTI ? blockDim.x : 32) * C;
  const int k0 = (MULTI ? threadIdx.x : lane) * C;
  const bool lead = MULTI ? threadIdx.x == 0 : lane == 0;
  const int nsum = max(16, (M + 15) & ~15);
  const float* im = img + k0;
  TeamTrans<C, IN, false> tr;
  tr.init(img, width, k0, T + width);
  float* FM = planes;
  float* FI = KEEP == kKeepDiag ? FM + diag_plane(L, M) : FM + (int64_t)(L + 1) * width;
  float* FD = FI + diag_plane(L, M);
  float bs[5], ball, b = 1.f;
  {
    const auto dd = tr.row(7);
#pragma unroll
    for (int c = 0; c < C; c++) b = b * dd[c];
  }
  const int steps = scan_factors<true>(b, lane, bs, ball);
  float bpre = __shfl_up_sync(kFull, ball, 1);
  if (lane == 0) bpre = 1.f;
  float mp[C], ip[C], dp[C], eo[C];
#pragma unroll
  for (int c = 0; c < C; c++) mp[c] = ip[c] = dp[c] = 0.f;
  float lm = 0.f, li = 0.f, ld = 0.f;  // the left warp's last column (lane 0)
  float xn = 1.f, xb = pmove, xj = 0.f, xc = 0.f;
  if (lead) {
#pragma unroll
    for (int q = 0; q < 6; q++) orow[q] = 0.f;
  }
  if (MULTI) {
    if (lead) sh.flag = 0;
    __syncthreads();
  }
  int x = L > 0 ? __ldg(s) : 24, x1 = L > 1 ? __ldg(s + 1) : 24;
  load_cols<C>(im + x * width, eo);
  for (int i = 0; i < L; i++) {
    const int x2 = i + 2 < L ? __ldg(s + i + 2) : 24;
    float eon[C];
    load_cols<C>(im + x1 * width, eon);
    const float ins = x != 24 ? 1.f : 0.f;
    float mpl = __shfl_up_sync(kFull, mp[C - 1], 1), ipl = __shfl_up_sync(kFull, ip[C - 1], 1);
    float dpl = __shfl_up_sync(kFull, dp[C - 1], 1);
    if (lane == 0) {
      mpl = lm;
      ipl = li;
      dpl = ld;
    }
    float mv[C], iv[C], a[C], dv[C];
    {
      const auto bm = tr.row(0), mm = tr.row(1), im = tr.row(2), dm = tr.row(3), mi = tr.row(4), ii = tr.row(5);
#pragma unroll
      for (int c = 0; c < C; c++) {
        float t = fmul(xb, bm[c]);
        t = fadd(t, fmul(c ? mp[c - 1] : mpl, mm[c]));
        t = fadd(t, fmul(c ? ip[c - 1] : ipl, im[c]));
        t = fadd(t, fmul(c ? dp[c - 1] : dpl, dm[c]));
        mv[c] = fmul(t, eo[c]);
        iv[c] = fmul(fadd(fmul(mp[c], mi[c]), fmul(ip[c], ii[c])), ins);
      }
    }
    float end = 0.f;
    const auto md = tr.row(6), dd = tr.row(7);
#pragma unroll
    for (int c = 0; c < C; c++) {
      a[c] = fmul(mv[c], md[c]);
      end = fadd(a[c], fmul(end, dd[c]));
    }
    float g = scan_guess<true>(end, lane, bs, steps);
    if (lane == 0) g = 0.f;
    end = settle_up<C>(dv, a, dd, g, 0.f, lane);
    if constexpr (MULTI) {
      if (lane == 31) sh.end[warp] = end;
      __syncthreads();
      if (warp) {
        const float in = sh.end[warp - 1], own = end;
        float c0 = __shfl_up_sync(kFull, own, 1);
        c0 = lane ? fadd(c0, fmul(bpre, in)) : in;
        end = settle_up<C>(dv, a, dd, c0, in, lane);
        if (lane == 31 && !same_bits(end, own)) sh.flag = 1;
      }
    }
    float t[C];
    auto publish = [&]() {
#pragma unroll
      for (int c = 0; c < C; c++) t[c] = fadd(mv[c], dv[c]);
      store_cols<C>(T + k0, t);
      if (MULTI && lane == 31) {
        sh.prev[0][warp] = mv[C - 1];
        sh.prev[1][warp] = iv[C - 1];
        sh.prev[2][warp] = dv[C - 1];
      }
      team_sync<MULTI>();
    };
    publish();
    if constexpr (MULTI) {
      if (sh.flag) {  // a warp's end changed: exchange the ends until none does
        for (int it = 0; it <= kXMaxWarps; it++) {
          const float own = end;
          if (lane == 31) sh.end[warp] = own;
          __syncthreads();
          const float in = warp ? sh.end[warp - 1] : 0.f;
          const float up = __shfl_up_sync(kFull, own, 1);
          end = settle_up<C>(dv, a, dd, lane ? up : in, in, lane);
          if (!__syncthreads_or(lane == 31 && !same_bits(end, own))) break;
        }
        publish();
      }
    }
    float xe = row_sum<C, MULTI>(t, T, nsum, sh, ss);
    if (MULTI && lead) sh.flag = 0;  // read by all before the sum's barrier, set again after the next row's
    if (MULTI && lane == 0 && warp) {
      lm = sh.prev[0][warp - 1];
      li = sh.prev[1][warp - 1];
      ld = sh.prev[2][warp - 1];
    }
    xj = fadd(fmul(xj, ploop), fmul(xe, pe_loop));
    xc = fadd(fmul(xc, ploop), fmul(xe, pe_move));
    xn = fmul(xn, ploop);
    xb = fadd(fmul(xn, pmove), fmul(xj, pmove));
    float scale = 0.f;
    if (xe > 1.0e4f) {
      const float inv = __fdiv_rn(1.0f, xe);
#pragma unroll
      for (int c = 0; c < C; c++) {
        mv[c] = fmul(mv[c], inv);
        iv[c] = fmul(iv[c], inv);
        dv[c] = fmul(dv[c], inv);
      }
      lm = fmul(lm, inv);
      li = fmul(li, inv);
      ld = fmul(ld, inv);
      xn = fmul(xn, inv);
      xb = fmul(xb, inv);
      xj = fmul(xj, inv);
      xc = fmul(xc, inv);
      scale = xe;
      xe = 1.0f;
    }
    if (lead) {
      float* o = orow + 6 * (int64_t)(i + 1);
      o[0] = xn; o[1] = xb; o[2] = xe; o[3] = xj; o[4] = xc; o[5] = scale;
    }
    if constexpr (KEEP == kKeepMI) {
      store_cols<C>(FM + (int64_t)(i + 1) * width + k0, mv);
      store_cols<C>(FI + (int64_t)(i + 1) * width + k0, iv);
    } else if constexpr (KEEP == kKeepDiag) {
#pragma unroll
      for (int c = 0; c < C; c++) {
        const int k = k0 + c + 1;
        if (k <= M) {
          const int64_t at = diag_at(i + 1, k, M);
          FM[at] = mv[c];
          FI[at] = iv[c];
          FD[at] = dv[c];
        }
      }
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      mp[c] = mv[c];
      ip[c] = iv[c];
      dp[c] = dv[c];
      eo[c] = eon[c];
    }
    x = x1;
    x1 = x2;
  }
}

// Backward (dp.rs:301-392, 516-601): row L (E, C), rows L-1..1 (N B E J C,
// rescale factor) and the row-0 B sum in slot 1 of row 0.
template <int C, bool MULTI, TransIn IN, Keep KEEP>
__device__ __forceinline__ void exact_backward(const float* __restrict__ img, int M, const uint8_t* __restrict__ s,
                                               int L, float ploop, float pmove, float pe_loop, float pe_move,
                                               float* orow, float* planes, float* T, XShared& sh, XSumShared* ss) {
  static_assert(KEEP != kKeepDiag, "only the Forward matrix is kept in the diagonal layout");
  const int lane = threadIdx.x & 31;
  const int warp = MULTI ? threadIdx.x >> 5 : 0;
  const int nw = MULTI ? blockDim.x >> 5 : 1;
  const int width = nw * 32 * C;
  const int k0 = (MULTI ? threadIdx.x : lane) * C;
  const bool lead = MULTI ? threadIdx.x == 0 : lane == 0;
  const int nsum = max(16, (M + 15) & ~15);
  const float* im = img + k0;
  TeamTrans<C, IN, true> tr;
  tr.init(img, width, k0, T + width);
  float bs[5], ball, b = 1.f;
  {
    const auto dd = tr.row(6);
#pragma unroll
    for (int c = 0; c < C; c++) b = b * dd[c];
  }
  const int steps = scan_factors<false>(b, lane, bs, ball);
  float bpre = __shfl_down_sync(kFull, ball, 1);  // product over the lanes right of this one
  if (lane == 31) bpre = 1.f;
  if (lead) {
#pragma unroll
    for (int q = 0; q < 6; q++) orow[q] = 0.f;
  }
  if (L <= 0) return;
  if (MULTI) {
    if (lead) sh.flag = 0;
    __syncthreads();
  }
  float mn[C], in_[C], al[C], dc[C];
  // The row's D chain from al = M(i+1) p_dm and e = E: every thread's dc and
  // the D right of its last column; true if the ends must be exchanged again
  auto d_chain = [&](float e) -> float {
    float end = 0.f;
    const auto dd = tr.row(6);
#pragma unroll
    for (int c = C - 1; c >= 0; c--) end = fadd(fadd(al[c], fmul(end, dd[c])), e);
    float g = scan_guess<false>(end, lane, bs, steps);
    if (lane == 31) g = 0.f;
    settle_down<C>(dc, al, dd, e, g, 0.f, lane);
    float in = 0.f;
    if constexpr (MULTI) {
      if (lane == 0) sh.end[warp] = dc[0];
      __syncthreads();
      if (warp + 1 < nw) {
        in = sh.end[warp + 1];
        const float own = dc[0];
        float c0 = __shfl_down_sync(kFull, own, 1);
        c0 = lane < 31 ? fadd(c0, fmul(bpre, in)) : in;
        settle_down<C>(dc, al, dd, e, c0, in, lane);
        if (lane == 0 && !same_bits(dc[0], own)) sh.flag = 1;
      }
    }
    const float dn = __shfl_down_sync(kFull, dc[0], 1);
    return lane < 31 ? dn : in;
  };
  auto d_again = [&](float e) -> float {  // a warp's end changed
    float in = 0.f;
    const auto dd = tr.row(6);
    for (int it = 0; it <= kXMaxWarps; it++) {
      const float own = dc[0];
      if (lane == 0) sh.end[warp] = own;
      __syncthreads();
      in = warp + 1 < nw ? sh.end[warp + 1] : 0.f;
      const float dn = __shfl_down_sync(kFull, own, 1);
      settle_down<C>(dc, al, dd, e, lane < 31 ? dn : in, in, lane);
      if (!__syncthreads_or(lane == 0 && !same_bits(dc[0], own))) break;
    }
    const float dn = __shfl_down_sync(kFull, dc[0], 1);
    return lane < 31 ? dn : in;
  };
  // row L
  float xc = pmove;
  float xe = fmul(xc, pe_move);
  float xj = 0.f, xn = 0.f;
#pragma unroll
  for (int c = 0; c < C; c++) al[c] = in_[c] = 0.f;
  float dnr = d_chain(xe);
  if constexpr (MULTI) {
    __syncthreads();
    if (sh.flag) dnr = d_again(xe);
    __syncthreads();
    if (lead) sh.flag = 0;
  }
  {
    const auto md = tr.row(2);
#pragma unroll
    for (int c = 0; c < C; c++) mn[c] = fadd(xe, fmul(c < C - 1 ? dc[c + 1] : dnr, md[c]));
  }
  float* BM = planes;
  float* BI = BM + (int64_t)(L + 1) * width;
  if constexpr (KEEP == kKeepMI) {
    store_cols<C>(BM + (int64_t)L * width + k0, mn);
    store_cols<C>(BI + (int64_t)L * width + k0, in_);
  }
  if (lead) {
    float* o = orow + 6 * (int64_t)L;
    o[0] = 0.f; o[1] = 0.f; o[2] = xe; o[3] = 0.f; o[4] = xc; o[5] = 0.f;
  }
  // B sum of row i from M(i+1) and the odds of residue i+1; leaves M(i+1) e in me
  float me[C];
  float bt[C];
  auto b_terms = [&](const float (&eo)[C]) {
    const auto bm = tr.row(7);
#pragma unroll
    for (int c = 0; c < C; c++) {
      me[c] = fmul(mn[c], eo[c]);
      bt[c] = fmul(fmul(mn[c], bm[c]), eo[c]);
    }
    store_cols<C>(T + k0, bt);
    if (MULTI && lane == 0) sh.mv[warp] = me[0];
    team_sync<MULTI>();
  };
  int x = __ldg(s + L - 1), x1 = L > 1 ? __ldg(s + L - 2) : 24;
  float eo[C];
  load_cols<C>(im + x * width, eo);
  for (int i = L - 1; i >= 1; i--) {
    const int x2 = i >= 2 ? __ldg(s + i - 2) : 24;
    float eon[C];
    load_cols<C>(im + x1 * width, eon);
    const float ins = x != 24 ? 1.f : 0.f;
    b_terms(eo);
    float me_up = __shfl_down_sync(kFull, me[0], 1);
    if (lane == 31) me_up = MULTI && warp + 1 < nw ? sh.mv[warp + 1] : 0.f;
    const float xb = row_sum<C, MULTI>(bt, T, nsum, sh, ss);
    xj = fadd(fmul(xj, ploop), fmul(xb, pmove));
    xc = fmul(xc, ploop);
    xe = fadd(fmul(xj, pe_loop), fmul(xc, pe_move));
    xn = fadd(fmul(xn, ploop), fmul(xb, pmove));
    float iv[C];
    {
      const auto dm = tr.row(5);
#pragma unroll
      for (int c = 0; c < C; c++) {
        iv[c] = fmul(in_[c], ins);
        al[c] = fmul(c < C - 1 ? me[c + 1] : me_up, dm[c]);
      }
    }
    dnr = d_chain(xe);
    float rowmax = 0.f;
    auto cells = [&]() {
      rowmax = fmaxf(fmaxf(fmaxf(fmaxf(xb, xe), xn), xj), xc);
      const auto mm = tr.row(0), mi = tr.row(1), md = tr.row(2), im = tr.row(3), ii = tr.row(4);
#pragma unroll
      for (int c = 0; c < C; c++) {
        const float mnext = c < C - 1 ? me[c + 1] : me_up, dnext = c < C - 1 ? dc[c + 1] : dnr;
        mn[c] = fadd(fadd(fadd(fmul(mnext, mm[c]), fmul(iv[c], mi[c])), xe), fmul(dnext, md[c]));
        in_[c] = fadd(fmul(mnext, im[c]), fmul(iv[c], ii[c]));
        rowmax = fmaxf(rowmax, mn[c]);
      }
      // values are never negative, so their bit patterns order as integers
      int mx = __reduce_max_sync(kFull, __float_as_int(rowmax));
      if constexpr (MULTI) {
        if (lane == 0) sh.mx[warp] = mx;
        __syncthreads();
        for (int q = 0; q < nw; q++) mx = max(mx, sh.mx[q]);
      }
      rowmax = __int_as_float(mx);
    };
    cells();
    if constexpr (MULTI) {
      if (sh.flag) {
        dnr = d_again(xe);  // its barriers also order the reads of sh.mx above before the writes below
        cells();
        __syncthreads();
        if (lead) sh.flag = 0;
      }
    }
    float scale = 0.f, xb_o = xb;
    if (rowmax > 1.0e4f) {
      const float inv = __fdiv_rn(1.0f, rowmax);
#pragma unroll
      for (int c = 0; c < C; c++) {
        mn[c] = fmul(mn[c], inv);
        in_[c] = fmul(in_[c], inv);
      }
      xb_o = fmul(xb, inv);
      xe = fmul(xe, inv);
      xn = fmul(xn, inv);
      xj = fmul(xj, inv);
      xc = fmul(xc, inv);
      scale = rowmax;
    }
    if (lead) {
      float* o = orow + 6 * (int64_t)i;
      o[0] = xn; o[1] = xb_o; o[2] = xe; o[3] = xj; o[4] = xc; o[5] = scale;
    }
    if constexpr (KEEP == kKeepMI) {
      store_cols<C>(BM + (int64_t)i * width + k0, mn);
      store_cols<C>(BI + (int64_t)i * width + k0, in_);
    }
#pragma unroll
    for (int c = 0; c < C; c++) eo[c] = eon[c];
    x = x1;
    x1 = x2;
  }
  // row 0: the B sum with residue 1
  b_terms(eo);
  const float b0 = row_sum<C, MULTI>(bt, T, nsum, sh, ss);
  if (lead) orow[1] = b0;
}

// Threads of the largest CTA of a kernel variant.
constexpr int team_threads(TransIn in) { return in == kTrReg ? 256 : 32 * kXMaxWarps; }

// Forward (blockIdx.y = 0) and Backward (1) rows of n pairs.  MULTI: a CTA per
// pair; otherwise a warp per pair.  Dynamic shared memory: one row per team,
// and the transition rows where they are kept there.
template <int C, bool MULTI, TransIn IN>
__global__ void __launch_bounds__(team_threads(IN)) exact_rows_kernel(const RowRec* __restrict__ recs, int n,
                                                         const DevProfile* __restrict__ profs,
                                                         const float* __restrict__ ximg,
                                                         const uint8_t* __restrict__ res,
                                                         const int64_t* __restrict__ toff,
                                                         const int32_t* __restrict__ tlen,
                                                         const float4* __restrict__ xsc, float* __restrict__ rows) {
  extern __shared__ float4 sm_row[];
  __shared__ XShared sh;
  XSumShared* ss = nullptr;
  if constexpr (MULTI) {
    __shared__ XSumShared sum_sh;
    ss = &sum_sh;
  }
  const int w = MULTI ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= n) return;  // uniform over the team
  float* T = reinterpret_cast<float*>(sm_row) + (MULTI ? 0 : (threadIdx.x >> 5) * 32 * C);
  const RowRec r = recs[w];
  const DevProfile& P = profs[r.p];
  const float* img = ximg + P.x_off;
  const int M = P.m, L = tlen[r.t];
  const uint8_t* s = res + toff[r.t];
  const float4 xs = xsc[r.t];
  if (blockIdx.y == 0)
    exact_forward<C, MULTI, IN, kKeepNone>(img, M, s, L, xs.z, xs.w, 0.5f, 0.5f, rows + r.row_off, nullptr, T, sh, ss);
  else
    exact_backward<C, MULTI, IN, kKeepNone>(img, M, s, L, xs.z, xs.w, 0.5f, 0.5f, rows + r.row_off + 6 * (int64_t)(L + 1),
                                        nullptr, T, sh, ss);
}

}  // namespace sxk
