// MSV and Viterbi of profiles wider than the lane-group kernels' 2048 columns
// (up to 8192): a CTA per pair, thread t holding columns t*C+1 .. t*C+C in
// registers, the scores read as float4 rows of the profile's row image.  The
// arithmetic is the reference's (src/hmmer/dp.rs:92-189): maxima are exact in
// any order, and the Viterbi D chain D[k+1] = max(M[k] + t_md, D[k] + t_dd)
// runs as the Forward one does (exact_rows.cuh) -- every lane at once from the
// carry its left neighbour had, repeated until no carry changes.  A row costs
// its barriers (one for MSV, two for Viterbi) and a few rounds of C columns.
// Measured on B200 against the kernels that kept the row in global scratch and
// ran the chain by one thread (still the ones past 8192 columns; two profiles of
// M 2,100 and 2,500 x 300 targets of up to 3,000 residues): MSV of 600 pairs
// 7.0 -> 0.76 ms, Viterbi of 36 pairs 196 -> 4.4 ms, and with the exact row
// shapes Forward and Backward of the 9 final pairs 565 -> 9.5 ms.
#pragma once
#include "exact_rows.cuh"

namespace sxk {

// further rows of a wide profile's image, -inf past column M
enum : int {
  kXMsc = kXRows,       // 25 rows: match log-odds
  kXVit = kXMsc + 25,   // log transitions: bm, mm im dm into the column, mi ii, md dd out of it
  kXWideRows = kXVit + 8
};

struct LongPair {
  int32_t p, t;
};

// Maximum over the CTA of every thread's v, through smx[warp]; the caller's
// barrier stands between this warp's write and the read.
__device__ __forceinline__ int order_key(float v) {  // monotone, its own inverse on the bits
  const int k = __float_as_int(v);
  return k ^ ((k >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float from_key(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
__device__ __forceinline__ float team_max(const int* smx, int lane, int nw) {
  return from_key(__reduce_max_sync(kFull, smx[lane < nw ? lane : 0]));
}

template <int C>
__global__ void __launch_bounds__(32 * kXMaxWarps) wide_msv_kernel(
    const LongPair* __restrict__ pairs, const DevProfile* __restrict__ profs, const float* __restrict__ ximg,
    const uint8_t* __restrict__ res, const int64_t* __restrict__ toff, const int32_t* __restrict__ tlen,
    const float4* __restrict__ tpar, float* __restrict__ out) {
  __shared__ float last[2][kXMaxWarps];  // the warps' last columns, by row parity
  __shared__ int smx[2][kXMaxWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int width = blockDim.x * C;
  const LongPair q = pairs[blockIdx.x];
  const DevProfile& P = profs[q.p];
  const float* im = ximg + P.x_off + (int64_t)kXMsc * width + threadIdx.x * C;
  const float tbm = P.msv_tbm;
  const uint8_t* s = res + toff[q.t];
  const int L = tlen[q.t];
  const float4 tp = tpar[q.t];
  float prev[C], e[C];
#pragma unroll
  for (int c = 0; c < C; c++) prev[c] = SX_NEG_INF;
  float xn = 0.f, xb = tp.y, xj = SX_NEG_INF, left = SX_NEG_INF;  // left: the left warp's last column (lane 0)
  load_cols<C>(im + (L > 0 ? __ldg(s) : 24) * width, e);
  for (int i = 0; i < L; i++) {
    float en[C];
    load_cols<C>(im + (i + 1 < L ? __ldg(s + i + 1) : 24) * width, en);
    const float be = fadd(xb, tbm);
    float l = __shfl_up_sync(kFull, prev[C - 1], 1);
    if (lane == 0) l = left;
    float xe = SX_NEG_INF;
#pragma unroll
    for (int c = C - 1; c >= 0; c--) {
      prev[c] = fadd(e[c], fmx(c ? prev[c - 1] : l, be));
      xe = fmx(xe, prev[c]);
      e[c] = en[c];
    }
    const int key = __reduce_max_sync(kFull, order_key(xe));
    if (lane == 31) {
      last[i & 1][warp] = prev[C - 1];
      smx[i & 1][warp] = key;
    }
    __syncthreads();
    xe = team_max(smx[i & 1], lane, nw);
    if (lane == 0 && warp) left = last[i & 1][warp - 1];
    // xc == xj, and max(xn + t, xj + t) == max(xn, xj) + t (as in msv_kernel)
    xj = fmx(fadd(xj, tp.x), fadd(xe, -kLn2));
    xn = fadd(xn, tp.x);
    xb = fadd(fmx(xn, xj), tp.y);
  }
  if (threadIdx.x == 0) out[blockIdx.x] = L > 0 ? fadd(xj, tp.y) : SX_NEG_INF;
}

// Ascending max-plus D chain of a warp whose first column has D = `in`.
template <int C>
__device__ __forceinline__ float settle_max(float (&d)[C], const float (&a)[C], const ColVec<C>& t, float cin, float in,
                                            int lane) {
  float v = 0.f;
  for (int it = 0; it < 32; it++) {
    v = cin;
#pragma unroll
    for (int c = 0; c < C; c++) {
      d[c] = v;
      v = fmx(a[c], fadd(v, t[c]));
    }
    const float up = __shfl_up_sync(kFull, v, 1);
    const float nc = lane ? up : in;
    if (__all_sync(kFull, same_bits(nc, cin))) break;
    cin = nc;
  }
  return v;
}

template <int C, TransIn IN>
__global__ void __launch_bounds__(32 * kXMaxWarps) wide_viterbi_kernel(
    const LongPair* __restrict__ pairs, const DevProfile* __restrict__ profs, const float* __restrict__ ximg,
    const uint8_t* __restrict__ res, const int64_t* __restrict__ toff, const int32_t* __restrict__ tlen,
    const float4* __restrict__ xsc, float* __restrict__ out) {
  extern __shared__ float4 sm_row[];  // the transition rows (kTrShared)
  __shared__ XShared sh;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int width = blockDim.x * C, k0 = threadIdx.x * C;
  const LongPair q = pairs[blockIdx.x];
  const DevProfile& P = profs[q.p];
  const float* img = ximg + P.x_off;
  const float* im = img + (int64_t)kXMsc * width + k0;
  const float* tv = img + (int64_t)kXVit * width + k0;
  const uint8_t* s = res + toff[q.t];
  const int L = tlen[q.t];
  const float4 xs = xsc[q.t];
  float* st = reinterpret_cast<float*>(sm_row) + k0;
  if constexpr (IN == kTrShared) {  // every thread reads back its own columns only
#pragma unroll
    for (int r = 0; r < 8; r++) {
      float v[C];
      load_cols<C>(tv + r * width, v);
      store_cols<C>(st + r * width, v);
    }
  }
  auto row = [&](int r) {
    ColVec<C> o;
    if constexpr (IN == kTrShared) {
#pragma unroll
      for (int u = 0; u < C / 4; u++) {
        const float4 x = reinterpret_cast<const float4*>(st + r * width)[u];
        o.v[4 * u] = x.x; o.v[4 * u + 1] = x.y; o.v[4 * u + 2] = x.z; o.v[4 * u + 3] = x.w;
      }
    } else {
      load_cols<C>(tv + r * width, o.v);
    }
    return o;
  };
  float mp[C], ip[C], dp[C], e[C];
#pragma unroll
  for (int c = 0; c < C; c++) mp[c] = ip[c] = dp[c] = SX_NEG_INF;
  float lm = SX_NEG_INF, li = SX_NEG_INF, ld = SX_NEG_INF;  // the left warp's last column (lane 0)
  float xn = 0.f, xb = xs.y, xj = SX_NEG_INF;
  if (threadIdx.x == 0) sh.flag = 0;
  __syncthreads();
  int x = L > 0 ? __ldg(s) : 24;
  load_cols<C>(im + x * width, e);
  for (int i = 0; i < L; i++) {
    const int xnext = i + 1 < L ? __ldg(s + i + 1) : 24;
    float en[C];
    load_cols<C>(im + xnext * width, en);
    float mpl = __shfl_up_sync(kFull, mp[C - 1], 1), ipl = __shfl_up_sync(kFull, ip[C - 1], 1);
    float dpl = __shfl_up_sync(kFull, dp[C - 1], 1);
    if (lane == 0) {
      mpl = lm;
      ipl = li;
      dpl = ld;
    }
    float mv[C], iv[C], a[C], dv[C];
    {
      const auto bm = row(0), mm = row(1), imr = row(2), dm = row(3), mi = row(4), ii = row(5);
#pragma unroll
      for (int c = 0; c < C; c++) {
        const float v = fmx(fmx(fadd(c ? mp[c - 1] : mpl, mm[c]), fadd(c ? ip[c - 1] : ipl, imr[c])),
                            fmx(fadd(xb, bm[c]), fadd(c ? dp[c - 1] : dpl, dm[c])));
        mv[c] = fadd(v, e[c]);
        iv[c] = x != 24 ? fmx(fadd(mp[c], mi[c]), fadd(ip[c], ii[c])) : SX_NEG_INF;
      }
    }
    const auto md = row(6), dd = row(7);
    float end = SX_NEG_INF;
#pragma unroll
    for (int c = 0; c < C; c++) {
      a[c] = fadd(mv[c], md[c]);
      end = fmx(a[c], fadd(end, dd[c]));
    }
    float g = __shfl_up_sync(kFull, end, 1);
    end = settle_max<C>(dv, a, dd, lane ? g : SX_NEG_INF, SX_NEG_INF, lane);
    if (lane == 31) sh.end[warp] = end;
    __syncthreads();
    if (warp) {
      const float in = sh.end[warp - 1], own = end;
      g = __shfl_up_sync(kFull, own, 1);
      end = settle_max<C>(dv, a, dd, lane ? g : in, in, lane);
      if (lane == 31 && !same_bits(end, own)) sh.flag = 1;
    }
    auto publish = [&]() {
      float xe = SX_NEG_INF;
#pragma unroll
      for (int c = 0; c < C; c++) xe = fmx3(xe, mv[c], dv[c]);
      const int key = __reduce_max_sync(kFull, order_key(xe));
      if (lane == 31) {
        sh.mx[warp] = key;
        sh.prev[0][warp] = mv[C - 1];
        sh.prev[1][warp] = iv[C - 1];
        sh.prev[2][warp] = dv[C - 1];
      }
      __syncthreads();
    };
    publish();
    if (sh.flag) {  // a warp's end changed: exchange the ends until none does
      for (int it = 0; it <= kXMaxWarps; it++) {
        const float own = end;
        if (lane == 31) sh.end[warp] = own;
        __syncthreads();
        const float in = warp ? sh.end[warp - 1] : SX_NEG_INF;
        g = __shfl_up_sync(kFull, own, 1);
        end = settle_max<C>(dv, a, dd, lane ? g : in, in, lane);
        if (!__syncthreads_or(lane == 31 && !same_bits(end, own))) break;
      }
      if (threadIdx.x == 0) sh.flag = 0;
      publish();
    }
    const float xe = team_max(sh.mx, lane, nw);
    if (lane == 0 && warp) {
      lm = sh.prev[0][warp - 1];
      li = sh.prev[1][warp - 1];
      ld = sh.prev[2][warp - 1];
    }
    xj = fmx(fadd(xj, xs.x), fadd(xe, -kLn2));
    xn = fadd(xn, xs.x);
    xb = fadd(fmx(xn, xj), xs.y);
#pragma unroll
    for (int c = 0; c < C; c++) {
      mp[c] = mv[c];
      ip[c] = iv[c];
      dp[c] = dv[c];
      e[c] = en[c];
    }
    x = xnext;
  }
  if (threadIdx.x == 0) out[blockIdx.x] = L > 0 ? fadd(xj, xs.y) : SX_NEG_INF;
}

}  // namespace sxk
