// Adjoint of the Forward score: gradients of lnZ (multihit, target-length
// config; src/hmmer/dp.rs:229-298) with respect to every log-space emission
// and transition score of the profile, i.e. the posterior expected counts
// that posterior decoding (src/hmmer/dp.rs:1278-1306) sums for domain
// definition.
//
// A team per pair (one warp up to 128 columns, a CTA of warps above), thread t
// holding columns 4t+1 .. 4t+4.  Kernel A runs Forward and keeps every S-th
// scaled row (S = ceil(sqrt(L))) plus the scaled special rows; kernel B runs
// Backward from row L down and, segment by segment, recomputes the S Forward
// rows it needs from the segment's checkpoint, so device scratch per pair is
// O(M sqrt(L)).  For each row i it accumulates, with per-row scale factors
// exp(lnF_a + lnB_b - lnZ) whose exponents are formed in f64:
//   emissions  F_M(i,k) B_M(i,k), F_I(i,k) B_I(i,k)
//   into row i F(i-1,k-1) t e(k,x_i) B_M(i,k)   (MM IM DM)  and  F_B(i-1) t_bm e B_M(i,k)
//   within i   F_M/F_D(i,k-1) t B_D(i,k)        (MD DD)
//   to row i+1 F_M/F_I(i,k) t ins(x_{i+1}) B_I(i+1,k)  (MI II)
// Every accumulator belongs to one thread (the owner of the transition's target
// column), so the sums have one order.  D chains are affine scans and row sums
// butterflies (the adjoint is checked against FP64, not bit for bit; Backward and
// the counts take fused multiply-adds, half the roundings).
//
// What bounds it: the latency of a row, two barriers each for a Backward and a
// recomputed Forward row.  Four columns a thread keep the transitions and
// their counts in registers (one warp per pair with 12 columns a lane needed
// 240 and left eight warps on an SM).  The emission counts of a row's residue
// go to scratch rows as reductions that return nothing: as loads, adds and
// stores in place each of a row's 120 updates waited for the one before it, the
// compiler not knowing them apart.  adjoint_out_kernel turns the scratch rows
// into the caller's.  Measured on B200, 4,096 pairs of M = 300, L 400-950, in
// one launch: kernel B 59.5 -> 11.4 ms, kernel A 2.8 -> 2.6; the call, whose
// copies and host split now run beside the kernels, 75 -> 16.4 ms (16.9 without
// the fused operations).
#pragma once
#include "exact_rows.cuh"

namespace sxk {

struct AdjPair {
  int32_t p, t;
  int32_t S;        // checkpoint interval
  int32_t pad;
  int64_t ck_off;   // float offset: floor(L/S)+1 checkpoint rows of M, I, D planes
  int64_t seg_off;  // float offset: S+1 rows of M, I, D planes
  int64_t sp_off;   // float offset: (L+1) x 6 scaled specials (xn xb xe xj xc scale)
  int64_t ls_off;   // double offset: (L+1) cumulative Forward ln scale
  int64_t acc_off;  // float offset: emission counts, 25 match and 25 insert rows of the team's width, zero on entry
  int64_t out_off;  // float offset in the output buffer: d_msc[25][M+1], d_isc[25][M+1], d_tr[8][M+1]
};
constexpr int kAdjEmRows = 50;
constexpr int kAdjC = 4;  // columns per thread
constexpr int adj_warps(int m) { return (m + 32 * kAdjC - 1) / (32 * kAdjC); }
constexpr int kAdjMaxWarps = 16;  // M <= 2048

struct AdjShared {  // exchange between the warps of a team, by use
  float a[kAdjMaxWarps], sum[kAdjMaxWarps], edge[3][kAdjMaxWarps];
  int mx[kAdjMaxWarps];
};

__device__ __forceinline__ void adj_add4(float* p, const float (&v)[4]) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]));
}
__device__ __forceinline__ float ffma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v = fadd(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// A team's view of its profile: transitions at the thread's columns, those of
// the column left of them, and the factors of the D scans.
template <bool MULTI, int C = kAdjC>
struct AdjTeam {
  int lane, warp, nw, k0, M, width;
  const float* im;  // the row image at the thread's first column
  float mm[C], mi[C], md[C], imr[C], ii[C], dm[C], dd[C], bm[C];
  float mm0, im0, dm0;        // out of column k0
  float up[5], dn[5];         // products of dd over the 2^s lanes ending / starting at this one
  float up_in, dn_in, whole;  // products over the lanes before / after this one, over the warp
  __device__ __forceinline__ void init(const float* __restrict__ img, int m, int w) {
    lane = threadIdx.x & 31;
    warp = MULTI ? threadIdx.x >> 5 : 0;
    nw = MULTI ? blockDim.x >> 5 : 1;
    k0 = (MULTI ? threadIdx.x : lane) * C;
    M = m;
    width = w;
    im = img + k0;
    load_cols<C>(im + (kXBwd + 0) * width, mm);
    load_cols<C>(im + (kXBwd + 1) * width, mi);
    load_cols<C>(im + (kXBwd + 2) * width, md);
    load_cols<C>(im + (kXBwd + 3) * width, imr);
    load_cols<C>(im + (kXBwd + 4) * width, ii);
    load_cols<C>(im + (kXBwd + 5) * width, dm);
    load_cols<C>(im + (kXBwd + 6) * width, dd);
    load_cols<C>(im + (kXBwd + 7) * width, bm);
    mm0 = __ldg(im + (kXFwd + 1) * width);
    im0 = __ldg(im + (kXFwd + 2) * width);
    dm0 = __ldg(im + (kXFwd + 3) * width);
    float b = 1.f, all;
#pragma unroll
    for (int c = 0; c < C; c++) b = fmul(b, dd[c]);
    scan_factors<true>(b, lane, up, all);
    up_in = __shfl_up_sync(kFull, all, 1);
    if (lane == 0) up_in = 1.f;
    whole = __shfl_sync(kFull, all, 31);
    scan_factors<false>(b, lane, dn, all);
    dn_in = __shfl_down_sync(kFull, all, 1);
    if (lane == 31) dn_in = 1.f;
  }
  // Every thread's sum, and the largest `key` (of non-negative floats).
  __device__ __forceinline__ float sum_max(float v, float& top, AdjShared& sh) const {
    v = warp_sum(v);
    int mx = __reduce_max_sync(kFull, __float_as_int(top));
    if constexpr (MULTI) {
      if (lane == 0) {
        sh.sum[warp] = v;
        sh.mx[warp] = mx;
      }
      __syncthreads();
      v = sh.sum[0];
      mx = sh.mx[0];
      for (int q = 1; q < nw; q++) {
        v = fadd(v, sh.sum[q]);
        mx = max(mx, sh.mx[q]);
      }
    }
    top = __int_as_float(mx);
    return v;
  }
  // Forward row with residue x, its odds in eo (dp.rs:254-296): (m, i, d) and
  // the specials move to the next row and eo to residue xnext's odds; returns the
  // row's rescale factor (0 if none).  left[3]: M, I, D of the column left of
  // the thread's, in and out.
  __device__ __forceinline__ float forward_row(int x, int xnext, float (&eo)[C], float (&m)[C], float (&i)[C], float (&d)[C], float (&left)[3],
                                               float& xn, float& xb, float& xj, float& xc, float& xe_out, float ploop,
                                               float pmove, AdjShared& sh) const {
    float en[C];
    load_cols<C>(im + xnext * width, en);
    const float ins = x != 24 ? 1.f : 0.f;
    float mv[C], iv[C], dv[C];
    float A = 0.f;
#pragma unroll
    for (int c = 0; c < C; c++) {
      float t = fmul(xb, bm[c]);
      t = fadd(t, fmul(c ? m[c - 1] : left[0], c ? mm[c - 1] : mm0));
      t = fadd(t, fmul(c ? i[c - 1] : left[1], c ? imr[c - 1] : im0));
      t = fadd(t, fmul(c ? d[c - 1] : left[2], c ? dm[c - 1] : dm0));
      mv[c] = fmul(t, eo[c]);
      iv[c] = fmul(fadd(fmul(m[c], mi[c]), fmul(i[c], ii[c])), ins);
      A = fadd(fmul(mv[c], md[c]), fmul(A, dd[c]));  // D right of the column, from a carry of 0
    }
#pragma unroll
    for (int s = 0; s < 5; s++) {
      const float a = __shfl_up_sync(kFull, A, 1 << s);
      if (lane >= 1 << s) A = fadd(A, fmul(up[s], a));
    }
    float cin = __shfl_up_sync(kFull, A, 1);
    if (lane == 0) cin = 0.f;
    if constexpr (MULTI) {
      if (lane == 31) {
        sh.a[warp] = A;
        sh.edge[0][warp] = whole;
        sh.edge[1][warp] = mv[C - 1];
        sh.edge[2][warp] = iv[C - 1];
      }
      __syncthreads();
      float in = 0.f;  // D at the warp's first column
      for (int q = 0; q < warp; q++) in = fadd(sh.a[q], fmul(in, sh.edge[0][q]));
      cin = fadd(cin, fmul(up_in, in));
    }
    float xe = 0.f, v = cin;
#pragma unroll
    for (int c = 0; c < C; c++) {
      dv[c] = v;
      xe = fadd(xe, fadd(mv[c], v));
      v = fadd(fmul(mv[c], md[c]), fmul(v, dd[c]));
    }
    float l0 = __shfl_up_sync(kFull, mv[C - 1], 1), l1 = __shfl_up_sync(kFull, iv[C - 1], 1);
    float l2 = __shfl_up_sync(kFull, dv[C - 1], 1);
    if constexpr (MULTI) {
      if (lane == 0 && warp) {
        l0 = sh.edge[1][warp - 1];
        l1 = sh.edge[2][warp - 1];
      }
    }
    if (lane == 0 && warp == 0) l0 = l1 = l2 = 0.f;
    if constexpr (MULTI) {
      // the left warp's last D goes with its partial sum
      xe = warp_sum(xe);
      if (lane == 0) sh.sum[warp] = xe;
      if (lane == 31) sh.mx[warp] = __float_as_int(dv[C - 1]);
      __syncthreads();
      xe = sh.sum[0];
      for (int q = 1; q < nw; q++) xe = fadd(xe, sh.sum[q]);
      if (lane == 0 && warp) l2 = __int_as_float(sh.mx[warp - 1]);
    } else {
      xe = warp_sum(xe);
    }
    xj = fadd(fmul(xj, ploop), fmul(xe, 0.5f));
    xc = fadd(fmul(xc, ploop), fmul(xe, 0.5f));
    xn = fmul(xn, ploop);
    xb = fadd(fmul(xn, pmove), fmul(xj, pmove));
    float scale = 0.f, inv = 1.f;
    if (xe > 1.0e4f) {
      inv = __fdiv_rn(1.0f, xe);
      xn = fmul(xn, inv);
      xb = fmul(xb, inv);
      xj = fmul(xj, inv);
      xc = fmul(xc, inv);
      scale = xe;
      xe = 1.0f;
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      m[c] = fmul(mv[c], inv);
      i[c] = fmul(iv[c], inv);
      d[c] = fmul(dv[c], inv);
      eo[c] = en[c];
    }
    left[0] = fmul(l0, inv);
    left[1] = fmul(l1, inv);
    left[2] = fmul(l2, inv);
    xe_out = xe;
    return scale;
  }
  // rows of M, I, D planes, `tw` columns each
  __device__ __forceinline__ void store_row(float* base, int tw, const float (&m)[C], const float (&i)[C], const float (&d)[C]) const {
    store_cols<C>(base + k0, m);
    store_cols<C>(base + tw + k0, i);
    store_cols<C>(base + 2 * tw + k0, d);
  }
  __device__ __forceinline__ void load_row(const float* base, int tw, float (&m)[C], float (&i)[C], float (&d)[C]) const {
    auto get = [&](const float* p, float (&v)[C]) {  // plain loads: this kernel wrote them
      static_assert(C == 4, "a float4 a row");
      const float4 x = *reinterpret_cast<const float4*>(p);
      v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    };
    get(base + k0, m);
    get(base + tw + k0, i);
    get(base + 2 * tw + k0, d);
  }
};

// The team's pair: a warp each (four to a CTA) or a CTA.
template <bool MULTI>
__device__ __forceinline__ int adj_pair_index() {
  return MULTI ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
}

// Kernel A: Forward with checkpoints every S rows; writes lnZ.
template <bool MULTI>
__global__ void __launch_bounds__(32 * kAdjMaxWarps) adjoint_forward_kernel(
    const AdjPair* __restrict__ pairs, int npairs, const DevProfile* __restrict__ profs, const float* __restrict__ ximg,
    int width, const uint8_t* __restrict__ res, const int64_t* __restrict__ toff, const int32_t* __restrict__ tlen,
    const float4* __restrict__ xsc, float* __restrict__ fbuf, double* __restrict__ dbuf, double* __restrict__ lnz) {
  constexpr int C = kAdjC;
  __shared__ AdjShared sh;
  const int w = adj_pair_index<MULTI>();
  if (w >= npairs) return;  // uniform over the team
  const AdjPair A = pairs[w];
  AdjTeam<MULTI> T;
  T.init(ximg + profs[A.p].x_off, profs[A.p].m, width);
  const int tw = 32 * C * T.nw, L = tlen[A.t], S = A.S;
  const bool lead = T.lane == 0 && T.warp == 0;
  const uint8_t* s = res + toff[A.t];
  const float4 xs = xsc[A.t];
  const float ploop = xs.z, pmove = xs.w;
  float* ck = fbuf + A.ck_off;
  float* sp = fbuf + A.sp_off;
  double* ls = dbuf + A.ls_off;
  float m[C], i_[C], d[C], left[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int c = 0; c < C; c++) m[c] = i_[c] = d[c] = 0.f;
  float xn = 1.f, xb = pmove, xj = 0.f, xc = 0.f, xe = 0.f;
  double lnscale = 0.0;
  T.store_row(ck, tw, m, i_, d);
  if (lead) {
    sp[0] = xn; sp[1] = xb; sp[2] = 0.f; sp[3] = xj; sp[4] = xc; sp[5] = 0.f;
    ls[0] = 0.0;
  }
  int x = L > 0 ? __ldg(s) : 24, x1 = L > 1 ? __ldg(s + 1) : 24;
  float eo[C];
  load_cols<C>(T.im + x * width, eo);
  for (int i = 1; i <= L; i++) {
    const int x2 = i + 1 < L ? __ldg(s + i + 1) : 24;
    const float scale = T.forward_row(x, x1, eo, m, i_, d, left, xn, xb, xj, xc, xe, ploop, pmove, sh);
    x = x1;
    x1 = x2;
    if (scale > 0.f) lnscale += log((double)scale);
    if (lead) {
      float* o = sp + 6 * (int64_t)i;
      o[0] = xn; o[1] = xb; o[2] = xe; o[3] = xj; o[4] = xc; o[5] = scale;
      ls[i] = lnscale;
    }
    if (i % S == 0) T.store_row(ck + (int64_t)(i / S) * 3 * tw, tw, m, i_, d);
  }
  if (lead) {
    const float v = fmul(xc, pmove);
    lnz[w] = (v > 0.f ? log((double)v) : -INFINITY) + lnscale;
  }
}

// Kernel B: Backward sweep with segment recomputation and count accumulation.
// A Backward row is rescaled when its successor is computed, with that row's
// sum; the factors exp(lnF + lnB - lnZ) carry whichever scale a row has.
template <bool MULTI>
__global__ void __launch_bounds__(32 * kAdjMaxWarps) adjoint_backward_kernel(
    const AdjPair* __restrict__ pairs, int npairs, const DevProfile* __restrict__ profs, const float* __restrict__ ximg,
    int width, const uint8_t* __restrict__ res, const int64_t* __restrict__ toff, const int32_t* __restrict__ tlen,
    const float4* __restrict__ xsc, float* __restrict__ fbuf, const double* __restrict__ dbuf,
    const double* __restrict__ lnz, float* __restrict__ accs, float* __restrict__ out) {
  constexpr int C = kAdjC;
  __shared__ AdjShared sh;
  const int w = adj_pair_index<MULTI>();
  if (w >= npairs) return;  // uniform over the team
  const AdjPair A = pairs[w];
  AdjTeam<MULTI> T;
  T.init(ximg + profs[A.p].x_off, profs[A.p].m, width);
  const int lane = T.lane, warp = T.warp, nw = T.nw, k0 = T.k0, M = T.M, W = T.M + 1;
  const int tw = 32 * C * nw, L = tlen[A.t], S = A.S;
  const int64_t rowf = 3 * (int64_t)tw;
  const uint8_t* s = res + toff[A.t];
  const float4 xs = xsc[A.t];
  const float ploop = xs.z, pmove = xs.w;
  const float* ck = fbuf + A.ck_off;
  float* seg = fbuf + A.seg_off;
  const float* sp = fbuf + A.sp_off;
  const double* lsf = dbuf + A.ls_off;
  const double lz = lnz[w];
  float* acc = accs + A.acc_off + k0;
  // transition counts: into the column MM IM DM MD DD (of the left source), BM, MI, II
  float cmm[C], cim[C], cdm[C], cmd[C], cdd[C], cbm[C], cmi[C], cii[C];
#pragma unroll
  for (int c = 0; c < C; c++) cmm[c] = cim[c] = cdm[c] = cmd[c] = cdd[c] = cbm[c] = cmi[c] = cii[c] = 0.f;
  const float md0 = __ldg(T.im + (kXFwd + 6) * width), dd0 = __ldg(T.im + (kXFwd + 7) * width);  // out of column k0
  const int rows = L > 0 && lz > -INFINITY ? L : 0;
  float mn[C], inx[C];  // Backward row i+1
  float bxc = pmove, bxe = fmul(pmove, 0.5f), bxj = 0.f, bxn = 0.f;
  double lnsb = 0.0;  // cumulative Backward ln scale of row i+1
  int seg_lo = -1;    // first row held in `seg` (rows seg_lo .. seg_lo+S)
  float fm1[C], fi1[C], fd1[C];  // Forward row i
  float eo[C];                   // odds of residue i+1
  int x = 24;                    // residue i+1
  // D chain of a Backward row, descending: D[k] = (al_k + e) + dd_k D[k+1];
  // returns the D right of the thread's last column
  auto d_chain = [&](const float (&al)[C], float e, float (&dc)[C]) -> float {
    float a = 0.f;
#pragma unroll
    for (int c = C - 1; c >= 0; c--) a = ffma(T.dd[c], a, fadd(al[c], e));
#pragma unroll
    for (int q = 0; q < 5; q++) {
      const float n = __shfl_down_sync(kFull, a, 1 << q);
      if (lane + (1 << q) < 32) a = ffma(T.dn[q], n, a);
    }
    float cin = __shfl_down_sync(kFull, a, 1);
    if (lane == 31) cin = 0.f;
    if constexpr (MULTI) {
      if (lane == 0) {
        sh.a[warp] = a;
        sh.edge[0][warp] = T.whole;
      }
      __syncthreads();
      float in = 0.f;  // D right of the warp's last column
      for (int q = nw - 1; q > warp; q--) in = ffma(in, sh.edge[0][q], sh.a[q]);
      cin = ffma(T.dn_in, in, cin);
    }
    float v = cin;
#pragma unroll
    for (int c = C - 1; c >= 0; c--) dc[c] = v = ffma(v, T.dd[c], fadd(al[c], e));
    return cin;
  };
  for (int i = rows; i >= 1; i--) {
    // ---- Forward rows i-1 and i from the current segment ----
    if (seg_lo < 0 || i - 1 < seg_lo) {
      if constexpr (MULTI) __syncthreads();  // the segment's and the exchange's last readers are done
      const int j = (i - 1) / S;
      seg_lo = j * S;
      float fm[C], fi[C], fd[C], left[3];
      T.load_row(ck + j * rowf, tw, fm, fi, fd);
      T.store_row(seg, tw, fm, fi, fd);
      // the column left of the thread's, from the checkpoint
#pragma unroll
      for (int q = 0; q < 3; q++) left[q] = k0 ? ck[j * rowf + q * tw + k0 - 1] : 0.f;
      const float* q = sp + 6 * (int64_t)seg_lo;
      float xn = q[0], xb = q[1], xj = q[3], xc = q[4], xe;
      const int hi = min(seg_lo + S, L);
      int x = __ldg(s + seg_lo), x1 = seg_lo + 1 < L ? __ldg(s + seg_lo + 1) : 24;
      float er[C];
      load_cols<C>(T.im + x * width, er);
      for (int r = seg_lo + 1; r <= hi; r++) {
        const int x2 = r + 1 < L ? __ldg(s + r + 1) : 24;
        T.forward_row(x, x1, er, fm, fi, fd, left, xn, xb, xj, xc, xe, ploop, pmove, sh);
        T.store_row(seg + (int64_t)(r - seg_lo) * rowf, tw, fm, fi, fd);
        x = x1;
        x1 = x2;
      }
      T.load_row(seg + (int64_t)(i - seg_lo) * rowf, tw, fm1, fi1, fd1);
      if constexpr (MULTI) __syncthreads();  // the rows' last exchange is read before a Backward row's first
    }
    float fm0[C], fi0[C], fd0[C];  // Forward row i-1, read while Backward row i is computed
    T.load_row(seg + (int64_t)(i - 1 - seg_lo) * rowf, tw, fm0, fi0, fd0);
    const int xi = __ldg(s + i - 1);  // residue i
    float ei[C];
    load_cols<C>(T.im + xi * width, ei);
    const float* spi = sp + 6 * (int64_t)(i - 1);
    const float fb0 = spi[1];
    const double lsf1 = lsf[i], lsf0 = lsf[i - 1];
    // ---- Backward row i ----
    float mc[C], ic[C], dc[C];
    float inn[C];  // I of row i+1, at its scale when row i is computed
    if (i == L) {
      float al[C];
#pragma unroll
      for (int c = 0; c < C; c++) al[c] = ic[c] = inn[c] = 0.f;
      const float dnr = d_chain(al, bxe, dc);
#pragma unroll
      for (int c = 0; c < C; c++) mc[c] = ffma(c < C - 1 ? dc[c + 1] : dnr, T.md[c], bxe);
    } else {
      const float ins = x != 24 ? 1.f : 0.f;
      float me[C];
      float b = 0.f, top = 0.f;
#pragma unroll
      for (int c = 0; c < C; c++) {
        me[c] = fmul(mn[c], eo[c]);
        b = ffma(me[c], T.bm[c], b);
        if (k0 + c < M) top = fmaxf(top, mn[c]);
      }
      if (MULTI && lane == 0) sh.edge[1][warp] = me[0];
      float bxb = T.sum_max(b, top, sh);
      float me_up = __shfl_down_sync(kFull, me[0], 1);
      if (lane == 31) me_up = MULTI && warp + 1 < nw ? sh.edge[1][warp + 1] : 0.f;
      if (top > 1.0e4f) {  // rescale row i+1
        const float inv = __fdiv_rn(1.0f, top);
#pragma unroll
        for (int c = 0; c < C; c++) {
          me[c] = fmul(me[c], inv);
          inx[c] = fmul(inx[c], inv);
        }
        me_up = fmul(me_up, inv);
        bxb = fmul(bxb, inv);
        bxn = fmul(bxn, inv);
        bxj = fmul(bxj, inv);
        bxc = fmul(bxc, inv);
        lnsb += log((double)top);
      }
      bxj = ffma(bxj, ploop, fmul(bxb, pmove));
      bxc = fmul(bxc, ploop);
      bxe = ffma(bxj, 0.5f, fmul(bxc, 0.5f));
      bxn = ffma(bxn, ploop, fmul(bxb, pmove));
      float al[C];
#pragma unroll
      for (int c = 0; c < C; c++) {
        al[c] = fmul(c < C - 1 ? me[c + 1] : me_up, T.dm[c]);
        inn[c] = fmul(inx[c], ins);
      }
      const float dnr = d_chain(al, bxe, dc);
#pragma unroll
      for (int c = 0; c < C; c++) {
        const float mnext = c < C - 1 ? me[c + 1] : me_up, dnext = c < C - 1 ? dc[c + 1] : dnr;
        mc[c] = ffma(dnext, T.md[c], ffma(mnext, T.mm[c], ffma(inn[c], T.mi[c], bxe)));
        ic[c] = ffma(mnext, T.imr[c], fmul(inn[c], T.ii[c]));
      }
    }
    // ---- accumulate counts (columns past M hold zeros in every Forward row) ----
    const float f_ii = expf((float)(lsf1 + lnsb - lz));  // F(i) . B(i), and F(i) . B(i+1): rows i and i+1 share a scale
    const float f_i0 = expf((float)(lsf0 + lnsb - lz));  // F(i-1) . B(i)
    float l[5] = {__shfl_up_sync(kFull, fm0[C - 1], 1), __shfl_up_sync(kFull, fi0[C - 1], 1),
                  __shfl_up_sync(kFull, fd0[C - 1], 1), __shfl_up_sync(kFull, fm1[C - 1], 1),
                  __shfl_up_sync(kFull, fd1[C - 1], 1)};
    if (MULTI && lane == 0 && warp) {  // the left warp's column, written by it before this segment's last barrier
      const float* r0 = seg + (int64_t)(i - 1 - seg_lo) * rowf + k0 - 1;
      l[0] = r0[0];
      l[1] = r0[tw];
      l[2] = r0[2 * tw];
      l[3] = r0[rowf];
      l[4] = r0[rowf + 2 * tw];
    }
    if (k0 == 0) l[0] = l[1] = l[2] = l[3] = l[4] = 0.f;
    float gm[C], gi[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      gm[c] = fm1[c] * mc[c] * f_ii;
      gi[c] = fi1[c] * ic[c] * f_ii;
      const float bme = ei[c] * mc[c] * f_i0;
      cbm[c] = ffma(fb0 * T.bm[c], bme, cbm[c]);  // B -> M_k
      cmm[c] = ffma((c ? fm0[c - 1] : l[0]) * (c ? T.mm[c - 1] : T.mm0), bme, cmm[c]);
      cim[c] = ffma((c ? fi0[c - 1] : l[1]) * (c ? T.imr[c - 1] : T.im0), bme, cim[c]);
      cdm[c] = ffma((c ? fd0[c - 1] : l[2]) * (c ? T.dm[c - 1] : T.dm0), bme, cdm[c]);
      cmd[c] = ffma((c ? fm1[c - 1] : l[3]) * (c ? T.md[c - 1] : md0) * dc[c], f_ii, cmd[c]);
      cdd[c] = ffma((c ? fd1[c - 1] : l[4]) * (c ? T.dd[c - 1] : dd0) * dc[c], f_ii, cdd[c]);
      cmi[c] = ffma(fm1[c] * T.mi[c] * inn[c], f_ii, cmi[c]);
      cii[c] = ffma(fi1[c] * T.ii[c] * inn[c], f_ii, cii[c]);
    }
    adj_add4(acc + (int64_t)xi * tw, gm);
    adj_add4(acc + (int64_t)(25 + xi) * tw, gi);
    // advance: row i becomes "next"
    x = xi;
#pragma unroll
    for (int c = 0; c < C; c++) {
      eo[c] = ei[c];
      mn[c] = mc[c];
      inx[c] = ic[c];
      fm1[c] = fm0[c];
      fi1[c] = fi0[c];
      fd1[c] = fd0[c];
    }
  }
  // transition counts, rows MM MI MD IM II DM DD BM: those into column k belong
  // to source node k - 1, MI II BM to k
  float* o = out + A.out_off + 50 * (int64_t)W;
#pragma unroll
  for (int c = 0; c < C; c++) {
    const int k = k0 + c + 1;
    if (k > M) break;
    o[0 * W + k - 1] = cmm[c];
    o[1 * W + k] = cmi[c];
    o[2 * W + k - 1] = cmd[c];
    o[3 * W + k - 1] = cim[c];
    o[4 * W + k] = cii[c];
    o[5 * W + k - 1] = cdm[c];
    o[6 * W + k - 1] = cdd[c];
    o[7 * W + k] = cbm[c];
  }
  if (lane == 0 && warp == 0) {
    o[0 * W + M] = o[2 * W + M] = o[3 * W + M] = o[5 * W + M] = o[6 * W + M] = 0.f;
    o[1 * W] = o[4 * W] = o[7 * W] = 0.f;
  }
}

// Emission counts from the scratch rows to the caller's, blockIdx.y = pair.
static __global__ void __launch_bounds__(256) adjoint_out_kernel(const AdjPair* __restrict__ pairs, int M, int tw,
                                                                 const float* __restrict__ accs,
                                                                 float* __restrict__ out) {
  const AdjPair A = pairs[blockIdx.y];
  const int W = M + 1;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < kAdjEmRows * W; q += gridDim.x * blockDim.x) {
    const int r = q / W, k = q - r * W;
    out[A.out_off + q] = k ? accs[A.acc_off + (int64_t)r * tw + k - 1] : 0.f;
  }
}

}  // namespace sxk
