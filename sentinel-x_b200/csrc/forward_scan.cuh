// Forward pre-screen of F3 (src/hmmer/dp.rs:229-298): probability space with the
// reference's sparse rescaling, a team per pair; the pair passes when the
// device estimate of the F3 statistic clears the threshold minus `slack`.
//
// The rows are the adjoint's (AdjTeam::forward_row): one warp up to 256 columns,
// of four columns a thread up to 128 and eight above, a CTA of warps of 256
// columns past that, the D chain an affine scan over lanes and then over warps,
// the row sum a butterfly and a sum over warps.
// The rounding differs from the reference's order, so the pass test adds a
// bound on the difference: for sums and products of non-negative numbers the
// relative errors of two evaluation orders add up along their longest paths,
// at most 2^-24 per operation.  A row's longest path is M operations of the
// chain's factors, 16 of a thread's columns, 10 and 2 a warp of the scans and 9
// and 1 a warp of the sum, below 2M + 6 ceil(M/32) + 64, i.e.
// |ln F_scan - ln F_ref| <= (L+1)(2M + 6 ceil(M/32) + 64) 2^-24, taken twice.
// The pre-screen therefore passes every pair the exact F3 test (on the host,
// from the exact rows of exact_rows.cuh) passes.
//
// What bounds it: the latency of a row.  With a row's columns over one warp's
// lanes whatever M (ceil(M/32) a lane) a row took that many dependent steps
// three times over, and registers spilled from M = 513 on; here they are four or
// eight, and two barriers from 257 columns on.  Eight columns a thread above 128
// spare barriers and repeat the scans less often than four.  Measured on B200,
// the pre-screen's stage of 296 profiles of one length x 12,000 targets, a row
// over one warp / four columns a thread / as here, ms: M = 100 1.09 / 0.86 / 0.86,
// 160 1.59 / 1.79 / 1.00, 250 2.17 / 2.23 / 1.22, 300 3.52 / 2.85 / 3.07, 600
// 7.32 / 5.04 / 4.04, 1000 7.35 / 5.71 / 4.64, 1500 20.9 / 10.6 / 7.3.
#pragma once
#include "adjoint.cuh"

namespace sxk {

template <bool MULTI, int C>
__global__ void __launch_bounds__(MULTI ? 256 : 32) forward_scan_kernel(
    const PairRec* __restrict__ in, const unsigned* __restrict__ in_counts, const BinRegion* __restrict__ in_bins,
    int bin, PairRec* __restrict__ out, const BinRegion* __restrict__ out_bins, unsigned* __restrict__ out_counts,
    unsigned* __restrict__ overflow, const DevProfile* __restrict__ profs, const Thresholds* __restrict__ thr,
    const float* __restrict__ ximg, const uint8_t* __restrict__ res, const int64_t* __restrict__ toff,
    const int32_t* __restrict__ tlen, const float4* __restrict__ xsc, float slack) {
  __shared__ AdjShared sh;
  const unsigned n = min(in_counts[bin], in_bins[bin].cap);
  for (unsigned w = blockIdx.x; w < n; w += gridDim.x) {
    PairRec r = in[in_bins[bin].off + w];
    const DevProfile& P = profs[r.p];
    AdjTeam<MULTI, C> T;
    T.init(ximg + P.x_off, P.m, P.x_width);
    const uint8_t* s = res + toff[r.t];
    const int L = tlen[r.t];
    const float4 xs = xsc[r.t];
    const float ploop = xs.z, pmove = xs.w;
    float m[C], i_[C], d[C], left[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < C; c++) m[c] = i_[c] = d[c] = 0.f;
    float xn = 1.f, xb = pmove, xj = 0.f, xc = 0.f, xe = 0.f;
    double lnscale = 0.0;
    int x = L > 0 ? __ldg(s) : 24, x1 = L > 1 ? __ldg(s + 1) : 24;
    float eo[C];
    load_cols<C>(T.im + x * T.width, eo);
    for (int i = 1; i <= L; i++) {
      const int x2 = i + 1 < L ? __ldg(s + i + 1) : 24;
      const float scale = T.forward_row(x, x1, eo, m, i_, d, left, xn, xb, xj, xc, xe, ploop, pmove, sh);
      x = x1;
      x1 = x2;
      if (scale > 0.f) lnscale += log((double)scale);
    }
    if (threadIdx.x == 0) {
      const int M = P.m;
      const float v = fmul(xc, pmove);
      const float fsc = (L > 0 && M > 0) ? (float)((double)(v > 0.f ? logf(v) : SX_NEG_INF) + lnscale) : SX_NEG_INF;
      r.fwd = fsc;
      const float sl = slack + 2.0f * (float)(L + 1) * (float)(2 * M + 6 * ((M + 31) / 32) + 64) * 5.9604645e-8f / kLn2;
      if (bits_stat(fsc, r.filtersc) >= thr[r.p].s3 - sl) push_pair(r, bin, out, out_bins, out_counts, overflow);
    }
  }
}

}  // namespace sxk
