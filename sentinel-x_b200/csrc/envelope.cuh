// Envelope rescoring on the device: the full-matrix passes of
// rescore_isolated_domain (src/hmmer/pipeline.rs:545-591) for a batch of
// envelopes, one team (a warp up to 256 columns, a CTA above) per envelope.
//
//   env_rows_kernel   forward_matrix (src/hmmer/dp.rs:442-513) and
//                     backward_matrix (dp.rs:516-601), by exact_rows.cuh
//   env_oa_kernel     decode (dp.rs:1278-1306) fused with the column sums of
//                     null2_from_posterior (dp.rs:1310-1350) and the
//                     optimal-accuracy DP and traceback (dp.rs:1355-1564)
//   env_insert_kernel the ordered sum of the insert posteriors
//
// The arithmetic is the reference's, operation for operation (no FMA, ordered
// sums in order), so the matrices, posteriors and coordinates equal the
// host's bit for bit.  Every log/exp stays on the host: env_rows_kernel writes
// raw scaled special rows and rescale factors, the host turns them into the
// per-row posterior factor exp(lnF + lnB - lnZ) and the N/J/C posteriors, and
// the other two read those back.
//
// Measured on B200 (wall time of the passes of one search; before: one warp
// per envelope handing the ordered chains from lane to lane, the insert sum in
// the optimal-accuracy row loop, the traceback over four planes of floats):
// marker-set genome (242 envelopes, M to 1,500) Forward/Backward 43.2 -> 8.3
// ms, posterior/OA 52.8 -> 3.9; Pfam-scale's last block (128) 5.4 -> 1.5 and
// 5.9 -> 1.0; 64 profiles of M 60-700 (61) 10.4 -> 2.4 and 13.0 -> 1.4.
#pragma once
#include <climits>
#include <type_traits>

#include "exact_rows.cuh"

namespace sxk {

// One envelope: residues i0 .. i0+lr-1 (0-based) of target t against profile p,
// with the unihit special transitions of the whole target's length.
struct EnvRec {
  int32_t p, t;
  int32_t i0, lr;
  float ploop, pmove, pe_loop, pe_move;
  int64_t plane_off;  // float offset: 5 planes of (lr+1) rows x width columns (FM FI BM BI OD), then the decisions
  int64_t row_off;    // float offset: forward raw rows 6(lr+1), then backward raw rows 6(lr+1)
  int64_t aux_off;    // float offset: pn pj pc (inputs), then OA specials xe xc; (lr+1) each
  int64_t fac_off;    // double offset: posterior factor per row (lr+1)
  int64_t out_off;    // float offset of kEnvOut outputs
  int32_t width, pad; // columns of a plane row (the profile's exact row shape)
};
// floats of an envelope's planes: 5 planes and half a byte of decision per cell
__host__ __device__ __forceinline__ int64_t env_plane_floats(int64_t lr, int width) {
  return 5 * (lr + 1) * width + (lr + 1) * (width / 8);
}
// Outputs: [0,20) sum_k (sm[k]*norm)*mo[x][k] for x < 20, [20] si (the row-major
// sum of insert posteriors), [21] found (1/0), [22..25] i0 i1 k0 k1 (as floats).
constexpr int kEnvOut = 32;

// Forward (blockIdx.y = 0) and Backward (1) matrices and raw rows of n
// envelopes; DIAG: the Forward matrices of regions in the diagonal layout.
template <int C, bool MULTI, TransIn IN, bool DIAG>
__global__ void __launch_bounds__(team_threads(IN)) env_rows_kernel(const EnvRec* __restrict__ recs, int n,
                                                       const DevProfile* __restrict__ profs,
                                                       const float* __restrict__ ximg,
                                                       const uint8_t* __restrict__ res,
                                                       const int64_t* __restrict__ toff, float* __restrict__ planes,
                                                       float* __restrict__ rows) {
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
  const EnvRec r = recs[w];
  const float* img = ximg + profs[r.p].x_off;
  const int M = profs[r.p].m;
  const uint8_t* s = res + toff[r.t] + r.i0;
  float* pl = planes + r.plane_off;
  float* orow = rows + r.row_off;
  if constexpr (DIAG) {
    exact_forward<C, MULTI, IN, kKeepDiag>(img, M, s, r.lr, r.ploop, r.pmove, r.pe_loop, r.pe_move, orow, pl, T, sh, ss);
  } else if (blockIdx.y == 0) {
    exact_forward<C, MULTI, IN, kKeepMI>(img, M, s, r.lr, r.ploop, r.pmove, r.pe_loop, r.pe_move, orow, pl, T, sh, ss);
  } else {
    exact_backward<C, MULTI, IN, kKeepMI>(img, M, s, r.lr, r.ploop, r.pmove, r.pe_loop, r.pe_move,
                                      orow + 6 * (int64_t)(r.lr + 1), pl + 2 * (int64_t)(r.lr + 1) * r.width, T, sh, ss);
  }
}

__device__ __forceinline__ float oa_gate(float t, float v) { return t > 0.0f ? v : 0.0f; }
__device__ __forceinline__ float oa_dis(float t, float v) { return t == 0.0f ? SX_NEG_INF : v; }

// Traceback decisions of a cell (i, k), four bits: 0-1 the predecessor of M (M,
// I, D at (i-1, k-1), or B), bit 2 set if I comes from I, bit 3 set if the D
// to the RIGHT of the cell, (i, k+1), comes from D.  A row's decisions are
// packed, column k at nibble k - 1.
enum : unsigned { kOaM = 0, kOaI = 1, kOaD = 2, kOaB = 3, kOaIfromI = 4, kOaDfromD = 8 };

enum St { kSM, kSI, kSD };  // traceback states

struct OaShared {  // exchange between the warps of a team
  float val[kXMaxWarps];      // composite D map of the warp: v -> max(val, v), or the constant val
  int cst[kXMaxWarps];
  float prev[3][kXMaxWarps];  // OA M, I, D of the last column
  float mx[kXMaxWarps];
};

// decode + null2 sums + optimal-accuracy DP and traceback.  Reads the forward
// and backward M/I planes, the host's per-row factor exp(lnF + lnB - lnZ) and
// N/J/C posteriors; overwrites the backward M plane with the OA M matrix (each
// row is read before its OA row is written), fills the OD plane, the cells'
// traceback decisions and the OA specials E and C.
//
// A row's latency: the D chain od[k+1] = max(gate(t_md, om[k]), gate(t_dd,
// od[k])) only selects and takes maxima of non-negative values (or -inf),
// exact in any order, so it runs as a scan.  The step out of column k maps the
// chain value v to max(a_k, v) when t_dd > 0 and to the constant max(a_k, 0)
// otherwise; lanes compose their columns' maps, a segmented max scan composes
// them across the warp (a constant starts a segment) and the warps' composites
// go through shared memory.  With the decisions noted while the row is in
// registers the traceback loads half a byte a step, 32 steps of a run of
// matches at a time, instead of following four chains of floats.
template <int C, bool MULTI, TransIn IN>
__global__ void __launch_bounds__(team_threads(IN)) env_oa_kernel(const EnvRec* __restrict__ recs, int n,
                                                     const DevProfile* __restrict__ profs,
                                                     const float* __restrict__ ximg, float* planes, float* aux,
                                                     const double* __restrict__ facs, float* __restrict__ outs) {
  extern __shared__ float4 sm_row[];
  __shared__ OaShared sh;
  const int w = MULTI ? blockIdx.x : blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (w >= n) return;  // uniform over the team
  const int lane = threadIdx.x & 31;
  const int warp = MULTI ? threadIdx.x >> 5 : 0;
  const int nw = MULTI ? blockDim.x >> 5 : 1;
  const int width = nw * 32 * C;
  const int k0 = (MULTI ? threadIdx.x : lane) * C;
  const bool lead = MULTI ? threadIdx.x == 0 : lane == 0;
  float* T = reinterpret_cast<float*>(sm_row) + (MULTI ? 0 : (threadIdx.x >> 5) * 32 * C);
  const EnvRec r = recs[w];
  const float* img = ximg + profs[r.p].x_off;
  const int M = profs[r.p].m;
  const int L = r.lr;
  const int64_t PL = (int64_t)(L + 1) * width;
  const float* FM = planes + r.plane_off;
  const float* FI = FM + PL;
  float* OM = planes + r.plane_off + 2 * PL;  // backward M, then OA M
  const float* BI = OM + PL;
  float* OD = OM + 2 * PL;
  uint8_t* dec = reinterpret_cast<uint8_t*>(OM + 3 * PL);
  const int dec_row = width / 2;  // bytes
  const float* pn = aux + r.aux_off;
  const float* pj = pn + (L + 1);
  const float* pc = pn + 2 * (L + 1);
  float* sxe = aux + r.aux_off + 3 * (L + 1);
  float* sxc = sxe + (L + 1);
  const double* fac = facs + r.fac_off;
  float* out = outs + r.out_off;
  const bool ploop0 = r.ploop == 0.0f, pe_loop0 = r.pe_loop == 0.0f, pe_move0 = r.pe_move == 0.0f,
             pmove0 = r.pmove == 0.0f;
  TeamTrans<C, IN, false> tr;
  tr.init(img, width, k0, T + width);
  float sm[C], omp[C], oip[C], odp[C], fm[C], fi[C], bm[C], bi[C];
#pragma unroll
  for (int c = 0; c < C; c++) {
    sm[c] = 0.f;
    omp[c] = oip[c] = odp[c] = SX_NEG_INF;
    fm[c] = fi[c] = bm[c] = bi[c] = 0.f;
  }
  // plane rows are read a row ahead, as plain loads (the OA M plane is written here)
  auto load_row = [&](int i) {
    const int64_t at = (int64_t)i * width + k0;
#pragma unroll
    for (int q = 0; q < C / 4; q++) {
      const float4 a = reinterpret_cast<const float4*>(FM + at)[q], b = reinterpret_cast<const float4*>(OM + at)[q];
      const float4 c = reinterpret_cast<const float4*>(FI + at)[q], d = reinterpret_cast<const float4*>(BI + at)[q];
      fm[4 * q] = a.x; fm[4 * q + 1] = a.y; fm[4 * q + 2] = a.z; fm[4 * q + 3] = a.w;
      bm[4 * q] = b.x; bm[4 * q + 1] = b.y; bm[4 * q + 2] = b.z; bm[4 * q + 3] = b.w;
      fi[4 * q] = c.x; fi[4 * q + 1] = c.y; fi[4 * q + 2] = c.z; fi[4 * q + 3] = c.w;
      bi[4 * q] = d.x; bi[4 * q + 1] = d.y; bi[4 * q + 2] = d.z; bi[4 * q + 3] = d.w;
    }
  };
  double f = 0.0;
  float pnv = 0.f, pjv = 0.f, pcv = 0.f;
  auto load_specials = [&](int i) {
    f = fac[i];
    pnv = pn[i];
    pjv = pj[i];
    pcv = pc[i];
  };
  if (L >= 1) {
    load_row(1);
    load_specials(1);
  }
  float lm = SX_NEG_INF, li = SX_NEG_INF, ld = SX_NEG_INF;  // the left warp's last column, previous row (lane 0)
  float xb = 0.f, xn = 0.f, xj = SX_NEG_INF, xc = SX_NEG_INF;
  if (lead) {
    sxe[0] = SX_NEG_INF;
    sxc[0] = SX_NEG_INF;
  }
  for (int i = 1; i <= L; i++) {
    float om[C], oi[C], od[C];
    float oml = __shfl_up_sync(kFull, omp[C - 1], 1), oil = __shfl_up_sync(kFull, oip[C - 1], 1);
    float odl = __shfl_up_sync(kFull, odp[C - 1], 1);
    if (lane == 0) {
      oml = lm;
      oil = li;
      odl = ld;
    }
    std::conditional_t<(C > 8), uint64_t, unsigned> bits = 0;  // four a column
    float emax = SX_NEG_INF;
    const auto tbm = tr.row(0), tmm = tr.row(1), tim = tr.row(2), tdm = tr.row(3), tmi = tr.row(4), tii = tr.row(5);
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int k = k0 + c + 1;
      const float pm = k <= M ? (float)__dmul_rn(__dmul_rn((double)fm[c], (double)bm[c]), f) : 0.f;
      const float pi = k < M ? (float)__dmul_rn(__dmul_rn((double)fi[c], (double)bi[c]), f) : 0.f;
      sm[c] = fadd(sm[c], pm);
      om[c] = oi[c] = SX_NEG_INF;
      if (k <= M) {
        const float omv = c ? omp[c - 1] : oml, oiv = c ? oip[c - 1] : oil, odv = c ? odp[c - 1] : odl;
        float sv = oa_gate(tbm[c], xb);
        unsigned best = kOaB;
        if (k >= 2) {
          sv = fmaxf(sv, oa_gate(tmm[c], omv));
          sv = fmaxf(sv, oa_gate(tim[c], oiv));
          sv = fmaxf(sv, oa_gate(tdm[c], odv));
          // the first of M, I, D, B with the largest value
          float top = oa_dis(tmm[c], omv);
          best = kOaM;
          float v = oa_dis(tim[c], oiv);
          if (v > top) { top = v; best = kOaI; }
          v = oa_dis(tdm[c], odv);
          if (v > top) { top = v; best = kOaD; }
          v = oa_dis(tbm[c], xb);
          if (v > top) best = kOaB;
        } else {
          sv = fmaxf(sv, 0.0f);
          // M, I and D have no cell to the left: the first of (-inf, -inf, -inf, B)
          best = oa_dis(tbm[c], xb) > SX_NEG_INF ? kOaB : kOaM;
        }
        om[c] = fadd(sv, pm);
        emax = fmaxf(emax, om[c]);
        oi[c] = fadd(fmaxf(oa_gate(tmi[c], omp[c]), oa_gate(tii[c], oip[c])), pi);
        const bool from_i = !(oa_dis(tmi[c], omp[c]) >= oa_dis(tii[c], oip[c]));
        bits |= (decltype(bits))(best | (from_i ? kOaIfromI : 0u)) << (4 * c);
      }
    }
    if (i < L) load_row(i + 1);
    // the lane's composite map of its columns' D steps
    bool lc = false;
    float lv = SX_NEG_INF, a[C];
    const auto md = tr.row(6), dd = tr.row(7);
#pragma unroll
    for (int c = 0; c < C; c++) {
      a[c] = oa_gate(md[c], om[c]);
      if (dd[c] > 0.0f) {
        lv = fmaxf(lv, a[c]);
      } else {
        lc = true;
        lv = fmaxf(a[c], 0.0f);
      }
    }
    const unsigned cm = __ballot_sync(kFull, lc);
    const unsigned below = (1u << lane) - 1u;
    const unsigned upto = cm & (below | (1u << lane));
    const int head = upto ? 31 - __clz(upto) : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float pv = __shfl_up_sync(kFull, lv, o);
      if (lane - o >= head) lv = fmaxf(lv, pv);
    }
    float in = SX_NEG_INF;  // D of the warp's first column
    if constexpr (MULTI) {
      if (lane == 31) {
        sh.val[warp] = lv;
        sh.cst[warp] = cm != 0;
      }
      __syncthreads();
      for (int q = 0; q < warp; q++) in = sh.cst[q] ? sh.val[q] : fmaxf(in, sh.val[q]);
    }
    float v = __shfl_up_sync(kFull, lv, 1);
    if (lane == 0) v = in;
    else if (!(cm & below)) v = fmaxf(v, in);
#pragma unroll
    for (int c = 0; c < C; c++) {
      const int k = k0 + c + 1;
      od[c] = k <= M ? v : SX_NEG_INF;
      if (k <= M) emax = fmaxf(emax, v);
      if (!(oa_dis(md[c], om[c]) >= oa_dis(dd[c], od[c]))) bits |= (decltype(bits))kOaDfromD << (4 * c);
      v = dd[c] > 0.0f ? fmaxf(a[c], v) : fmaxf(a[c], 0.0f);
    }
    emax = warp_max_f32(emax);
    if constexpr (MULTI) {
      if (lane == 31) {
        sh.mx[warp] = emax;
        sh.prev[0][warp] = om[C - 1];
        sh.prev[1][warp] = oi[C - 1];
        sh.prev[2][warp] = od[C - 1];
      }
      __syncthreads();
      for (int q = 0; q < nw; q++) emax = fmaxf(emax, sh.mx[q]);
      if (lane == 0 && warp) {
        lm = sh.prev[0][warp - 1];
        li = sh.prev[1][warp - 1];
        ld = sh.prev[2][warp - 1];
      }
    }
    float t1 = ploop0 ? 0.0f : fadd(xj, pjv), t2 = pe_loop0 ? 0.0f : emax;
    xj = fmaxf(t1, t2);
    t1 = ploop0 ? 0.0f : fadd(xc, pcv);
    t2 = pe_move0 ? 0.0f : emax;
    xc = fmaxf(t1, t2);
    xn = ploop0 ? 0.0f : fadd(xn, pnv);
    t1 = pmove0 ? 0.0f : xn;
    t2 = pmove0 ? 0.0f : xj;
    xb = fmaxf(t1, t2);
    if (i < L) load_specials(i + 1);
    const int64_t at = (int64_t)i * width + k0;
    store_cols<C>(OM + at, om);
    store_cols<C>(OD + at, od);
    uint8_t* db = dec + (int64_t)i * dec_row + k0 / 2;
    if constexpr (C == 16) *reinterpret_cast<uint64_t*>(db) = bits;
    else if constexpr (C == 8) *reinterpret_cast<uint32_t*>(db) = (uint32_t)bits;
    else *reinterpret_cast<uint16_t*>(db) = (uint16_t)bits;
    if (lead) {
      sxe[i] = emax;
      sxc[i] = xc;
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      omp[c] = om[c];
      oip[c] = oi[c];
      odp[c] = od[c];
    }
  }
  // null2 column sums: v[x] = sum_k (sm[k] * norm) * mo[x][k], k ascending, one
  // residue a lane
  const float norm = __fdiv_rn(1.0f, (float)max(L, 1));
#pragma unroll
  for (int c = 0; c < C; c++) sm[c] = fmul(sm[c], norm);
  store_cols<C>(T + k0, sm);
  team_sync<MULTI>();  // also makes the planes and decisions of every thread visible to the first warp
  if (MULTI && warp) return;
  if (lane < 20) {
    const float4* s4 = reinterpret_cast<const float4*>(T);
    const float4* m4 = reinterpret_cast<const float4*>(img + (kXMo + lane) * width);
    float v = 0.f;
#pragma unroll 4
    for (int q = 0; q < (M + 3) / 4; q++) {
      const float4 a = s4[q], b = __ldg(m4 + q);
      v = fadd(fadd(fadd(fadd(v, fmul(a.x, b.x)), fmul(a.y, b.y)), fmul(a.z, b.z)), fmul(a.w, b.w));
    }
    out[lane] = v;
  }
  __syncwarp();
  // traceback (optimal_accuracy_coords, dp.rs:1420-1564): every lane follows
  // the same path.  C loops down to the last row whose E is not below it.
  int i = L;
  while (i >= 1) {
    const int q = i - lane;
    bool stop = q < 1;
    if (!stop) {
      const float a = ploop0 ? SX_NEG_INF : fadd(sxc[q - 1], pc[q]);
      const float b = pe_move0 ? SX_NEG_INF : sxe[q];
      stop = !(a > b);
    }
    const unsigned m = __ballot_sync(kFull, stop);
    if (m) {
      i -= __ffs(m) - 1;
      break;
    }
    i -= 32;
  }
  int k = 0;
  St s0 = kSM;
  if (i >= 1) {
    // E: among the cells equal to the row's maximum the last M in striped
    // order, or else the first D
    const int Q = max(2, (M - 1) / 4 + 1);
    const float mx = sxe[i];
    int mkey = -1, dkey = INT_MAX;
    for (int kk = lane + 1; kk <= M; kk += 32) {
      const int key = ((kk - 1) % Q) * 4 + (kk - 1) / Q;
      if (OM[(int64_t)i * width + kk - 1] == mx) mkey = max(mkey, key);
      if (OD[(int64_t)i * width + kk - 1] == mx) dkey = min(dkey, key);
    }
    mkey = __reduce_max_sync(kFull, mkey);
    dkey = __reduce_min_sync(kFull, dkey);
    if (mkey >= 0) {
      k = (mkey & 3) * Q + (mkey >> 2) + 1;
    } else if (dkey != INT_MAX) {
      k = (dkey & 3) * Q + (dkey >> 2) + 1;
      s0 = kSD;
    }
  }
  bool found = false;
  int ci0 = 0, ci1 = 0, ck0 = 0, ck1 = 0;
  auto nibble = [&](int ii, int kk) -> unsigned {
    return ii >= 1 && kk >= 1 ? (dec[(int64_t)ii * dec_row + (kk - 1) / 2] >> (4 * ((kk - 1) & 1))) & 15u : 0u;
  };
  while (i >= 1 && k >= 1) {  // every turn moves up or left
    if (s0 == kSM) {
      const unsigned mine = nibble(i - lane, k - lane);
      const bool on = i - lane >= 1 && k - lane >= 1;
      if (!found) {
        found = true;
        ci1 = i;
        ck1 = k;
      }
      // the run of matches: lanes before the first whose predecessor is not M
      const unsigned stop = __ballot_sync(kFull, !on || (mine & 3u) != kOaM);
      const int run = stop ? __ffs(stop) - 1 : 32;
      const bool inside = run < 32 && i - run >= 1 && k - run >= 1;  // lane `run` is a cell (a match) of the path
      const int last = inside ? run : run - 1;  // run >= 1 here if not inside: lane 0 is a cell
      ci0 = i - last;
      ck0 = k - last;
      if (run == 32) {
        i -= 32;
        k -= 32;
        continue;
      }
      if (!inside) break;  // the path left the matrix
      const unsigned p = __shfl_sync(kFull, mine, run) & 3u;
      i -= run + 1;
      k -= run + 1;
      if (p == kOaB) break;
      s0 = p == kOaI ? kSI : kSD;
    } else if (s0 == kSI) {
      const unsigned d = nibble(i, k);
      i -= 1;
      if (!(d & kOaIfromI)) s0 = kSM;
    } else {
      const unsigned d = nibble(i, k - 1);  // 0 for k = 1: no D there, the path ends at the left edge
      k -= 1;
      if (!(d & kOaDfromD)) s0 = kSM;
    }
  }
  if (lane == 0) {
    out[21] = found ? 1.f : 0.f;
    out[22] = (float)ci0;
    out[23] = (float)ci1;
    out[24] = (float)ck0;
    out[25] = (float)ck1;
  }
}

// si: every insert posterior of the envelope added in row-major order (the
// null2 length correction, dp.rs:1310-1350).  The sum is one chain of L * M
// adds, but a term below half an ulp of the running sum leaves it unchanged,
// and the sum never falls: up to kInsertRows warps compute one row each against the
// sum as it stood a batch earlier and keep, in order, the groups of four
// columns with a term that can still count; one warp adds those while the
// others prepare the next rows.
constexpr int kInsertRows = 8;  // at most: blockDim.x / 32 - 1 rows a batch
static __global__ void __launch_bounds__(32 * (kInsertRows + 1)) env_insert_kernel(
    const EnvRec* __restrict__ recs, int n, const DevProfile* __restrict__ profs, const float* __restrict__ planes,
    const double* __restrict__ facs, float* __restrict__ outs, int max_width) {
  extern __shared__ float4 sm_row[];  // 2 batches x `rows` lists of max_width / 4 groups
  __shared__ int s_n[2][kInsertRows];
  __shared__ float s_si;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rows = (blockDim.x >> 5) - 1;
  const EnvRec r = recs[blockIdx.x];
  const int M = profs[r.p].m, L = r.lr, width = r.width;
  const int64_t PL = (int64_t)(L + 1) * width;
  const float* FI = planes + r.plane_off + PL;
  const float* BI = planes + r.plane_off + 3 * PL;
  const double* fac = facs + r.fac_off;
  const int cap = max_width / 4;
  if (threadIdx.x == 0) s_si = 0.f;
  __syncthreads();
  const int batches = (L + rows - 1) / rows;
  float si = 0.f;
  for (int b = 0; b <= batches; b++) {  // batch b is prepared while batch b - 1 is added
    if (warp == 0) {
      if (b) {
        for (int q = 0; q < rows; q++) {
          const float4* t = sm_row + (((b - 1) & 1) * rows + q) * cap;
          const int m = s_n[(b - 1) & 1][q];
          float4 x = m ? t[0] : make_float4(0.f, 0.f, 0.f, 0.f);
          for (int e = 0; e < m; e++) {
            const float4 nx = e + 1 < m ? t[e + 1] : x;
            si = fadd(fadd(fadd(fadd(si, x.x), x.y), x.z), x.w);
            x = nx;
          }
        }
      }
    } else {
      const int q = warp - 1, i = b * rows + q + 1;
      int m = 0;
      if (i <= L) {
        // half an ulp of the sum: 2^(exponent - 24), 0 for a sum below 2^-102
        const int e = (__float_as_int(s_si) >> 23) - 24;
        const float half = e > 0 ? __int_as_float(e << 23) : 0.f;
        const double f = fac[i];
        float4* list = sm_row + ((b & 1) * rows + q) * cap;
        const float4* fi = reinterpret_cast<const float4*>(FI + (int64_t)i * width) + lane;
        const float4* bi = reinterpret_cast<const float4*>(BI + (int64_t)i * width) + lane;
        for (int base = 0; base < M; base += 512) {  // four loads of each plane in flight
          float4 x[4], y[4];
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (base + 128 * u < M) {  // width is a multiple of 128
              x[u] = __ldg(fi + base / 4 + 32 * u);
              y[u] = __ldg(bi + base / 4 + 32 * u);
            }
#pragma unroll
          for (int u = 0; u < 4; u++) {
            if (base + 128 * u >= M) break;
            const int k = base + 128 * u + 4 * lane;  // columns k+1 .. k+4
            auto post = [&](float a, float c, int kk) {
              return kk < M ? (float)__dmul_rn(__dmul_rn((double)a, (double)c), f) : 0.f;
            };
            const float4 p = make_float4(post(x[u].x, y[u].x, k + 1), post(x[u].y, y[u].y, k + 2),
                                         post(x[u].z, y[u].z, k + 3), post(x[u].w, y[u].w, k + 4));
            // counts unless zero or below half an ulp (NaN counts)
            auto counts = [&](float t) { return t != 0.f && !(t < half); };
            const bool any = counts(p.x) || counts(p.y) || counts(p.z) || counts(p.w);
            const unsigned mask = __ballot_sync(kFull, any);
            if (any) list[m + __popc(mask & ((1u << lane) - 1u))] = p;
            m += __popc(mask);
          }
        }
      }
      if (lane == 0) s_n[b & 1][q] = m;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_si = si;
    __syncthreads();
  }
  if (threadIdx.x == 0) outs[r.out_off + 20] = si;
}


// ---- stochastic traceback ensembles of multi-domain regions ------------------
// region_trace_ensemble (src/hmmer/pipeline.rs:360-477) up to the clustering:
// kTraceSamples sampled traces (stochastic_trace, src/hmmer/dp.rs:1075-1258)
// through the region's multihit Forward matrix (env_rows_kernel<..., DIAG>,
// diagonal layout), one Easel LCG stream per region, the per-trace null2 of
// every sampled domain and its per-position sums.  The host clusters the
// samples and takes the logs.

constexpr int kTraceSamples = 200;
constexpr int kTraceDoms = 32;   // sampled domains of one trace held in shared memory
constexpr int kTraceRecord = 6;  // region, trace, sqfrom, sqto, hmmfrom, hmmto (target coordinates)
constexpr int kTraceRes = 20;    // canonical residues; codes 20..23 degenerate, 24 '*'
// Per profile column k (1-based), kTraceCol floats at (k-1)*kTraceCol:
// p_bm[k] p_mm[k-1] p_im[k-1] p_dm[k-1] p_mi[k] p_ii[k] p_md[k-1] p_dd[k-1],
// then the match odds mo[x][k] of the 20 canonical residues.
constexpr int kTraceCol = 28;

struct TraceRec {
  int32_t m, t;        // profile length, target
  int32_t i0, lr;      // region residues i0 .. i0+lr-1 (0-based)
  float ploop, pmove;  // multihit special transitions of the target's length
  float pe_loop, pe_move;
  int64_t plane_off;   // diagonal M I D planes of env_rows_kernel<..., DIAG>
  int64_t row_off;     // its raw special rows, 6 (lr+1)
  int64_t n2_off;      // per-position null2 sums, lr+1 floats (slot 0 unused)
  int64_t col_off;     // the profile's column table (kTraceCol floats per column)
};

struct TraceConsts {
  uint32_t lcg0;        // LCG state after seeding (esl_mix3 of seed 42)
  int32_t deg_n[4];     // member counts of the degenerate codes B J Z X
  int8_t deg_m[4][20];  // their members (esl_abc_FAvgScVec order)
};

__device__ __forceinline__ double trace_uniform(uint32_t& rng) {
  rng = rng * 69069u + 1u;
  return (double)rng * 2.3283064365386962890625e-10;  // / 2^32, exact
}

// esl_vec_FNorm (Kahan) then esl_rnd_FChoose (src/hmmer/dp.rs:1026-1059); the
// quotients acc/norm are independent, so all are formed before the first test.
// The last candidate needs none: with no earlier hit the choice is N-1 whether
// or not its test passes.
template <int N>
__device__ __forceinline__ int trace_choose(uint32_t& rng, float (&v)[N]) {
  float s = 0.f, comp = 0.f;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const float y = __fsub_rn(v[i], comp);
    const float t = __fadd_rn(s, y);
    comp = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
#pragma unroll
  for (int i = 0; i < N; i++) v[i] = s != 0.f ? __fdiv_rn(v[i], s) : 1.f / (float)N;
  double norm = 0.0, acc[N];
#pragma unroll
  for (int i = 0; i < N; i++) norm = __dadd_rn(norm, (double)v[i]);
  double a = 0.0;
#pragma unroll
  for (int i = 0; i < N; i++) acc[i] = a = __dadd_rn(a, (double)v[i]);
  const double roll = trace_uniform(rng);
  int pick = N - 1;
#pragma unroll
  for (int i = N - 2; i >= 0; i--)
    if (roll < __ddiv_rn(acc[i], norm)) pick = i;
  return pick;
}

// One warp per region; every lane follows the same trace (same loads, same LCG
// draws), lanes 0..19 carry the null2 sums of the residues, the warp scans the
// E-state entry candidates 32 at a time (each lane forms the running sum up to
// its candidate, in order) and all lanes update the per-position sums.  A
// region that leaves the matrix, or whose samples overflow the pool or the
// per-trace buffer, is flagged (status 1) for the host to redo.  Pool records
// carry the region's index `first + w` within the caller's batch.
static __global__ void __launch_bounds__(128) env_trace_kernel(const TraceRec* __restrict__ recs, int n,
                                                        const float* __restrict__ cols,
                                                        const uint8_t* __restrict__ res,
                                                        const int64_t* __restrict__ toff,
                                                        const float* __restrict__ planes,
                                                        const float* __restrict__ rows, float* __restrict__ n2sum,
                                                        int32_t* __restrict__ pool, int32_t* __restrict__ pool_count,
                                                        int32_t pool_cap, int32_t first, int32_t* __restrict__ status,
                                                        TraceConsts tc) {
  __shared__ float sn2[4][32];
  __shared__ int4 sdom[4][kTraceDoms];
  const int lane = threadIdx.x & 31;
  const int wib = (threadIdx.x >> 5) & 3;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  enum { SC, SE, SM, SI, SD, SB, SJ, SN };
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += warps) {
    const TraceRec r = recs[w];
    const int M = r.m;
    const int L = r.lr;
    const int64_t PL = diag_plane(L, M);
    const float* FM = planes + r.plane_off;
    const float* FI = FM + PL;
    const float* FD = FI + PL;
    const float* xr = rows + r.row_off;
    const float* col = cols + r.col_off;
    const uint8_t* s = res + toff[r.t] + r.i0;
    float* ns = n2sum + r.n2_off;
    bool bad = L < 1 || M < 1;
    for (int pos = lane; pos <= L; pos += 32) ns[pos] = 0.f;
    __syncwarp();
    // planes at (row, k), 1 <= k <= M; row 0 of the matrix is all zero
    auto plane = [&](const float* X, int row, int k) { return row ? __ldg(X + diag_at(row, k, M)) : 0.f; };
    auto prob = [&](int q, int k) { return __ldg(col + (k - 1) * kTraceCol + q); };
    const float pmove = r.pmove, ploop = r.ploop;
    // special row i, slots N B E J C and the rescale factor (1 when the row was
    // not rescaled); row 0 is the start state N = 1, B = pmove
    auto spec = [&](int slot, int i) -> float {
      if (i == 0) return slot == 0 || slot == 5 ? 1.f : slot == 1 ? pmove : 0.f;
      const float v = __ldg(xr + 6 * (int64_t)i + slot);
      return slot == 5 && !(v > 0.f) ? 1.f : v;
    };
    const int q_stripes = max(2, (M - 1) / 4 + 1);
    const int ncand = 8 * q_stripes;
    // entry candidate c of the E-state scan (the reference's striped order):
    // stripe c/8, M (c%8 < 4) or D, node (c%4)*q_stripes + c/8 + 1
    auto cand_k = [&](int c) { return (c & 3) * q_stripes + (c >> 3) + 1; };
    const int64_t limit = 8 * (int64_t)(L + 2) * (int64_t)(M + 2) + 64;
    uint32_t rng = tc.lcg0;
    for (int tr = 0; tr < kTraceSamples && !bad; tr++) {
      int s0 = SC;
      int i = L, k = 0;
      bool have = false;
      int sqfrom = 0, sqto = 0, hmmfrom = 0, hmmto = 0, nn = 0;
      float vs = 0.f;  // lane x < 20: sum of mo[x][node] over the domain's nodes
      int hi = L + 1;  // positions >= hi have their sum for this trace
      int nd = 0;      // domains of this trace so far (in discovery order: last first)
      for (int64_t guard = 1; guard <= limit; guard++) {
        int s1;
        if (s0 == SC) {
          if (i == 0) break;
          float path[2] = {fmul(spec(4, i - 1), ploop), fmul(fmul(spec(2, i), r.pe_move), spec(5, i))};
          s1 = trace_choose(rng, path) == 0 ? SC : SE;
        } else if (s0 == SE) {
          const double roll = trace_uniform(rng);
          const float norm = (float)__ddiv_rn(1.0, (double)spec(2, i));
          double acc = 0.0;
          int pick = 0, pst = SM;
          for (int pass = 0; pick == 0 && pass < 1000; pass++) {
            auto load = [&](int c) {
              const int kk = cand_k(c);
              return c < ncand && kk <= M ? (double)fmul(plane((c & 4) ? FD : FM, i, kk), norm) : 0.0;
            };
            double val = load(lane);
            for (int c0 = 0; c0 < ncand; c0 += 32) {
              const double nxt = c0 + 32 < ncand ? load(c0 + 32 + lane) : 0.0;
              // lane j: the running sum through candidate c0 + j, in order;
              // a skipped candidate adds +0, which leaves the sum unchanged
              double run = acc;
              for (int j = 0; j < 32; j++) {
                const double v = __shfl_sync(kFull, val, j);
                if (j <= lane) run = __dadd_rn(run, v);
              }
              const unsigned hit = __ballot_sync(kFull, roll < run);
              if (hit) {
                const int j = __ffs(hit) - 1;
                pick = cand_k(c0 + j);
                pst = ((c0 + j) & 4) ? SD : SM;
                break;
              }
              acc = __shfl_sync(kFull, run, 31);
              val = nxt;
            }
            if (pick == 0 && acc <= 0.0) break;
          }
          if (pick == 0) break;
          k = pick;
          have = true;
          sqfrom = sqto = hmmfrom = hmmto = nn = 0;
          vs = 0.f;
          s1 = pst;
        } else if (s0 == SM) {
          if (i < 1 || k < 1 || k > M) { bad = true; break; }
          if (have) {
            if (sqto == 0) { sqto = i; hmmto = k; }
            sqfrom = i;
            hmmfrom = k;
            nn++;
            if (lane < kTraceRes) vs = __fadd_rn(vs, prob(8 + lane, k));
          }
          float path[4] = {fmul(spec(1, i - 1), prob(0, k)), 0.f, 0.f, 0.f};
          if (k >= 2) {
            path[1] = fmul(plane(FM, i - 1, k - 1), prob(1, k));
            path[2] = fmul(plane(FI, i - 1, k - 1), prob(2, k));
            path[3] = fmul(plane(FD, i - 1, k - 1), prob(3, k));
          }
          const int c = trace_choose(rng, path);
          k -= 1;
          i -= 1;
          s1 = c == 0 ? SB : c == 1 ? SM : c == 2 ? SI : SD;
        } else if (s0 == SD) {
          float path[2] = {0.f, 0.f};
          if (k >= 2) {
            if (k > M) { bad = true; break; }
            path[0] = fmul(plane(FM, i, k - 1), prob(6, k));
            path[1] = fmul(plane(FD, i, k - 1), prob(7, k));
          }
          const int c = trace_choose(rng, path);
          k -= 1;
          s1 = c == 0 ? SM : SD;
        } else if (s0 == SI) {
          if (i < 1 || k < 1 || k > M) { bad = true; break; }
          if (have) {
            nn++;
            if (lane < kTraceRes) vs = __fadd_rn(vs, prob(8 + lane, k));
          }
          float path[2] = {fmul(plane(FM, i - 1, k), prob(4, k)), fmul(plane(FI, i - 1, k), prob(5, k))};
          const int c = trace_choose(rng, path);
          i -= 1;
          s1 = c == 0 ? SM : SI;
        } else if (s0 == SB) {
          if (have) {  // a sampled domain is complete: its null2 and its positions' sums
            if (nd >= kTraceDoms) { bad = true; break; }
            const float ld = (float)max(nn, 1);
            if (lane < kTraceRes) sn2[wib][lane] = __fdiv_rn(vs, ld);
            __syncwarp();
            if (lane >= kTraceRes && lane < kTraceRes + 4) {
              const int d = lane - kTraceRes;
              float a = 0.f;
              for (int q = 0; q < tc.deg_n[d]; q++) a = __fadd_rn(a, sn2[wib][tc.deg_m[d][q]]);
              sn2[wib][lane] = __fdiv_rn(a, (float)tc.deg_n[d]);
            } else if (lane == kTraceRes + 4) {
              sn2[wib][lane] = 1.f;
            }
            __syncwarp();
            for (int pos = sqto + 1 + lane; pos < hi; pos += 32) ns[pos] = __fadd_rn(ns[pos], 1.f);
            for (int pos = sqfrom + 1 + lane; pos <= sqto; pos += 32)
              ns[pos] = __fadd_rn(ns[pos], sn2[wib][__ldg(s + pos - 1)]);
            __syncwarp();
            hi = sqfrom + 1;
            if (lane == 0) sdom[wib][nd] = make_int4(sqfrom, sqto, hmmfrom, hmmto);
            nd++;
            have = false;
          }
          float path[2] = {fmul(spec(0, i), pmove), fmul(spec(3, i), pmove)};
          s1 = trace_choose(rng, path) == 0 ? SN : SJ;
        } else if (s0 == SJ) {
          if (i == 0) break;
          float path[2] = {fmul(spec(3, i - 1), ploop), fmul(fmul(spec(2, i), r.pe_loop), spec(5, i))};
          s1 = trace_choose(rng, path) == 0 ? SJ : SE;
        } else {
          if (i == 0) break;
          s1 = SN;
        }
        if ((s1 == SN || s1 == SJ || s1 == SC) && s1 == s0) i -= 1;
        s0 = s1;
      }
      if (bad) break;
      for (int pos = 1 + lane; pos < hi; pos += 32) ns[pos] = __fadd_rn(ns[pos], 1.f);
      __syncwarp();
      // this trace's domains in sequence order, as one block of the pool
      int base = 0;
      if (lane == 0 && nd > 0) base = atomicAdd(pool_count, nd);
      base = __shfl_sync(kFull, base, 0);
      if (nd > 0 && (int64_t)base + nd > (int64_t)pool_cap) {  // mark the reserved slots that exist as unused
        for (int q = lane; q < nd && base + q < pool_cap; q += 32) pool[(int64_t)(base + q) * kTraceRecord] = -1;
        bad = true;
        break;
      }
      for (int q = lane; q < nd; q += 32) {
        const int4 d = sdom[wib][nd - 1 - q];
        int32_t* o = pool + (int64_t)(base + q) * kTraceRecord;
        o[0] = first + w;
        o[1] = tr;
        o[2] = d.x + r.i0;
        o[3] = d.y + r.i0;
        o[4] = d.z;
        o[5] = d.w;
      }
      __syncwarp();
    }
    if (lane == 0) status[w] = bad ? 1 : 0;
  }
}

}  // namespace sxk
