// Packed-integer MSV pre-screen: an upper bound of the reference's f32 MSV
// score (src/hmmer/dp.rs:92-145) for two profiles at once, in int16x2 lanes.
//
// Why: the exact f32 MSV kernel is bound by its ALU pipe and by the 4 bytes of
// shared memory each DP cell reads.  Here every 32-bit word carries the same
// column of two profiles (profile a in the low half, b in the high half), so
// one LDS.128 feeds 8 cells, a fused max(a + b, c) and half a three-input
// maximum do 2 cells, and the pair shares the target's residues and the diagonal
// shuffle.
//
// Exactness.  The pre-screen never decides a pair; it only rejects pairs whose
// bound fails F1, and every pair it passes is rescored by the exact kernel.
// The bound holds by construction:
//   * cells are integers in units of q = 2^-9 nat.  Every match score is
//     rounded up (e_u = ceil((e + rho)/q), rho = 2^-12 nat, which exceeds the
//     f32 rounding of one addition for |value| < 4096 nats) and clamped up to
//     -16 nats; the entry score is rounded up the same way and clamped up to
//     -32 nats.  Integer max-plus over rounded-up scores is >= the real-valued
//     recurrence, which is >= the f32 recurrence minus its rounding, so by
//     induction every integer cell is >= the f32 cell (max is exact and
//     monotone; raising an input only raises the result);
//   * the row maximum is an int16 max, exact; it enters the special states,
//     kept as int32 in units of 2^-20 nat with every constant (tloop, tmove,
//     tbm, -ln 2) rounded up after adding 2^-17 nat, the f32 rounding bound of
//     one addition for |value| <= 128 nats; the specials are therefore upper
//     bounds of the reference's f32 specials row by row;
//   * the final bound (xC + tmove, rounded up to f32) goes through the same
//     f32 bit statistic as the exact kernel, which is monotone.
// int16 headroom: cells stay in [-32768, cap + emax] (the entry's floor and a
// padding column's score add up to -32768); a row maximum above the
// profile's cap (32767 minus its largest rounded score) marks the pair as
// passing before any cell can wrap, and the flag is sticky.
#pragma once
#include <cstdint>

#include "kernels.cuh"

namespace sxk {

constexpr int kQ16Shift = 9;        // cells: units of 2^-9 nat
constexpr int kQ32Shift = 20;       // specials: units of 2^-20 nat
constexpr int kQ32Rho = 8;          // 2^-17 nat in units of 2^-20
constexpr int kQ16EFloor = -8192;   // -16 nats: lowest match score of a real column
constexpr int kQ16EPad = -16384;    // columns past M
constexpr int kQ16BeFloor = -16384; // -32 nats: lowest entry score
constexpr int kQ32Neg = -(1 << 30); // f32 -inf of the special states
constexpr unsigned kQ16Neg2 = 0x80008000u;  // (-32768, -32768)
static_assert(kQ16BeFloor + kQ16EPad >= -32768 && kQ16BeFloor + kQ16EFloor >= -32768, "MSV sums leave int16");

// A pair of profiles of one MSV shape x a slice [begin, end) of the target list
// (pb = -1: the high half is padding and produces no decisions).
struct PackedTile {
  int32_t pa, pb, begin, end;
};

__device__ __forceinline__ unsigned max2s16(unsigned a, unsigned b) {
  unsigned d;
  asm("max.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ unsigned add2s16(unsigned a, unsigned b) {
  unsigned d;
  asm("add.s16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
// f32 constant in units of 2^-20 nat, plus rho, rounded up (exact: x * 2^20 is
// exact in f32 and the integers involved stay below 2^24 in magnitude).
__device__ __forceinline__ int q32_up(float x) {
  return (int)ceilf(__fmul_rn(x, 1048576.0f)) + kQ32Rho;
}

// The recurrence cell = max(diagonal, B) + e and the row maximum cost three
// packed ALU operations a column as they stand, and the ALU pipe (64 packed
// operations per clock per SM, fused or not: add, max, max(a + b, c) and
// max(a, b, c) all issue at that rate on B200) is the kernel's bound.  So a
// lane holds w = max(cell, B) instead, the next row's input:
//     w'[k] = max(w[k-1] + e[k], B')            one fused operation,
//     E = max over w'                           half a three-input maximum,
// 1.5 operations a column, with B' the B of the row being computed.  That
// depends on the row's own E only when E raises base = max(N, J), which is rare
// (a pair's few best rows): B' is predicted from base decayed by tloop, the
// lanes vote on whether any E lies above the threshold at which it raises base,
// and only then the group takes its maximum, updates base and raises w to the
// row's B (w' = max(cell, B') and B >= B', so max(w', B) = max(cell, B)).
// The two profiles' base and constants are int32 in units of 2^-25 nat here,
// so the int16 value of a state is the upper half of its word.  J itself
// matters only at the target's end: above N it is base; below N the pair's
// bound is below N's, which fails F1 (where it might not, or where the bound
// itself is asked for, the tile also tracks J).
//   * E taken over w' is max(E, B').  That cannot raise base, as B' plus the
//     E->J cost is below it.
//   * rows past the target's end in its last block of four read '*' (-16 nats
//     everywhere): they raise nothing and their decay is undone.
//   * a target long enough to reach the entry floor or to have tloop rounded
//     up to 0 (L > 390,000) is recomputed by the plain recurrence.
//   * a tile that tracks J keeps it per lane, of the lane's own columns, and
//     the group combines them once, which is exact, as max and the common decay
//     commute; a final J at or below the final B's level may come from B' and is
//     recomputed by the plain recurrence too (no row of the target scored above
//     its entry: all '*', say).
// Bound now: the ALU pipe, about 70 operations per row of 40 columns, and 2
// bytes of shared memory per cell (64 cells per clock per SM).  The next row's
// first scores are loaded before the vote, whose branch would otherwise keep
// them behind it.  Measured on B200 (296 profiles of one length x 12,000
// targets, useful cells per clock per SM, before -> now): M = 100 40.0 -> 46.1,
// 160 42.9 -> 50.7, 208 44.4 -> 54.2, 300 40.1 -> 49.6, 600 39.6 -> 50.7, 1000
// 45.3 -> 53.9; the Pfam-scale search's pre-screen 298 -> 255 ms, and 211 with
// tiles of equal work.
//
// Plain recurrence of one target for the group (see above); w is scratch.
// Returns J of both halves at row L (units of 2^-20 nat) and the caps' flags.
template <int G, int C, int ROWP>
__device__ __noinline__ int4 msv16_plain(const uint4* __restrict__ rows, const uint8_t* __restrict__ seq, int L, int j,
                                         unsigned gmask, int tloop, int tmove, int tbm_a, int tbm_b, int cap_a,
                                         int cap_b, int nln2) {
  unsigned w[C];
#pragma unroll
  for (int c = 0; c < C; c++) w[c] = kQ16Neg2;
  int xn = 0, xja = kQ32Neg, xjb = kQ32Neg;
  bool biga = false, bigb = false;
  auto entry = [&](int xb, int tbm) { return max((xb + tbm + 2047) >> (kQ32Shift - kQ16Shift), kQ16BeFloor); };
  unsigned bew = __byte_perm((unsigned)entry(tmove, tbm_a), (unsigned)entry(tmove, tbm_b), 0x5410);
  for (int i = 0; i < L; i++) {
    const uint4* rowp = rows + (int)seq[i] * ROWP + j;
    unsigned left = __shfl_up_sync(gmask, w[C - 1], 1, G);
    if (j == 0) left = kQ16Neg2;
    unsigned xe = kQ16Neg2;
#pragma unroll
    for (int c = C - 1; c >= 0; c--) {
      const uint4 a4 = rowp[(c >> 2) * G];
      const unsigned ra = (c & 3) == 0 ? a4.x : (c & 3) == 1 ? a4.y : (c & 3) == 2 ? a4.z : a4.w;
      w[c] = add2s16(max2s16(c ? w[c - 1] : left, bew), ra);
      xe = max2s16(xe, w[c]);
    }
#pragma unroll
    for (int o = G / 2; o >= 1; o >>= 1) xe = max2s16(xe, __shfl_xor_sync(gmask, xe, o, G));
    const int ea = (int)(short)(xe & 0xffffu), eb = (int)xe >> 16;
    biga |= ea > cap_a;
    bigb |= eb > cap_b;
    xja = max(xja + tloop, ea * 2048 + nln2);
    xjb = max(xjb + tloop, eb * 2048 + nln2);
    xn += tloop;
    bew = __byte_perm((unsigned)entry(max(xn, xja) + tmove, tbm_a), (unsigned)entry(max(xn, xjb) + tmove, tbm_b), 0x5410);
  }
  return make_int4(xja, xjb, biga, bigb);
}

// Bound of a profile pair against a slice of targets.  Each profile has its
// own quantized image (25 rows of int16, the lane-major chunk layout of its
// f32 MSV image, 4 columns per uint2); the CTA interleaves the two into words
// while staging them in shared memory.  Per target and half: with `rlist`,
// a pair whose bound passes F1 (or hit the cap) is appended to its profile's
// rescoring list (region (p - p0) * rcap); with `bound_out`, the bound
// (f32 nats, +inf when capped) is written at slot[entry] (profile a) and
// bound_stride + slot[entry] (profile b).
template <int G, int C>
__global__ void __launch_bounds__(256, 2) msv16_kernel(
    const PackedTile* __restrict__ tiles, const DevProfile* __restrict__ profs, const Thresholds* __restrict__ thr,
    const uint2* __restrict__ qimg, const uint8_t* __restrict__ res, const int64_t* __restrict__ toff,
    const int32_t* __restrict__ tlen, const float4* __restrict__ tpar, const int32_t* __restrict__ list,
    int32_t* __restrict__ rlist, unsigned rcap, unsigned* __restrict__ rcount, int p0, unsigned* __restrict__ overflow,
    float* __restrict__ bound_out, const int32_t* __restrict__ slot, int64_t bound_stride) {
  static_assert(C % 4 == 0 && (G & (G - 1)) == 0 && G <= 32, "bad MSV shape");
  constexpr int NC4 = C / 4;
  constexpr int ROW4 = NC4 * G;
  constexpr int NCOPY = G < 8 ? 8 / G : 1;   // bank-conflict-free copies, as in msv_kernel
  constexpr int ROWP = (ROW4 + 7) & ~7;
  constexpr int COPY4 = 25 * ROWP + 8;
  extern __shared__ uint4 sm_img[];
  __shared__ int s_next;
  const PackedTile tile = tiles[blockIdx.x];
  const DevProfile& PA = profs[tile.pa];
  const bool has_b = tile.pb >= 0;
  const DevProfile& PB = profs[has_b ? tile.pb : tile.pa];
  {
    const uint2* sa = qimg + PA.q_off;
    const uint2* sb = qimg + PB.q_off;
    for (int q = threadIdx.x; q < 25 * ROW4; q += blockDim.x) {
      const int x = q / ROW4, e = q - x * ROW4;
      const uint2 va = sa[q];
      const uint2 vb = has_b ? sb[q] : make_uint2(0xc000c000u, 0xc000c000u);
      const uint4 v = make_uint4(__byte_perm(va.x, vb.x, 0x5410), __byte_perm(va.x, vb.x, 0x7632),
                                 __byte_perm(va.y, vb.y, 0x5410), __byte_perm(va.y, vb.y, 0x7632));
#pragma unroll
      for (int cp = 0; cp < NCOPY; cp++) sm_img[cp * COPY4 + cp * G + x * ROWP + e] = v;
    }
  }
  if (threadIdx.x == 0) s_next = tile.begin;
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const int j = lane & (G - 1);
  const uint4* my_rows = sm_img + (lane / G % NCOPY) * (COPY4 + G);
  const int gl = lane - j;
  const unsigned gmask = (G == 32) ? kFull : (((1u << G) - 1u) << gl);
  const int cap_a = PA.q_cap, cap_b = has_b ? PB.q_cap : 32767;
  const int tbm_a = PA.q_tbm, tbm_b = PB.q_tbm;
  const int nln2 = (int)ceilf(-0.693147182464599609375f * 1048576.0f) + kQ32Rho;
  const int nln2_25 = 32 * nln2;
  constexpr int kJStart = -60 * (1 << 25);             // below every J a row can set
  const int base_idle = 32767 * 65536 + nln2_25;       // a base no E raises
  const float s1a = thr[tile.pa].s1, s1b = has_b ? thr[tile.pb].s1 : __int_as_float(0x7f800000);
  // J below N matters where the bound is asked for and where a bound at N's
  // level might pass: that is -1.3 to -0.4 bits, and above 0.5 only from about
  // 150,000 residues on, when tloop's rounding has eaten its decay (such a pair
  // may then pass at N's level, which costs a rescoring and loses nothing)
  const bool track = bound_out != nullptr || !(s1a >= 0.5f) || !(s1b >= 0.5f);

  unsigned w[C];
#pragma unroll
  for (int c = 0; c < C; c++) w[c] = kQ16Neg2;
  // of the current target, both halves, in 2^-25 nat: base at the block's start,
  // the entry constant tmove + tbm + 2047 / 2^20, and J of this lane's columns
  int base_a = base_idle, base_b = base_idle, ka = 0, kb = 0, ja = kJStart, jb = kJStart;
  int tloop = 0;
  unsigned bcur = kQ16Neg2;  // B of the last row computed
  bool biga = false, bigb = false;
  int entry = -1, L = 0, row = 0, boff = 0;
  const uint8_t* seq = res;
  uint4 rcur = make_uint4(0x18181818u, 0x18181818u, 0x18181818u, 0x18181818u), rnext = rcur;
  bool active = false, done = false;
  auto upper = [](int a, int b) { return __byte_perm((unsigned)a, (unsigned)b, 0x7632); };  // int16 of two states

  for (;;) {
    if (!done && row >= L) {  // group-uniform: finish the current target, fetch the next
      if (active) {
        const int tgt = list[entry];
        const float4 tp = tpar[tgt];
        const int tmove = q32_up(tp.y);
        auto bound = [&](int xj) { return __fmul_rn(__int2float_ru(xj + tmove), 9.5367431640625e-7f); };
        const int undo = (row - L) * tloop;
        int xja = (base_a - undo) >> 5, xjb = (base_b - undo) >> 5;  // J where it is above N
        bool plain = tloop >= 0 || row * tloop + min(ka, kb) < (kQ16BeFloor + 1) * 65536;
        if (track) {
#pragma unroll
          for (int o = G / 2; o >= 1; o >>= 1) {
            ja = max(ja, __shfl_xor_sync(gmask, ja, o, G));
            jb = max(jb, __shfl_xor_sync(gmask, jb, o, G));
          }
          xja = ((ja - undo) >> 5) + nln2;
          xjb = ((jb - undo) >> 5) + nln2;
          plain |= ja <= base_a + ka || (has_b && jb <= base_b + kb);
        }
        if (plain) {
          const int4 v = msv16_plain<G, C, ROWP>(my_rows, seq, L, j, gmask, tloop / 32, tmove, tbm_a, tbm_b, cap_a, cap_b, nln2);
          xja = v.x;
          xjb = v.y;
          biga = v.z;
          bigb = v.w;
        }
        if (j == 0) {
          const float uba = biga ? __int_as_float(0x7f800000) : bound(xja);
          const float ubb = bigb ? __int_as_float(0x7f800000) : bound(xjb);
          if (bound_out) {
            const int64_t o = slot ? slot[entry] : entry;
            bound_out[o] = uba;
            if (has_b) bound_out[bound_stride + o] = ubb;
          }
          if (rlist) {
            if (biga || bits_stat(uba, tp.z) >= s1a) {
              const unsigned pos = atomicAdd(&rcount[tile.pa - p0], 1u);
              if (pos < rcap) rlist[(int64_t)(tile.pa - p0) * rcap + pos] = tgt;
              else atomicOr(overflow, 1u);
            }
            if (has_b && (bigb || bits_stat(ubb, tp.z) >= s1b)) {
              const unsigned pos = atomicAdd(&rcount[tile.pb - p0], 1u);
              if (pos < rcap) rlist[(int64_t)(tile.pb - p0) * rcap + pos] = tgt;
              else atomicOr(overflow, 1u);
            }
          }
        }
      }
      int e = 0;
      if (j == 0) e = atomicAdd(&s_next, 1);
      e = __shfl_sync(gmask, e, gl);
      if (e < tile.end) {
        entry = e;
        const int tgt = list[e];
        L = tlen[tgt];
        seq = res + toff[tgt];
        const float4 tp = tpar[tgt];
        tloop = 32 * q32_up(tp.x);
        const int tmove = q32_up(tp.y);
        ka = 32 * (tmove + tbm_a + 2047);
        kb = 32 * (tmove + tbm_b + 2047);
        base_a = base_b = 0;  // N of row 0
        ja = jb = kJStart;
        biga = bigb = false;
        bcur = upper(ka, kb);
        active = L > 0;
      } else {
        active = false;
        done = true;
        L = 0;
        tloop = 0;
        base_a = base_b = base_idle;
      }
#pragma unroll
      for (int c = 0; c < C; c++) w[c] = bcur;
      row = 0;
      boff = 0;
      rcur = __ldg(reinterpret_cast<const uint4*>(seq));
      rnext = __ldg(reinterpret_cast<const uint4*>(seq + 16));
    }
    if (__all_sync(kFull, done)) break;

    const int q = (row - boff) >> 2;
    uint32_t word = q == 0 ? rcur.x : q == 1 ? rcur.y : q == 2 ? rcur.z : rcur.w;
    if (done) word = 0x18181818u;
    // the E (both halves) above which a row of the block can raise base: the
    // lowest of its rows, floor((base - nln2) / 2^-9 nat)
    unsigned limit = upper(base_a + 4 * tloop - nln2_25, base_b + 4 * tloop - nln2_25);
    auto row_of = [&](int r) { return my_rows + (int)((word >> (8 * r)) & 0xff) * ROWP + j; };
    constexpr int NPF = NC4 < 6 ? NC4 : 6;  // score chunks of a row loaded ahead, the highest columns (used first)
    uint4 ahead[NPF];
    const uint4* rowp = row_of(0);
#pragma unroll
    for (int u = 0; u < NPF; u++) ahead[u] = rowp[(NC4 - 1 - u) * G];
#pragma unroll
    for (int r = 0; r < 4; r++) {
      // B of the row unless its E raises base
      const unsigned bp = upper(base_a + ka + (r + 1) * tloop, base_b + kb + (r + 1) * tloop);
      uint4 rv[NC4];
#pragma unroll
      for (int c4 = 0; c4 < NC4; c4++) rv[c4] = c4 >= NC4 - NPF ? ahead[NC4 - 1 - c4] : rowp[c4 * G];
      unsigned left = __shfl_up_sync(kFull, w[C - 1], 1, G);
      if (j == 0) left = bcur;
      unsigned acc[4];
#pragma unroll
      for (int c = C - 1; c >= 0; c--) {
        const uint4& a4 = rv[c >> 2];
        const unsigned ra = (c & 3) == 0 ? a4.x : (c & 3) == 1 ? a4.y : (c & 3) == 2 ? a4.z : a4.w;
        w[c] = __viaddmax_s16x2(c ? w[c - 1] : left, ra, bp);
        if ((c & 1) == 0) {
          const int p = c / 2, a = p & 3;
          acc[a] = p + 4 < C / 2 ? __vimax3_s16x2(acc[a], w[c], w[c + 1]) : max2s16(w[c], w[c + 1]);
        }
      }
      if (r < 3) {
        rowp = row_of(r + 1);
#pragma unroll
        for (int u = 0; u < NPF; u++) ahead[u] = rowp[(NC4 - 1 - u) * G];
      }
      unsigned xe = __vimax3_s16x2(acc[0], acc[1], acc[2]);
      if (track) {
        const unsigned e = max2s16(xe, acc[3]);
        ja = __viaddmax_s32(ja, tloop, (int)(e << 16));
        jb = __viaddmax_s32(jb, tloop, (int)(e & 0xffff0000u));
      }
      xe = __vimax3_s16x2(xe, acc[3], limit);
      bcur = bp;
      if (__any_sync(kFull, xe != limit)) {
        // a row of some group may raise its base: every group takes its row
        // maximum (an E at the limit raises nothing), and w the B that follows
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) xe = max2s16(xe, __shfl_xor_sync(kFull, xe, o, G));
        biga |= (int)(short)(xe & 0xffffu) > cap_a;
        bigb |= ((int)xe >> 16) > cap_b;
        const int decay = (r + 1) * tloop;
        const int na = max(base_a + decay, (int)(xe << 16) + nln2_25), nb = max(base_b + decay, (int)(xe & 0xffff0000u) + nln2_25);
        base_a = na - decay;
        base_b = nb - decay;
        bcur = upper(na + ka, nb + kb);
        limit = upper(base_a + 4 * tloop - nln2_25, base_b + 4 * tloop - nln2_25);
#pragma unroll
        for (int c = 0; c < C; c++) w[c] = max2s16(w[c], bcur);
      }
    }
    base_a += 4 * tloop;
    base_b += 4 * tloop;
    row += 4;
    if (row - boff == 16) {
      boff += 16;
      rcur = rnext;
      if (active) rnext = __ldg(reinterpret_cast<const uint4*>(seq + boff + 16));
    }
  }
}

}  // namespace sxk

namespace sxk {

// ---------------------------------------------------------------------------
// Packed-integer Viterbi pre-screen: an upper bound of the reference's f32
// Viterbi score (src/hmmer/dp.rs:152-189) for 2 W targets of one profile at
// once, in W words of int16x2 (one target per half).
//
// Why: the exact lane-group kernel (viterbi_g_kernel) is bound by the
// latency of each row's sequential parts -- the D chain, the carry vote, the
// row-maximum butterfly, the special states -- by the per-row control around
// them, and by the 32 bytes of transitions it reads for every cell.  Here one
// pass of all of that serves 2 W pairs: every max(a + b, c) is one fused
// operation on two cells, W words share the transitions read from shared
// memory and fill each other's latency, and rows run in blocks of four without
// control flow:
//   * the D chain runs in every lane at once, first without a carry, then the
//     carries their left neighbours ended with run beside it until none changes
//     a lane's first column (integers: the fixed point is the sequential chain);
//   * N, J and B as in the MSV pre-screen: base = max(N, J) decays, a vote finds
//     the rows whose E raises it, J is kept per lane and combined at the end;
//   * rows past a target's end in its last block read a score row of -24 nats
//     (row 25 of the image), which raises nothing, and J's decay is undone.
// Bound: shared memory (8 transition words and 2 W score halves per W words of
// cells, 10 bytes a cell at W = 2 and 18 at W = 1) and the ALU pipe, about 11
// operations a word; short of either, the latency of a row at 8 to 12 warps
// per SM.  Measured on B200 (296 profiles of one length, their ~67,000 bias
// survivors of 12,000 targets; before: one word, carries pushed column by
// column, specials and a butterfly every row, list order): M = 60 4.3 -> 1.5
// ms, 100 5.2 -> 2.4, 208 7.5 -> 3.7, 300 14.2 -> 5.5, and the Pfam-scale
// search's 61 -> 33 ms (34 with the chains of all terms run again from every
// carry, 36 with a branch around lanes whose carry does not win).  M = 513 to 1536, exact before (600: 35 ms, 1000: 44),
// is pre-screened with one word: 1000 11.7 + 4.7 ms exact; 48 columns a lane
// spill, but still run 1.8 times the exact kernel's cells (a marker-set
// genome's Viterbi stage 18.3 -> 10.5 ms).
//
// Exactness.  As for the MSV pre-screen, the bound never decides a pair: a
// pair passes when its bound passes F2 (with the exact kernel's slack), and
// every passing pair is rescored by viterbi_g_kernel, so the survivors of
// the stage are exactly the reference's.  The bound holds by construction:
//   * cells are integers in units of q = 2^-9 nat.  Match scores are rounded
//     up after adding 2^-12 nat (more than the f32 rounding of one addition
//     for |value| < 4096 nats) and clamped up to -8 nats; transition scores
//     the same way, clamped up to -8 nats (t_bm: -16 nats) and down to 0 --
//     a transition t <= 0 never raises a value (fl(a + t) <= a), so 0 bounds
//     any t in [-2^-12, 0]; -inf scores become the floor.  Integer max-plus
//     over rounded-up scores is >= the real-valued recurrence, which is >=
//     the f32 recurrence minus its rounding; by induction every integer cell
//     is >= the f32 cell (max is exact and monotone; raising an input only
//     raises the result).  The insert rows ignore the '*' residue's
//     insert-state cut (dp.rs:172), which only raises I;
//   * the row maximum is taken over M alone: with every transition <= 0,
//     D[k] <= max over k' < k of M[k'] in f32 and in the integers alike;
//   * the specials are int32 in units of 2^-20 nat with every constant
//     rounded up after adding 2^-17 nat, as in the MSV pre-screen;
//   * the final bound (xJ + tmove at row L, rounded up to f32) goes through
//     the exact kernel's f32 bit statistic, which is monotone.
// int16 range: B + t_bm >= -24 nats, so M >= -32 nats in a row of real scores
// and -48 in a row past a target's end (at -24 nats a score; the three rows
// after a target at most, before its words are set anew), D, I and pre one
// transition below, and no sum more than one transition below those: -64 nats,
// the least an int16 holds.  Every value is <= the previous rows' maximum plus
// the largest match score, so a row maximum above the profile's cap (32767 minus
// that score) marks the pair as passing before anything can wrap (sticky).
// Columns past M carry the floor scores; the profile's quantized image has
// the kernel's width G*C and the CPU model follows the same columns.
// ---------------------------------------------------------------------------
constexpr int kV16TFloor = -4096;    // -8 nats: lowest transition score (t_bm excepted)
constexpr int kV16BmFloor = -8192;   // -16 nats: lowest t_bm
constexpr int kV16EFloor = -4096;    // -8 nats: lowest match score, and columns past M
constexpr int kV16BFloor = -4096;    // -8 nats: lowest B state
constexpr unsigned kV16Init2 = 0xc000c000u;  // (-16384, -16384): -inf before row 1 / left of column 1
constexpr unsigned kV16Low2 = 0xa000a000u;   // (-24576, -24576): no D carry into a lane
constexpr int kV16EPast = -12288;    // -24 nats: scores of the rows past a target's end
constexpr unsigned kV16BFloor2 = 0xf000f000u;
// B + t_bm + e, then D, I or pre from it, then a further transition
static_assert(kV16BFloor + kV16BmFloor + kV16EPast + 2 * kV16TFloor >= -32768 && kV16EPast <= kV16EFloor,
              "Viterbi sums leave int16");
constexpr int kV16Rows = 26;         // score rows of an image: 25 residue codes and the row past the end

constexpr int kV16Tile = 1024;       // entries of a tile that are ordered by length
constexpr int kV16Buckets = 64;      // of 32 residues

// One profile x every nsub-th entry (from sub) of its Viterbi pre-screen list.
struct VitTile {
  int32_t p, sub, nsub, pad;
};

// int16x2 helper: replace one half of a word by the same half of v.
__device__ __forceinline__ unsigned set_half(unsigned w, int h, unsigned v) {
  return h ? __byte_perm(w, v, 0x7610) : __byte_perm(w, v, 0x3254);
}

// Bound of pairs of one profile (tile.p) against the targets of its list
// (region (p - p0) * vcap of `vlist`, vcount[p - p0] entries).  The profile's
// quantized image (qv_off, uint4 units): 8 transition rows of W/4 uint4 (each
// column's score in both halves: t_mm t_im t_dm at k-1, t_bm t_mi t_ii at k,
// t_md t_dd at k-1), then kV16Rows match-score rows of W/4 uint2 (4 columns of
// int16), both in the lane-major chunk layout of the f32 Viterbi image.
// Per pair: with `score_out`, the bound (f32 nats; +inf when capped, NaN for
// an empty target) goes to score_out[slot]; otherwise a pair whose bound
// passes F2 is appended to the exact Viterbi's list (bin vshape).  stats[0..2]
// accumulate the DP cells bounded, the cells of the passing pairs and the
// passing pairs.
template <int G, int C, int W>
__global__ void __launch_bounds__(128, (C * W <= 16 ? 3 : 2)) vit16_kernel(
    const VitTile* __restrict__ tiles, const DevProfile* __restrict__ profs, const Thresholds* __restrict__ thr,
    const uint4* __restrict__ qvimg, const uint8_t* __restrict__ res, const int64_t* __restrict__ toff,
    const int32_t* __restrict__ tlen, const float4* __restrict__ xsc, const PairRec* __restrict__ vlist,
    unsigned vcap, const unsigned* __restrict__ vcount, int p0, PairRec* __restrict__ out,
    const BinRegion* __restrict__ out_bins, unsigned* __restrict__ out_counts, unsigned* __restrict__ overflow,
    float slack, float* __restrict__ score_out, double* __restrict__ stats) {
  static_assert(C % 8 == 0 && (G & (G - 1)) == 0 && G <= 32, "bad packed Viterbi shape");
  constexpr int NC4 = C / 4;
  constexpr int ROW4 = NC4 * G;  // uint4 per transition row, uint2 per score row
  constexpr int H = 2 * W;       // targets of a group
  constexpr int NIMG4 = 8 * ROW4 + kV16Rows * ROW4 / 2;
  extern __shared__ uint4 sm_v[];
  __shared__ unsigned s_next;
  __shared__ unsigned s_at[kV16Buckets];
  __shared__ uint16_t s_order[kV16Tile];
  const VitTile tile = tiles[blockIdx.x];
  const DevProfile& P = profs[tile.p];
  {
    const uint4* src = qvimg + P.qv_off;
    for (int q = threadIdx.x; q < NIMG4; q += blockDim.x) sm_v[q] = src[q];
  }
  const unsigned n = min(vcount[tile.p - p0], vcap);
  const PairRec* lst = vlist + (int64_t)(tile.p - p0) * vcap;
  // the tile's entries, longest targets first, so that no long target starts
  // when the others are about to end (a tile past the order's room keeps the
  // list's)
  const unsigned mine = n > (unsigned)tile.sub ? (n - tile.sub + tile.nsub - 1) / tile.nsub : 0;
  const bool ordered = mine <= kV16Tile;
  if (threadIdx.x == 0) s_next = 0;
  for (int q = threadIdx.x; q < kV16Buckets; q += blockDim.x) s_at[q] = 0;
  __syncthreads();
  if (ordered) {
    auto bucket = [&](unsigned k) {
      return kV16Buckets - 1 - min(kV16Buckets - 1, tlen[lst[tile.sub + k * tile.nsub].t] >> 5);
    };
    for (unsigned k = threadIdx.x; k < mine; k += blockDim.x) atomicAdd(&s_at[bucket(k)], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive prefix sums
      unsigned before = 0;
      for (int q = 0; q < kV16Buckets; q += 32) {
        const unsigned v = s_at[q + threadIdx.x];
        unsigned inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned up = __shfl_up_sync(kFull, inc, o);
          if ((int)threadIdx.x >= o) inc += up;
        }
        s_at[q + threadIdx.x] = before + inc - v;
        before += __shfl_sync(kFull, inc, 31);
      }
    }
    __syncthreads();
    for (unsigned k = threadIdx.x; k < mine; k += blockDim.x) s_order[atomicAdd(&s_at[bucket(k)], 1u)] = (uint16_t)k;
  }
  __syncthreads();

  const int lane = threadIdx.x & 31;
  const int j = lane & (G - 1);
  const int gl = lane - j;
  const unsigned gmask = (G == 32) ? kFull : (((1u << G) - 1u) << gl);
  const int cap = P.qv_cap;
  const int nln2 = (int)ceilf(-0.693147182464599609375f * 1048576.0f) + kQ32Rho;
  const int nln2_25 = 32 * nln2;
  constexpr int kJStart = -60 * (1 << 25);
  const int base_idle = 32767 * 65536 + nln2_25;  // a base no E raises
  const uint4* tr = sm_v + j;
  const uint2* es = reinterpret_cast<const uint2*>(sm_v + 8 * ROW4) + j;
  const uint32_t* words = reinterpret_cast<const uint32_t*>(res);  // targets start on 16-byte boundaries
  auto T = [&](int q, int c4) -> uint4 { return tr[(q * NC4 + c4) * G]; };
  auto pick = [](const uint4& v, int e) -> unsigned { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; };
  auto upper = [](int a, int b) { return __byte_perm((unsigned)a, (unsigned)b, 0x7632); };  // int16 of two states

  // rows carried on: I, D and pre = max(M + t_mm, I + t_im) of the next row
  unsigned ip[W][C], dp[W][C], pre[W][C];
  unsigned dpl[W], bw[W];  // D left of the lane's first column; B of the row being computed
#pragma unroll
  for (int w = 0; w < W; w++) {
#pragma unroll
    for (int c = 0; c < C; c++) ip[w][c] = dp[w][c] = pre[w][c] = kV16Init2;
    dpl[w] = kV16Init2;
    bw[w] = kV16BFloor2;
  }
  // per target, in 2^-25 nat: base, tloop, the constant of B (tmove + 2047 /
  // 2^20) and J of this lane's columns; rows left, its list entry, the index of
  // the residue word after the fetched ones, this block's word and the next
  int base[H], tl[H], tk[H], jj[H], rem[H];
  unsigned idx[H], wi[H], cur[H], nxt[H];
#pragma unroll
  for (int h = 0; h < H; h++) {
    base[h] = base_idle;
    tl[h] = tk[h] = rem[h] = 0;
    jj[h] = kJStart;
    idx[h] = wi[h] = 0;
    cur[h] = nxt[h] = 0;
  }
  unsigned active = 0, done = 0, big = 0;  // by target
  double cells_in = 0.0, cells_pass = 0.0, npass = 0.0;

  for (;;) {
#pragma unroll
    for (int h = 0; h < H; h++) {
      if (!(done >> h & 1) && rem[h] <= 0) {  // group-uniform: finish this target, take the next one
        if (active >> h & 1) {
          int jm = jj[h];
#pragma unroll
          for (int o = G / 2; o >= 1; o >>= 1) jm = max(jm, __shfl_xor_sync(gmask, jm, o, G));
          if (j == 0) {
            const PairRec r = lst[idx[h]];
            const int L = tlen[r.t];
            const int xj = ((jm + rem[h] * tl[h]) >> 5) + nln2;  // at row L: rem is minus the rows past it
            const float ub = L == 0              ? __int_as_float(0x7fc00000)
                             : (big >> h & 1)    ? __int_as_float(0x7f800000)
                                                 : __fmul_rn(__int2float_ru(xj + q32_up(xsc[r.t].y)), 9.5367431640625e-7f);
            if (score_out) {
              score_out[r.slot] = ub;
            } else if (L > 0) {
              const double cells = (double)P.m * (double)L;
              cells_in += cells;
              if ((big >> h & 1) || bits_stat(ub, r.filtersc) >= thr[tile.p].s2 - slack) {
                push_pair(r, P.vshape, out, out_bins, out_counts, overflow);
                cells_pass += cells;
                npass += 1.0;
              }
            }
          }
        }
        unsigned k = 0;
        if (j == 0) k = atomicAdd(&s_next, 1u);
        k = __shfl_sync(gmask, k, gl);
        big &= ~(1u << h);
        jj[h] = kJStart;
        if (k < mine) {
          const unsigned e = (unsigned)tile.sub + (ordered ? s_order[k] : k) * (unsigned)tile.nsub;
          idx[h] = e;
          const int t = lst[e].t;
          rem[h] = tlen[t];
          wi[h] = (unsigned)(toff[t] >> 2);
          cur[h] = __ldg(words + wi[h]);
          nxt[h] = __ldg(words + wi[h] + 1);
          wi[h] += 2;
          const float4 xs = xsc[t];
          tl[h] = 32 * q32_up(xs.x);
          tk[h] = 32 * (q32_up(xs.y) + 2047);
          base[h] = 0;  // N of row 0
          active |= 1u << h;
          const int w = h >> 1;
#pragma unroll
          for (int c = 0; c < C; c++) {
            ip[w][c] = set_half(ip[w][c], h & 1, kV16Init2);
            dp[w][c] = set_half(dp[w][c], h & 1, kV16Init2);
            pre[w][c] = set_half(pre[w][c], h & 1, kV16Init2);
          }
          dpl[w] = set_half(dpl[w], h & 1, kV16Init2);
          bw[w] = set_half(bw[w], h & 1, max2s16(upper(tk[h], tk[h]), kV16BFloor2));
        } else {
          active &= ~(1u << h);
          done |= 1u << h;
          rem[h] = 0;
          tl[h] = 0;
          base[h] = base_idle;
        }
      }
    }
    if (__all_sync(kFull, done == (1u << H) - 1u)) break;

    // the block's residues; 25 from the target's end on
    unsigned rw[H];
#pragma unroll
    for (int h = 0; h < H; h++) {
      const unsigned past = rem[h] >= 4 ? 0u : 0xffffffffu << (8 * max(rem[h], 0));
      rw[h] = (cur[h] & ~past) | (0x19191919u & past);
      cur[h] = nxt[h];
      if (active >> h & 1) nxt[h] = __ldg(words + wi[h]);
      wi[h]++;
    }
#pragma unroll 1
    for (int r = 0; r < 4; r++) {
      unsigned m[W][C];
      // match scores of both halves, interleaved into words
#pragma unroll
      for (int w = 0; w < W; w++) {
        const uint2* ea = es + (int)(rw[2 * w] & 0xffu) * ROW4;
        const uint2* eb = es + (int)(rw[2 * w + 1] & 0xffu) * ROW4;
        rw[2 * w] >>= 8;
        rw[2 * w + 1] >>= 8;
#pragma unroll
        for (int c4 = 0; c4 < NC4; c4++) {
          const uint2 a = ea[c4 * G], b = eb[c4 * G];
          m[w][4 * c4 + 0] = __byte_perm(a.x, b.x, 0x5410);
          m[w][4 * c4 + 1] = __byte_perm(a.x, b.x, 0x7632);
          m[w][4 * c4 + 2] = __byte_perm(a.y, b.y, 0x5410);
          m[w][4 * c4 + 3] = __byte_perm(a.y, b.y, 0x7632);
        }
      }
      // ---- M: max(pre, D[k-1] + t_dm, B + t_bm) + msc (dp.rs:167-169) ----
#pragma unroll
      for (int c4 = 0; c4 < NC4; c4++) {
        const uint4 tdm = T(2, c4), tbm = T(3, c4);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const int c = 4 * c4 + e;
#pragma unroll
          for (int w = 0; w < W; w++) {
            const unsigned v = __viaddmax_s16x2(c ? dp[w][c - 1] : dpl[w], pick(tdm, e), pre[w][c]);
            m[w][c] = add2s16(__viaddmax_s16x2(bw[w], pick(tbm, e), v), m[w][c]);
          }
        }
      }
      // ---- D: every lane's chain without a carry, then from its neighbour's end ----
      unsigned ml[W], il[W], cin[W];
#pragma unroll
      for (int w = 0; w < W; w++) {
        ml[w] = __shfl_up_sync(kFull, m[w][C - 1], 1, G);
        il[w] = __shfl_up_sync(kFull, ip[w][C - 1], 1, G);
        if (j == 0) ml[w] = il[w] = kV16Init2;
        cin[w] = j ? kV16Low2 : kV16Init2;
      }
      {
        unsigned d[W];
#pragma unroll
        for (int w = 0; w < W; w++) d[w] = cin[w];
#pragma unroll
        for (int c4 = 0; c4 < NC4; c4++) {
          const uint4 tmd = T(6, c4), tdd = T(7, c4);
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const int c = 4 * c4 + e;
#pragma unroll
            for (int w = 0; w < W; w++)
              dp[w][c] = d[w] = __viaddmax_s16x2(d[w], pick(tdd, e), add2s16(c ? m[w][c - 1] : ml[w], pick(tmd, e)));
          }
        }
      }
      // a lane's D is the larger of its own chain and its carry's; every round that changes a
      // lane's end moves the carries one lane on, so the vote ends the loop.
      for (int it = 0; it < G; it++) {
        const unsigned t0 = T(7, 0).x;
        bool need = false;
#pragma unroll
        for (int w = 0; w < W; w++) {
          const unsigned up = __shfl_up_sync(kFull, dp[w][C - 1], 1, G);
          cin[w] = j ? up : kV16Init2;
          need |= __viaddmax_s16x2(cin[w], t0, dp[w][0]) != dp[w][0];
        }
        if (!__any_sync(kFull, need)) break;
        unsigned d[W];
#pragma unroll
        for (int w = 0; w < W; w++) d[w] = cin[w];
#pragma unroll
        for (int c4 = 0; c4 < NC4; c4++) {
          const uint4 tdd = T(7, c4);
#pragma unroll
          for (int e = 0; e < 4; e++)
#pragma unroll
            for (int w = 0; w < W; w++) dp[w][4 * c4 + e] = d[w] = __viaddmax_s16x2(d[w], pick(tdd, e), dp[w][4 * c4 + e]);
        }
      }
#pragma unroll
      for (int w = 0; w < W; w++) dpl[w] = cin[w];
      // ---- the next row's pre and I, in place ----
#pragma unroll
      for (int c4 = NC4 - 1; c4 >= 0; c4--) {
        const uint4 tmm = T(0, c4), tim = T(1, c4), tmi = T(4, c4), tii = T(5, c4);
#pragma unroll
        for (int e = 3; e >= 0; e--) {
          const int c = 4 * c4 + e;
#pragma unroll
          for (int w = 0; w < W; w++) {
            pre[w][c] = __viaddmax_s16x2(c ? m[w][c - 1] : ml[w], pick(tmm, e), add2s16(c ? ip[w][c - 1] : il[w], pick(tim, e)));
            ip[w][c] = __viaddmax_s16x2(m[w][c], pick(tmi, e), add2s16(ip[w][c], pick(tii, e)));
          }
        }
      }
      // ---- row maximum over M (D never exceeds it) of the lane's columns, J, base and B ----
      bool raise = false;
      unsigned xe[W];
#pragma unroll
      for (int w = 0; w < W; w++) {
        unsigned a = max2s16(m[w][0], m[w][1]), b = max2s16(m[w][2], m[w][3]);
#pragma unroll
        for (int c = 4; c < C; c += 4) {
          a = __vimax3_s16x2(a, m[w][c], m[w][c + 1]);
          b = __vimax3_s16x2(b, m[w][c + 2], m[w][c + 3]);
        }
        xe[w] = max2s16(a, b);
        jj[2 * w] = __viaddmax_s32(jj[2 * w], tl[2 * w], (int)(xe[w] << 16));
        jj[2 * w + 1] = __viaddmax_s32(jj[2 * w + 1], tl[2 * w + 1], (int)(xe[w] & 0xffff0000u));
        base[2 * w] += tl[2 * w];
        base[2 * w + 1] += tl[2 * w + 1];
        const unsigned limit = upper(base[2 * w] - nln2_25, base[2 * w + 1] - nln2_25);
        raise |= max2s16(xe[w], limit) != limit;
      }
      if (__any_sync(kFull, raise)) {
#pragma unroll
        for (int w = 0; w < W; w++) {
          unsigned x = xe[w];
#pragma unroll
          for (int o = G / 2; o >= 1; o >>= 1) x = max2s16(x, __shfl_xor_sync(kFull, x, o, G));
          if ((int)(short)(x & 0xffffu) > cap) big |= 1u << (2 * w);
          if (((int)x >> 16) > cap) big |= 2u << (2 * w);
          base[2 * w] = max(base[2 * w], (int)(x << 16) + nln2_25);
          base[2 * w + 1] = max(base[2 * w + 1], (int)(x & 0xffff0000u) + nln2_25);
        }
      }
#pragma unroll
      for (int w = 0; w < W; w++) bw[w] = max2s16(upper(base[2 * w] + tk[2 * w], base[2 * w + 1] + tk[2 * w + 1]), kV16BFloor2);
    }
#pragma unroll
    for (int h = 0; h < H; h++) rem[h] -= done >> h & 1 ? 0 : 4;
  }
  // stats: one atomic per warp
  if (stats) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
      cells_in += __shfl_xor_sync(kFull, cells_in, o);
      cells_pass += __shfl_xor_sync(kFull, cells_pass, o);
      npass += __shfl_xor_sync(kFull, npass, o);
    }
    if (lane == 0 && cells_in != 0.0) {
      atomicAdd(stats + 0, cells_in);
      atomicAdd(stats + 1, cells_pass);
      atomicAdd(stats + 2, npass);
    }
  }
}

}  // namespace sxk
