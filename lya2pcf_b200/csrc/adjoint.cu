// Adjoint of the pair histograms (no reference counterpart).
//
// Loss L = sum_b g_b xi_b with xi_b = DW_b / W_b (totals over all owner slots
// of the last lya_corr_run), pair bins held fixed.  For every in-range pixel
// pair (i, j) in bin b:
//   dL/d(dw_i) += (g_b / W_b) dw_j            dL/d(w_i) += -(g_b xi_b / W_b) w_j
// and symmetrically for j.  Bins with W_b == 0 contribute nothing (xi_b = 0,
// as post_processing.py:147 defines it).
//
// Two kernels share the work queue.  k_adjoint_band takes the pairs of forests
// whose dc are sorted, finite and not negative (the LYA_LEAN flag), where that
// pays (band_takes_lean), and serves both forests of a pair in one pass;
// k_adjoint takes the others: the gather
// form, walked in both directions, one lane per pixel i over its partners j,
// every bin from the reference FP64 formula.  The pair bin is symmetric under
// the swap (|dc1-dc2|, dc1+dc2 and the FMA-ordered cos12 are).
#include <algorithm>
#include <cmath>

#include "lya_internal.cuh"

namespace {

struct AdjParams {
  const double* __restrict__ dc;
  const double* __restrict__ w;
  const double* __restrict__ dw;
  const int64_t* __restrict__ pstart;
  const int32_t* __restrict__ len;
  const uint8_t* __restrict__ sorted;
  const double* __restrict__ ux;
  const double* __restrict__ uy;
  const double* __restrict__ uz;
  const int32_t* __restrict__ f1;
  const int32_t* __restrict__ f2;
  int64_t n_items;
  double binner_rp, binner_rt;
  int np, nt, nb, cos_variant;
  int skip_lean;                     // k_adjoint: leave the pairs k_adjoint_band takes
  const double* __restrict__ coef;   // [2][nb]: g/W, -g xi/W
  double* __restrict__ g_dw;         // padded pixel layout
  double* __restrict__ g_w;
};

__global__ void k_coef(int nslots, int nb, const double* __restrict__ hist, const double* __restrict__ g,
                       double* __restrict__ coef) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
    double W = 0.0, DW = 0.0;
    for (int s = 0; s < nslots; ++s) {
      const double* h = hist + (size_t)s * LYA_NQ * 2 * nb;
      W += h[(0 * 2 + 0) * nb + b] + h[(0 * 2 + 1) * nb + b];
      DW += h[(1 * 2 + 0) * nb + b] + h[(1 * 2 + 1) * nb + b];
    }
    double cdw = 0.0, cw = 0.0;
    if (W != 0.0) {
      cdw = g[b] / W;
      cw = -g[b] * (DW / W) / W;
    }
    coef[b] = cdw;
    coef[nb + b] = cw;
  }
}

// Totals over all slots of the last run: W[b] and DW[b] (hi + lo of each slot).
__global__ void k_totals(int nslots, int nb, const double* __restrict__ hist, double* __restrict__ W,
                         double* __restrict__ DW) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < nb; b += gridDim.x * blockDim.x) {
    double w = 0.0, dw = 0.0;
    for (int s = 0; s < nslots; ++s) {
      const double* h = hist + (size_t)s * LYA_NQ * 2 * nb;
      w += h[(0 * 2 + 0) * nb + b] + h[(0 * 2 + 1) * nb + b];
      dw += h[(1 * 2 + 0) * nb + b] + h[(1 * 2 + 1) * nb + b];
    }
    W[b] = w;
    DW[b] = dw;
  }
}

// Reversed-direction flag is in the item index: items [0, n) are (f1, f2),
// items [n, 2n) are (f2, f1).
__global__ void __launch_bounds__(256) k_adjoint(const AdjParams p) {
  extern __shared__ __align__(16) double s_coef[];   // [nb][2]: g/W, -g xi/W of a bin side by side (one 16-byte load)
  for (int k = threadIdx.x; k < 2 * p.nb; k += blockDim.x) s_coef[k] = p.coef[(k & 1) * p.nb + (k >> 1)];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t gw = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t t = gw; t < 2 * p.n_items; t += nw) {
    const bool rev = t >= p.n_items;
    const int64_t k = rev ? t - p.n_items : t;
    const int fa = rev ? p.f2[k] : p.f1[k];
    const int fb = rev ? p.f1[k] : p.f2[k];
    if (p.skip_lean && (p.sorted[fa] & p.sorted[fb] & LYA_LEAN)) continue;
    const int L1 = p.len[fa], L2 = p.len[fb];
    if (L1 <= 0 || L2 <= 0) continue;
    const int64_t a = p.pstart[fa], b = p.pstart[fb];
    double c = lya_cos12(p.ux[fa], p.uy[fa], p.uz[fa], p.ux[fb], p.uy[fb], p.uz[fb], p.cos_variant);
    c = fmin(1.0, fmax(-1.0, c));
    const double ch = __dsqrt_rn(__dmul_rn(0.5, __dadd_rn(1.0, c)));
    const double sh = __dsqrt_rn(__dmul_rn(0.5, __dsub_rn(1.0, c)));
    const bool srt = p.sorted[fa] && p.sorted[fb];
    const double rp_reach = ch > 0.0 ? ((double)p.np + 1e-3) / (ch * p.binner_rp) : 1e300;
    const double rt_reach = sh > 0.0 ? ((double)p.nt + 1e-3) / (sh * p.binner_rt) : 1e300;
    const double* __restrict__ D2 = p.dc + b;
    const double* __restrict__ W2 = p.w + b;
    const double* __restrict__ DW2 = p.dw + b;
    for (int i0 = 0; i0 < L1; i0 += 32) {
      const int i = i0 + lane;
      double gdw = 0.0, gw_ = 0.0;
      if (i < L1) {
        const double d1 = p.dc[a + i];
        int jlo = 0, jhi = L2;
        if (srt) {
          const double margin = 1e-6 * fabs(d1) + 1e-6;
          const double tlo = d1 - rp_reach - margin;
          const double thi = fmin(d1 + rp_reach, rt_reach - d1) + margin;
          int x = 0, y = L2;
          while (x < y) { const int m = (x + y) >> 1; if (D2[m] > tlo) y = m; else x = m + 1; }
          jlo = x;
          y = L2;
          while (x < y) { const int m = (x + y) >> 1; if (D2[m] < thi) x = m + 1; else y = m; }
          jhi = x;
        }
        // bin of (d1, d2) with the reference FP64 formula, -1 out of range
        auto pbin = [&](double d2) {
          const double rp = __dmul_rn(fabs(__dsub_rn(d1, d2)), ch);
          const double rt = __dmul_rn(__dadd_rn(d1, d2), sh);
          const double fp = floor(__dmul_rn(rp, p.binner_rp));
          const double ft = floor(__dmul_rn(rt, p.binner_rt));
          return (fp >= 0.0 && fp < (double)p.np && ft >= 0.0 && ft < (double)p.nt) ? (int)fp * p.nt + (int)ft : -1;
        };
        // four partners at a time: independent bin chains, then the sums in partner order
        int j = jlo;
        for (; j + 4 <= jhi; j += 4) {
          int bin[4];
          double dwj[4], wj[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            bin[u] = pbin(D2[j + u]);
            dwj[u] = DW2[j + u];
            wj[u] = W2[j + u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            if (bin[u] >= 0) {
              const double2 cc = reinterpret_cast<const double2*>(s_coef)[bin[u]];
              gdw = __fma_rn(cc.x, dwj[u], gdw);
              gw_ = __fma_rn(cc.y, wj[u], gw_);
            }
          }
        }
        for (; j < jhi; ++j) {
          const int bn = pbin(D2[j]);
          if (bn >= 0) {
            const double2 cc = reinterpret_cast<const double2*>(s_coef)[bn];
            gdw = __fma_rn(cc.x, DW2[j], gdw);
            gw_ = __fma_rn(cc.y, W2[j], gw_);
          }
        }
        if (gdw != 0.0) atomicAdd(&p.g_dw[a + i], gdw);
        if (gw_ != 0.0) atomicAdd(&p.g_w[a + i], gw_);
      }
    }
  }
}

// ------------------------------------------------------------------ pairs of lean forests
// One warp per forest pair, 64 rows (f1 pixels) at a time: lane l holds rows
// r = i0 + 2l and r + 1 and at step m the f2 pixel j = r + m, so all lanes are
// on the same two diagonals, nearly the same |dc1 - dc2|, and cross the rp edges
// within a step or two of one another.
// * Bins: x = dc_j - dc_i and s = dc_j + dc_i grow with m, so each row walks the
//   pair's rp edges (both signs of x) and rt edges upwards, comparing x and s
//   with the next exact edge (lya_edge) instead of forming the bin of every
//   pixel pair.  The steps of a row's rt edges, at most a few, are found before
//   the walk, which leaves one FP64 addition and one comparison per pair.
// * Gradients: a row's sums stay in its lane.  The sums of pixel j move one
//   lane down every second step (two sets, even and odd steps), leave at lane 0
//   into a ring of 32 pixels and go to memory 32 pixels at a time.
// * f2 pixels pass through a ring in shared memory, even and odd pixels apart,
//   so that the lanes' reads (two pixels apart) are conflict-free.
// Bound: issue (72% of cycles) and shared-memory wavefronts (70%); the FP64 pipe
// is at 25% (6 operations per pixel pair for both directions; the gather form
// needs 28).  One gradient of 2.80e10 pixel pairs (2,500 forests of 374 pixels):
// 48.9 ms, the gather form over both directions 99.6 ms; 1.85e9 pairs of
// 200-pixel forests: 4.56 against 8.6 ms.  24 warps at 80 registers: 20 warps
// take 50.4 ms, 28 warps 55.3 ms.  Byte offsets in place of indices and 32-bit
// words for the rt steps: 62.8 -> 48.9 ms.
constexpr int BAND_WARPS = 24;   // at most (80 registers)
constexpr int BAND_RING = 128;   // f2 pixels in a warp's ring: 64 in use, 32 ahead, 32 spare

// Shared memory, as offsets in doubles: the coefficients (2 values) of the nt
// bins of every number of rp edges passed (0 .. 2 np, the first and the last out
// of range), then per warp the ring (w, dw) of even and odd pixels, the ring's
// distances, the (grad dw, grad w) of 32 finished f2 pixels, the rp edges
// [2 np + 1] and the rt edges [nt + 1].
constexpr int BAND_D = 2 * BAND_RING, BAND_OUT = BAND_D + BAND_RING, BAND_EX = BAND_OUT + 64;
__host__ __device__ __forceinline__ int band_table(int np, int nt) { return 2 * (2 * np + 1) * nt; }
__host__ __device__ __forceinline__ int band_per_warp(int np, int nt) { return BAND_EX + ((2 * np + 1 + nt + 1 + 1) & ~1); }
extern __shared__ __align__(16) double s_band[];
// shared memory at a byte offset (rows keep byte offsets: no address arithmetic in the walk)
__device__ __forceinline__ double band_d(int at) { return *reinterpret_cast<const double*>(reinterpret_cast<const char*>(s_band) + at); }
__device__ __forceinline__ double2 band_d2(int at) { return *reinterpret_cast<const double2*>(reinterpret_cast<const char*>(s_band) + at); }

// Bin state of a row: the byte offsets ox of the next rp edge and oc of the bin's
// coefficients, the next rp edge, and the steps of its next four rt edges (kt,
// then kt2: 16 bits each, the nearest lowest).  The row's partners are in range
// on steps kb .. kb + kn - 1.
struct BandRow {
  double d, w, dw;
  double ex;
  double gdw, gw;
  unsigned kt, kt2;
  int ox, oc, kb, kn;
};

__device__ __forceinline__ int edges_passed(int e, int n, double v) {   // entries of s_band[e .. e + n) that are <= v
  int lo = 0, hi = n;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (v >= s_band[e + mid]) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ void band_sums(BandRow& r, int k, const double2& wdw, double& jdw, double& jw) {
  const double2 c = band_d2(r.oc);
  if ((unsigned)(k - r.kb) < (unsigned)r.kn) {
    r.gdw = __fma_rn(c.x, wdw.y, r.gdw);
    r.gw = __fma_rn(c.y, wdw.x, r.gw);
    jdw = __fma_rn(c.x, r.dw, jdw);
    jw = __fma_rn(c.y, r.w, jw);
  }
}

// Pass the edges up to the pixel at distance d2, step k.  SINGLE: at most one rp
// and one rt edge per step (half of the lanes pass an rp edge at each step of
// 2 Mpc/h) and at most four rt edges per row, whose steps are known: no branch.
template <bool SINGLE>
__device__ __forceinline__ void band_edges(BandRow& r, double d2, int k, int nt16, int es) {
  const double x = __dsub_rn(d2, r.d);
  if (SINGLE) {
    if (x >= r.ex) { r.ox += 8; r.oc += nt16; }
    r.ex = band_d(r.ox);
    if ((r.kt & 0xffffu) == (unsigned)k) {
      r.oc += 16;
      r.kt = __funnelshift_r(r.kt, r.kt2, 16);
      r.kt2 = r.kt2 >> 16 | 0xffff0000u;
    }
  } else {
    while (x >= r.ex) { r.ox += 8; r.ex = band_d(r.ox); r.oc += nt16; }
    const double s = __dadd_rn(d2, r.d);
    while (s >= s_band[es + (int)r.kt]) { ++r.kt; r.oc += 16; }   // kt: rt edges passed
  }
}

// The pixel pairs of both rows and the f2 pixel at ring position q of parity
// par (step k), whose sums are jdw, jw.
template <bool SINGLE>
__device__ __forceinline__ void band_pair(BandRow& ra, BandRow& rb, int ring, int par, int q, int k, double& jdw,
                                          double& jw, int nt16, int es) {
  const double2 wdw = band_d2(8 * ring + par * 8 * BAND_RING + 16 * q);
  const double d2 = band_d(8 * ring + 8 * BAND_D + par * 4 * BAND_RING + 8 * q);
  band_edges<SINGLE>(ra, d2, k, nt16, es);
  band_edges<SINGLE>(rb, d2, k, nt16, es);
  band_sums(ra, k, wdw, jdw, jw);
  band_sums(rb, k, wdw, jdw, jw);
}

// Sums of the f2 pixels of the current two steps (even, odd), one pixel per lane each.
struct BandCols {
  double pdw, pw, qdw, qw;
};

// n steps (rounded up to even: a step past the band meets only pairs out of
// range or outside the forest) from ring position k0.
template <bool SINGLE>
__device__ __forceinline__ void band_walk(BandRow& ra, BandRow& rb, BandCols& c, int ring, int k0, int n, int nt16, int es) {
  const int lane = threadIdx.x & 31;
  for (int k = 0; k < n; k += 2) {
    const int q = (((k0 + k) >> 1) + lane) & (BAND_RING / 2 - 1);
    band_pair<SINGLE>(ra, rb, ring, 0, q, k0 + k, c.pdw, c.pw, nt16, es);
    band_pair<SINGLE>(ra, rb, ring, 1, q, k0 + k + 1, c.qdw, c.qw, nt16, es);
    if (lane == 0) {
      *reinterpret_cast<double2*>(&s_band[ring + BAND_OUT + 2 * k]) = make_double2(c.pdw, c.pw);
      *reinterpret_cast<double2*>(&s_band[ring + BAND_OUT + 2 * k + 2]) = make_double2(c.qdw, c.qw);
    }
    c.pdw = __shfl_down_sync(0xffffffffu, c.pdw, 1); c.pw = __shfl_down_sync(0xffffffffu, c.pw, 1);
    c.qdw = __shfl_down_sync(0xffffffffu, c.qdw, 1); c.qw = __shfl_down_sync(0xffffffffu, c.qw, 1);
    if (lane == 31) { c.pdw = 0.0; c.pw = 0.0; c.qdw = 0.0; c.qw = 0.0; }
  }
}

__global__ void __launch_bounds__(BAND_WARPS * 32, 1) k_adjoint_band(const AdjParams p) {
  constexpr unsigned FULL = 0xffffffffu;
  const int np = p.np, nt = p.nt, nb = p.nb;
  for (int k = threadIdx.x; k < (2 * np + 1) * nt; k += blockDim.x) {
    const int q = abs(k / nt - np) * nt + k % nt;
    s_band[2 * k] = q < nb ? p.coef[q] : 0.0;
    s_band[2 * k + 1] = q < nb ? p.coef[nb + q] : 0.0;
  }
  const int nt16 = 16 * nt;   // bytes of a coefficient row
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ring = band_table(np, nt) + warp * band_per_warp(np, nt);
  const int ex = ring + BAND_EX, es = ex + 2 * np + 1;
  const double NaN = __longlong_as_double(0x7ff8000000000000ll), INF = __longlong_as_double(0x7ff0000000000000ll);
  __syncthreads();
  const int warps = blockDim.x >> 5;
  const int64_t nw = (int64_t)gridDim.x * warps;
  for (int64_t t = blockIdx.x * (int64_t)warps + warp; t < p.n_items; t += nw) {
    const int fa = p.f1[t], fb = p.f2[t];
    if (!(p.sorted[fa] & p.sorted[fb] & LYA_LEAN)) continue;
    const int L1 = p.len[fa], L2 = p.len[fb];
    if (L1 <= 0 || L2 <= 0) continue;
    const int64_t a = p.pstart[fa], b = p.pstart[fb];
    double c = lya_cos12(p.ux[fa], p.uy[fa], p.uz[fa], p.ux[fb], p.uy[fb], p.uz[fb], p.cos_variant);
    c = fmin(1.0, fmax(-1.0, c));
    const double ch = __dsqrt_rn(__dmul_rn(0.5, __dadd_rn(1.0, c)));
    const double sh = __dsqrt_rn(__dmul_rn(0.5, __dsub_rn(1.0, c)));
    __syncwarp();   // every lane is done with the previous pair's edges
    // passing edge k: x < 0 enters rp bin np - 1 - k (k < np), x >= 0 bin k - np + 1
    for (int k = lane; k < np; k += 32) {
      const double e = lya_edge((double)(k + 1), ch, p.binner_rp);   // |x| >= e: bin k + 1 or above
      s_band[ex + np - 1 - k] = -lya_below(e);
      s_band[ex + np + k] = e;
    }
    for (int k = lane; k < nt; k += 32) s_band[es + k] = lya_edge((double)(k + 1), sh, p.binner_rt);
    if (lane == 0) { s_band[ex + 2 * np] = INF; s_band[es + nt] = INF; }
    __syncwarp();
    // in range: x_lo <= x < x_hi, s < s_hi
    const double x_lo = s_band[ex], x_hi = s_band[ex + 2 * np - 1], s_hi = s_band[es + nt - 1];
    const double* __restrict__ D2 = p.dc + b;
    const double* __restrict__ W2 = p.w + b;
    const double* __restrict__ DW2 = p.dw + b;
    double gap = 0.0;   // largest step along f2
    for (int k = lane; k + 1 < L2; k += 32) gap = fmax(gap, D2[k + 1] - D2[k]);
    const bool one_edge = __all_sync(FULL, gap * ch * p.binner_rp < 0.999 && gap * sh * p.binner_rt < 0.999);
    for (int i0 = 0; i0 < L1; i0 += 64) {
      BandRow ra, rb;
      const int i = i0 + 2 * lane;
      // the rows' diagonals: first and last partner in range (x and s grow with j)
      int m_lo = INT_MAX, m_hi = INT_MIN, first_ss = 0, second_ss = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        BandRow& r = h ? rb : ra;
        const bool ok = i + h < L1;
        r.d = ok ? p.dc[a + i + h] : NaN;
        r.w = ok ? p.w[a + i + h] : 0.0;
        r.dw = ok ? p.dw[a + i + h] : 0.0;
        r.gdw = 0.0; r.gw = 0.0;
        if (ok) {
          int lo = 0, hi = L2;
          while (lo < hi) { const int k = (lo + hi) >> 1; if (__dsub_rn(D2[k], r.d) >= x_lo) hi = k; else lo = k + 1; }
          const int j0 = lo;
          hi = L2;
          while (lo < hi) {
            const int k = (lo + hi) >> 1;
            if (__dsub_rn(D2[k], r.d) >= x_hi || __dadd_rn(D2[k], r.d) >= s_hi) hi = k; else lo = k + 1;
          }
          if (lo > j0) {
            m_lo = min(m_lo, j0 - i);      // step m of row h has partner i + m
            m_hi = max(m_hi, lo - 1 - i);
          }
          r.kb = j0;                       // as pixels of f2 until m_lo is known
          r.kn = lo - j0;
        } else {
          r.kb = 0;
          r.kn = 0;
        }
      }
      m_lo = __reduce_min_sync(FULL, m_lo);
      m_hi = __reduce_max_sync(FULL, m_hi);
      if (m_lo > m_hi) continue;
      // bin states before the first step: as of the first partner there is
      const int steps = m_hi - m_lo + 1;
      bool single = one_edge && steps < 0xffff;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        BandRow& r = h ? rb : ra;
        const int j = max(0, i + m_lo);
        const double d2 = j < L2 ? D2[j] : NaN;
        const int sx = edges_passed(ex, 2 * np, __dsub_rn(d2, r.d));
        // the rt bin as of the first partner in range
        const int ss = r.kn > 0 ? edges_passed(es, nt, __dadd_rn(D2[r.kb], r.d)) : 0;
        r.ox = 8 * (ex + sx);
        r.oc = sx * nt16 + 16 * ss;
        r.ex = s_band[ex + sx];
        r.kt = r.kt2 = ~0u;
        int at = r.kb;   // the row's partners are at, at + 1, ... end - 1
        const int end = r.kb + r.kn;
        for (int q = 0; at < end; ++q) {   // steps of the rt edges the row passes
          const double e = s_band[es + ss + q];
          int hi = end;
          while (at < hi) { const int k = (at + hi) >> 1; if (__dadd_rn(D2[k], r.d) >= e) hi = k; else at = k + 1; }
          if (at == end) break;
          if (q == 4) { single = false; break; }
          unsigned& word = q < 2 ? r.kt : r.kt2;
          word = (word & ~(0xffffu << 16 * (q & 1))) | (unsigned)(at - i - m_lo) << 16 * (q & 1);
        }
        if (h) second_ss = ss; else first_ss = ss;
        r.kb -= i + m_lo;
      }
      single = __all_sync(FULL, single);
      if (!single) { ra.kt = first_ss; rb.kt = second_ss; }
      // pixels jb .. jb + 31 of f2 into the ring (pixels outside the forest: NaN, no weight)
      const int j00 = i0 + m_lo;      // lane 0's partner at step 0
      auto stage = [&](int k0) {
        const int j = j00 + k0 + lane, q = (k0 + lane) & (BAND_RING - 1);
        const bool ok = j >= 0 && j < L2;
        s_band[ring + BAND_D + (q & 1) * (BAND_RING / 2) + (q >> 1)] = ok ? D2[j] : NaN;
        *reinterpret_cast<double2*>(&s_band[ring + (q & 1) * BAND_RING + 2 * (q >> 1)]) =
            ok ? make_double2(W2[j], DW2[j]) : make_double2(0.0, 0.0);
      };
      __syncwarp();
      stage(0);
      stage(32);
      BandCols col = {0.0, 0.0, 0.0, 0.0};
      for (int k0 = 0; k0 < steps; k0 += 32) {
        stage(k0 + 64);
        __syncwarp();
        const int n = min(32, steps - k0);
        if (single) band_walk<true>(ra, rb, col, ring, k0, n, nt16, es);
        else band_walk<false>(ra, rb, col, ring, k0, n, nt16, es);
        __syncwarp();
        const int j = j00 + k0 + lane;
        if (lane < ((n + 1) & ~1) && j >= 0 && j < L2) {
          const double2 g = *reinterpret_cast<const double2*>(&s_band[ring + BAND_OUT + 2 * lane]);
          if (g.x != 0.0) atomicAdd(&p.g_dw[b + j], g.x);
          if (g.y != 0.0) atomicAdd(&p.g_w[b + j], g.y);
        }
        __syncwarp();
      }
      // the f2 pixels still in the lanes, and the rows
      const int js = j00 + ((steps + 1) & ~1) + 2 * lane;
      if (js >= 0 && js < L2) {
        if (col.pdw != 0.0) atomicAdd(&p.g_dw[b + js], col.pdw);
        if (col.pw != 0.0) atomicAdd(&p.g_w[b + js], col.pw);
      }
      if (js + 1 >= 0 && js + 1 < L2) {
        if (col.qdw != 0.0) atomicAdd(&p.g_dw[b + js + 1], col.qdw);
        if (col.qw != 0.0) atomicAdd(&p.g_w[b + js + 1], col.qw);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const BandRow& r = h ? rb : ra;
        if (i + h < L1) {
          if (r.gdw != 0.0) atomicAdd(&p.g_dw[a + i + h], r.gdw);
          if (r.gw != 0.0) atomicAdd(&p.g_w[a + i + h], r.gw);
        }
      }
    }
  }
}

__global__ void k_unpad(int64_t n, const int64_t* __restrict__ start, const int64_t* __restrict__ pstart,
                        const double* __restrict__ src, double* __restrict__ dst) {
  for (int64_t f = blockIdx.x; f < n; f += gridDim.x) {
    const int64_t s = start[f], L = start[f + 1] - s, d = pstart[f];
    for (int64_t k = threadIdx.x; k < L; k += blockDim.x) dst[s + k] = src[d + k];
  }
}

}  // namespace

// Whether the band kernel takes the lean pairs.  Its table has to leave shared
// memory for 8 warps or more (50 x 50 bins: 81 KB, 24 warps of 4.8 KB); and it has
// to pay, by the catalogue's mean length and pixel step.  Times of the band and
// of the gather kernel:
// * a pair costs the band its np + nt edges and full passes of 64 rows whatever its
//   length: 32 pixels, 50 x 50 bins 1.45 / 1.38 ms, 36 pixels 1.34 / 1.43; 200 x 12
//   bins, 100 pixels 3.16 / 2.99, 150 pixels 5.67 / 6.24; 10 x 300 bins, 80 pixels
//   1.76 / 1.61, 150 pixels 4.39 / 4.74; above 3,584 bins only three CTAs of the
//   gather kernel fit an SM, and the band pays sooner: 64 x 64 bins, 20 pixels
//   2.29 / 2.38, 32 pixels 1.70 / 2.32;
// * a row passes its rp edges one by one: 1,000 forests of 375 pixels, 200 x 12
//   bins (two edges a step) 32.7 / 38.1 ms, 250 x 10 38.9 / 33.3, 600 x 4 80 / 37;
//   and rt bins in narrower rows than its four known steps: 8 x 500 44.7 / 46.6,
//   4 x 600 35.3 / 33.2;
// * with masked stretches (three per forest) the rows' edges have to be met in
//   loops, and the other lanes wait: 45 x 45 bins 25.6 / 26.0 ms, 55 x 55 27.3 /
//   26.4, 100 x 25 30.4 / 26.1, 10 x 300 28.6 / 26.4; above 3,584 bins 64 x 64
//   33.8 / 39.8, 100 x 40 37.5 / 47.5, 200 x 20 63 / 46.
static bool band_takes_lean(int np, int nt, int warps, double binner_rp, const CatalogSteps& st) {
  if (warps < 8) return false;
  const bool many = np * nt > 3584;   // gather: three CTAs per SM
  if (st.len < (many ? 20.0 : 36.0) + 0.7 * std::max(0, np - 90) + 0.65 * std::max(0, nt - 190)) return false;
  const double edges = st.step * binner_rp;   // rp edges a step
  if (st.masked < 0.5) return edges <= 2.1 && nt <= 500;
  return edges <= (many ? 1.7 : 0.5) && nt <= 200;
}

// Scratch of the adjoint, kept in the context between calls (grown, never shrunk).
static cudaError_t adjoint_reserve(lya_ctx* ctx, int nb, int64_t n, int64_t npad, int64_t npix) {
  AdjScratch& S = ctx->adj;
  if (S.g && S.nb >= nb && S.n >= n && S.npad >= npad && S.npix >= npix) return cudaSuccess;
  lya_free(S.g); lya_free(S.coef); lya_free(S.gdw); lya_free(S.gw); lya_free(S.out); lya_free(S.start);
  S = AdjScratch{};
  cudaError_t e = lya_alloc(&S.g, nb);
  if (e == cudaSuccess) e = lya_alloc(&S.coef, 2 * (size_t)nb);
  if (e == cudaSuccess) e = lya_alloc(&S.gdw, npad);
  if (e == cudaSuccess) e = lya_alloc(&S.gw, npad);
  if (e == cudaSuccess) e = lya_alloc(&S.out, npix);
  if (e == cudaSuccess) e = lya_alloc(&S.start, n + 1);
  if (e != cudaSuccess) {
    lya_free(S.g); lya_free(S.coef); lya_free(S.gdw); lya_free(S.gw); lya_free(S.out); lya_free(S.start);
    S = AdjScratch{};
    return e;
  }
  S.nb = nb; S.n = n; S.npad = npad; S.npix = npix;
  return cudaSuccess;
}

int lya_adjoint_launch(lya_ctx* ctx, const double* g, double* grad_dw, double* grad_w, int device_ptrs) {
  const int nb = ctx->np * ctx->nt;
  const int64_t n = ctx->cat.n;
  const int64_t npad = ctx->cat.npad, npix = ctx->cat.npix;
  cudaStream_t s = ctx->stream;
  cudaError_t e = adjoint_reserve(ctx, nb, n, npad, npix);
  if (e != cudaSuccess) return lya_fail(ctx, LYA_ERR_ALLOC, "lya_corr_adjoint: allocation failed");
  CatalogSteps steps;
  e = lya_catalog_steps(ctx, &steps);
  if (e != cudaSuccess) return lya_fail(ctx, LYA_ERR_CUDA, "lya_corr_adjoint: %s", cudaGetErrorString(e));
  AdjScratch& S = ctx->adj;
  double *d_g = S.g, *coef = S.coef, *gdw = S.gdw, *gw = S.gw, *out = S.out;
  int64_t* d_start = S.start;
  e = cudaMemcpyAsync(d_g, g, sizeof(double) * nb, (device_ptrs & 2) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice,
                      s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_start, ctx->h_start.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(gdw, 0, sizeof(double) * npad, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(gw, 0, sizeof(double) * npad, s);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev0, s);
  if (e == cudaSuccess) {
    k_coef<<<(nb + 255) / 256, 256, 0, s>>>(ctx->hist_slots, nb, ctx->hist, d_g, coef);
    ctx->launches++;
    AdjParams p;
    p.dc = ctx->cat.dc; p.w = ctx->cat.w; p.dw = ctx->cat.dw; p.pstart = ctx->cat.pstart; p.len = ctx->cat.len;
    p.sorted = ctx->cat.sorted; p.ux = ctx->cat.ux; p.uy = ctx->cat.uy; p.uz = ctx->cat.uz;
    p.f1 = ctx->wq.f1; p.f2 = ctx->wq.f2; p.n_items = ctx->wq.n_pairs;
    p.binner_rp = (double)ctx->np / ctx->rpmax; p.binner_rt = (double)ctx->nt / ctx->rtmax;
    p.np = ctx->np; p.nt = ctx->nt; p.nb = nb; p.cos_variant = ctx->cos_variant;
    p.coef = coef; p.g_dw = gdw; p.g_w = gw;
    // the band kernel, and the gather kernel for the pairs it leaves
    const size_t smem = sizeof(double) * 2 * nb, smem_max = 226 * 1024;
    const size_t table = sizeof(double) * (size_t)band_table(ctx->np, ctx->nt);
    const size_t per_warp = sizeof(double) * (size_t)band_per_warp(ctx->np, ctx->nt);
    const int warps = table < smem_max ? (int)std::min<size_t>(BAND_WARPS, (smem_max - table) / per_warp) : 0;
    const bool band = band_takes_lean(ctx->np, ctx->nt, warps, p.binner_rp, steps);
    p.skip_lean = band ? 1 : 0;
    if (band && p.n_items > 0) {
      const size_t smem_band = table + warps * per_warp;
      e = cudaFuncSetAttribute(k_adjoint_band, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_band);
      if (e == cudaSuccess) {
        k_adjoint_band<<<ctx->num_sms, warps * 32, smem_band, s>>>(p);
        ctx->launches++;
      }
    }
    if (p.n_items > 0 && (!band || ctx->cat.n_not_lean > 0)) {
      if (e == cudaSuccess) e = cudaFuncSetAttribute(k_adjoint, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e == cudaSuccess) {
        k_adjoint<<<ctx->num_sms * 4, 256, smem, s>>>(p);
        ctx->launches++;
      }
    }
    if (e == cudaSuccess) e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev1, s);
  if (e == cudaSuccess && n > 0) {
    const int blocks = (int)std::min<int64_t>(n, (int64_t)ctx->num_sms * 16);
    if (device_ptrs & 1) {
      if (grad_dw) { k_unpad<<<blocks, 128, 0, s>>>(n, d_start, ctx->cat.pstart, gdw, grad_dw); ctx->launches++; }
      if (grad_w) { k_unpad<<<blocks, 128, 0, s>>>(n, d_start, ctx->cat.pstart, gw, grad_w); ctx->launches++; }
    } else {
      k_unpad<<<blocks, 128, 0, s>>>(n, d_start, ctx->cat.pstart, gdw, out);
      ctx->launches++;
      e = lya_touch_pages(grad_dw, sizeof(double) * npix);   // beside the kernels
      if (e == cudaSuccess) e = lya_touch_pages(grad_w, sizeof(double) * npix);
      if (e == cudaSuccess && grad_dw) e = cudaMemcpyAsync(grad_dw, out, sizeof(double) * npix, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      k_unpad<<<blocks, 128, 0, s>>>(n, d_start, ctx->cat.pstart, gw, out);
      ctx->launches++;
      if (e == cudaSuccess && grad_w) e = cudaMemcpyAsync(grad_w, out, sizeof(double) * npix, cudaMemcpyDeviceToHost, s);
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  float ms = 0.f;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  if (e != cudaSuccess) return lya_fail(ctx, LYA_ERR_CUDA, "lya_corr_adjoint: %s", cudaGetErrorString(e));
  ctx->last.adjoint_ms = ms;
  return LYA_OK;
}

extern "C" int lya_corr_totals(lya_ctx* ctx, double* W, double* DW, int32_t device_ptrs) {
  if (!ctx) return lya_fail(nullptr, LYA_ERR_ARG, "lya_corr_totals: ctx is NULL");
  if (!W || !DW) return lya_fail(ctx, LYA_ERR_ARG, "lya_corr_totals: NULL output");
  if (!ctx->have_result) return lya_fail(ctx, LYA_ERR_STATE, "lya_corr_totals: run lya_corr_run first");
  LYA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  const int nb = ctx->np * ctx->nt;
  cudaStream_t s = ctx->stream;
  if (device_ptrs) {
    k_totals<<<(nb + 255) / 256, 256, 0, s>>>(ctx->hist_slots, nb, ctx->hist, W, DW);
    ctx->launches++;
    LYA_CHECK_CUDA(ctx, cudaGetLastError());
    LYA_CHECK_CUDA(ctx, cudaStreamSynchronize(s));
    return LYA_OK;
  }
  cudaError_t e = adjoint_reserve(ctx, nb, ctx->cat.n, ctx->cat.npad, ctx->cat.npix);
  if (e != cudaSuccess) return lya_fail(ctx, LYA_ERR_ALLOC, "lya_corr_totals: allocation failed");
  double* t = ctx->adj.coef;   // [2][nb]
  k_totals<<<(nb + 255) / 256, 256, 0, s>>>(ctx->hist_slots, nb, ctx->hist, t, t + nb);
  ctx->launches++;
  LYA_CHECK_CUDA(ctx, cudaGetLastError());
  LYA_CHECK_CUDA(ctx, cudaMemcpyAsync(W, t, sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
  LYA_CHECK_CUDA(ctx, cudaMemcpyAsync(DW, t + nb, sizeof(double) * nb, cudaMemcpyDeviceToHost, s));
  LYA_CHECK_CUDA(ctx, cudaStreamSynchronize(s));
  return LYA_OK;
}

extern "C" int lya_corr_adjoint(lya_ctx* ctx, const double* g, double* grad_dw, double* grad_w, int32_t device_ptrs) {
  if (!ctx) return lya_fail(nullptr, LYA_ERR_ARG, "lya_corr_adjoint: ctx is NULL");
  if (!g) return lya_fail(ctx, LYA_ERR_ARG, "lya_corr_adjoint: g is NULL");
  if (!ctx->have_result) return lya_fail(ctx, LYA_ERR_STATE, "lya_corr_adjoint: run lya_corr_run first");
  LYA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  return lya_adjoint_launch(ctx, g, grad_dw, grad_w, device_ptrs);
}
