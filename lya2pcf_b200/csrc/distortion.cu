// Distortion-matrix numerator of the lya2pcf B200 library.
//
// Reference: distortion_per_pixel (distortion_procedures_pycuda.py:195-279)
// with the kernels precompute_distances, compute_etas, order_active and
// compute_d (cuda_kernels.cpp:46-87, 165-278).  For a forest pair (f1, f2)
// and pixel pairs (i, j) in bin A, (k, l) in bin B, with
//   eta1_ik = delta_ik - w_k/Om1 - dl_i w_k dl_k / O1,   O = sum w dl^2,
// the reference scatters, per in-range pair and per active bin B,
//   D_AB += w_i w_j sum_{(k,l) in B} eta1_ik eta2_jl.
//
// This kernel evaluates the same sum in factored form.  With per-pixel columns
//   S2[A,i] = sum_{j:(i,j) in A} w_j,   L2[A,i] = sum_{j:(i,j) in A} w_j dl_j
//   S1[A,j] = sum_{i:(i,j) in A} w_i,   L1[A,j] = sum_{i:(i,j) in A} w_i dl_i
// and per-bin moments M0_A = sum w_i w_j, Mi_A = sum w_i dl_i w_j,
// Mj_A = sum w_i w_j dl_j, Mij_A = sum w_i dl_i w_j dl_j (over (i,j) in A):
//   D_AB = [A==B] M0_A
//        + M0_A M0_B/(Om1 Om2) + Mj_A Mj_B/(Om1 O2) + Mi_A Mi_B/(O1 Om2) + Mij_A Mij_B/(O1 O2)
//        - sum_i w_i (S2[A,i] S2[B,i]/Om2 + L2[A,i] L2[B,i]/O2)
//        - sum_j w_j (S1[A,j] S1[B,j]/Om1 + L1[A,j] L1[B,j]/O1)
// (expand eta1_ik eta2_jl; the delta terms give the diagonal, the products of
// the two projections the rank-4 part, the cross terms the columns).  The
// column of a pixel spans a few rt bins only, so the column products are
// 50x50 dense blocks (rp x rp) per pair of rt bins.
//
// One CTA per forest pair (dynamic queue).  Bins are those of the reference FP64
// formula.  Phase 1: the columns of every pixel go to CTA-private global scratch
// as dense [TS rt bins][np] rows, from exact bin edges for pairs of long lean
// forests (build_columns, lanes over the bins), otherwise from the bin of every
// pixel pair (a warp per pixel, lanes over its partners).  Phase 2: the 50x50
// (rp x rp) blocks (t, u) of D over the pair's window of rt bins, diagonal blocks
// first (they complete the moments of bin t, read from the same staged rows: the
// f1 weights placed in padding columns NS..NS+3 of the staged rows make
// accumulator columns NS..NS+3 of the diagonal block's MMAs the four moments, when
// NS + 4 <= 64; otherwise a loop over the staged rows; a diagonal block is
// symmetric, so only the tiles that reach its upper triangle are multiplied).  A
// block whose rt bins are both spanned by some pixel column gets the column
// products as a small dense FP64 GEMM on the tensor cores: the rows of the pixels
// covering t and u are staged in shared memory in chunks of CH pixels, and each
// warp accumulates 16 x 8 tiles of the block (four tiles of 16 rp bins down, 8
// across; mma.sync m16n8k8 f64, FP64 having no tcgen05 kind; rows at or beyond np
// enter as zeros); the rank-4 and diagonal terms are added to the accumulators,
// and each D entry of the window gets one atomic add per forest pair (both (A, B)
// and (B, A): D is symmetric).
// A forest whose sum w dl^2 is 0 has no slope to project out: its slope terms
// are 0.
#include <cuda_pipeline.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "lya_internal.cuh"

namespace {

constexpr int TS = 8;         // rt bins a pixel column may span
constexpr int TSB = TS + 2;   // rows of a column being built (its window may be one bin wider at each end)
constexpr int NP_MAX = 64;    // np of the blocks: at most 4 x 8 tiles of 16 x 8
// Launch shapes the autotuner chooses from: threads per CTA (DT) and pixels per
// staged chunk of a block (CH, a multiple of 8: the K of one MMA).  Shape 0 is the default.
struct DistShape { int dt, ch; };
constexpr DistShape DIST_SHAPES[] = {{512, 32}, {512, 16}, {512, 24}, {256, 32}, {256, 16}};
constexpr int N_DIST_SHAPES = sizeof(DIST_SHAPES) / sizeof(DIST_SHAPES[0]);
// Staged row length for np bins: 8 * ceil(np/8) plus 4, so the four rows of an
// MMA fragment load fall in disjoint shared-memory banks.
__host__ __device__ __forceinline__ int stage_npad(int np) { return 8 * ((np + 7) / 8) + 4; }
// Row stride of the column scratch: np rounded up to even, so every row starts
// on a 16-byte boundary (the asynchronous 16-byte copies of the staging).
__host__ __device__ __forceinline__ int col_stride(int np) { return (np + 1) & ~1; }
// Shared-memory doubles of the staging area: two buffers of four [CH][NPAD]
// row sets (double buffering), or the per-warp column builders of phase 1.
__host__ __device__ __forceinline__ int stage_doubles(int CH, int NW, int np) {
  const int a = 2 * 4 * CH * stage_npad(np), b = NW * 2 * (TS + 2) * np;
  return a > b ? a : b;
}

struct DistParams {
  const double4* __restrict__ pix8;   // (dc, w, dw, z)
  const double* __restrict__ dl;
  const int64_t* __restrict__ pstart;
  const int32_t* __restrict__ len;
  const uint8_t* __restrict__ sorted;
  const double* __restrict__ ux;
  const double* __restrict__ uy;
  const double* __restrict__ uz;
  const double* __restrict__ omega;
  const double* __restrict__ odl2;
  const int32_t* __restrict__ f1;
  const int32_t* __restrict__ f2;
  const long long* n_items;   // [1] forest pairs of the queue (device: the captured graph serves any count)
  int max_len;
  double binner_rp, binner_rt;
  int np, nt, nb, cos_variant;
  int npad;                // staged row length (stage_npad(np))
  double* col;             // scratch [grid][2 sides][max_len][TS][col_stride(np)] x {S, L}
  double* moments;         // scratch [grid][4][nt][np]: moments of the window's bins
  double* D;               // [nb][nb]
  double* W;               // [nb]
  unsigned long long* err; // [1] pixels whose column spans more than TS rt bins
  unsigned long long* next;// [1] work queue counter
  // [1] block-product work in m8n8k4 units, for the roofline: 8x8 tiles of a block (of a diagonal block, the
  // tiles that are multiplied for its upper triangle and the moments), pixels rounded to 4
  unsigned long long* mma;
  int shape;               // launch shape (DIST_SHAPES index); part of the captured graph's key
};

// Bin of a pixel pair with the reference FP64 formula, as (bp, bt); false when
// out of range.
__device__ __forceinline__ bool pair_bin2(double d1, double d2, double ch, double sh, const DistParams& p, int& bp,
                                          int& bt) {
  const double rp = __dmul_rn(fabs(__dsub_rn(d1, d2)), ch);
  const double rt = __dmul_rn(__dadd_rn(d1, d2), sh);
  const double fp = floor(__dmul_rn(rp, p.binner_rp));
  const double ft = floor(__dmul_rn(rt, p.binner_rt));
  if (!(fp >= 0.0 && fp < (double)p.np && ft >= 0.0 && ft < (double)p.nt)) return false;
  bp = (int)fp;
  bt = (int)ft;
  return true;
}

// rt bin coordinate floor(rt * nt / rtmax) of a pixel pair (reference formula, unclamped)
__device__ __forceinline__ double pair_ft(double d1, double d2, double sh, const DistParams& p) {
  return floor(__dmul_rn(__dmul_rn(__dadd_rn(d1, d2), sh), p.binner_rt));
}

// First index in [lo, hi) of the sorted shared array a at which the monotone
// predicate holds (hi when it holds nowhere), found by the whole warp: 32
// probes and one vote per level, ceil(log32(hi - lo)) + 1 levels instead of
// log2(hi - lo) dependent steps of a binary search.
template <class Pred>
__device__ __forceinline__ int warp_first(const double* a, int lo, int hi, Pred pred) {
  const int lane = threadIdx.x & 31;
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) >> 5;
    const int idx = lo + (lane + 1) * step - 1;
    const bool t = lane == 31 || idx >= hi || pred(a[idx]);   // the last lane closes the range
    const unsigned bal = __ballot_sync(0xffffffffu, t);
    const int f = __ffs(bal) - 1;
    const int pf = lo + (f + 1) * step - 1;     // lane f's probe (true, or the closing lane)
    const int nhi = (f == 31 || pf >= hi) ? hi : pf;
    lo += f * step;                             // lane f-1's probe was false
    hi = nhi;
  }
  const int idx = lo + lane;
  const unsigned bal = __ballot_sync(0xffffffffu, idx < hi && pred(a[idx]));
  return bal ? lo + __ffs(bal) - 1 : hi;
}

// Whether a pair of lean forests takes its columns from edges (build_columns).
// That costs a pixel about the same whatever its partners are, and twice with
// more than 32 rp bins (two bins per lane); the general builder's cost grows with
// the partners, of which a pixel has at most the other forest's length: the line
// is drawn at the lengths' harmonic mean.  Kernel, edges against general builder,
// 120,000 pairs of equal forests: 50 x 50 bins, 80 pixels 31.9 against 27.7 ms,
// 150 pixels 70.3 against 69.0, 200 pixels 108.3 against 110.6; 16 x 16 bins, 60
// pixels 27.1 against 26.3, 80 pixels 20.9 against 21.7, 200 pixels 52.9 against 69.3.
__device__ __forceinline__ bool columns_from_edges(int L1, int L2, int np) {
  return 2 * L1 * L2 >= (np > 32 ? 175 : 75) * (L1 + L2);   // lengths below 2^15: shared memory
}

// Columns of the pixels m0 .. m1-1 of one side for a pair of lean forests, by
// one warp: lane b holds rp bins b and b + 32 of every column and rt edges b and
// b + 32.  The partners of an rp bin are two index ranges (below and above the
// pixel's distance) and those of an rt bin one, all bounded by exact edges
// (lya_edge: ex[b] of rp bin b + 1, es[b] of rt bin b + 1).  From pixel to pixel
// the bounds move by about one partner, so they are kept and moved by up to
// three partners at a time (independent loads, no search).  A row of a column
// (one rt bin) is the sum over the few partners of the lane's two ranges that
// fall in it, stored to the scratch as it is formed: no bin of a pixel pair is
// computed, nothing is zeroed, and there are no atomics.  72,415 forest pairs
// (600 clustered forests): the kernel takes 154 ms, 174 ms with a bin per pixel
// pair and rows built by shared atomics.  Bound: issue, about 1,000
// warp-instructions per pixel; loading three partners at a time instead of the
// next one only, or the partners of even and odd index apart, is not faster
// (156-159 ms).  Up to 64 rt edges fit the lanes; a binning with more takes the
// builder of the other pairs.
// tlo, span: the columns' rows; T0, T1, smax: the warp's rt bins and widest column.
__device__ __forceinline__ void build_columns(const DistParams& p, const double* dm, const double* dO, const double* wO,
                                              const double* lO, int Lo, int m0, int m1, const double* ex,
                                              const double* es, int* tlo, int* span, double* cS, double* cL, int NS,
                                              int& T0, int& T1, int& smax) {
  constexpr unsigned FULL = 0xffffffffu;
  const double INF = __longlong_as_double(0x7ff0000000000000ll);
  const int lane = threadIdx.x & 31, np = p.np, nt = p.nt;
  const bool two = np > 32;
  // first partner with x >= e_lo (x > -ex), with x >= e_hi, with s >= e_t
  double e_lo[2], e_hi[2], e_t[2];
  int l1[2], r1[2], jt[2];
  if (m0 >= m1) return;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int b = lane + 32 * h;
    e_lo[h] = b < np ? -lya_below(ex[b]) : -INF;
    e_hi[h] = b < np ? ex[b] : -INF;
    e_t[h] = b < nt ? es[b] : INF;
    const double d = dm[m0];
    auto first = [&](auto at_or_above) {
      int lo = 0, hi = Lo;
      while (lo < hi) { const int k = (lo + hi) >> 1; if (at_or_above(dO[k])) hi = k; else lo = k + 1; }
      return lo;
    };
    l1[h] = first([&](double v) { return __dsub_rn(v, d) >= e_lo[h]; });
    r1[h] = first([&](double v) { return __dsub_rn(v, d) >= e_hi[h]; });
    jt[h] = first([&](double v) { return __dadd_rn(v, d) >= e_t[h]; });
  }
  for (int m = m0; m < m1; ++m) {
    const double d = dm[m];
    for (bool more = m > m0; more;) {   // the bounds of this pixel from the previous one's
      bool far = false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        int cl = 0, cr = 0, ct = 0;
#pragma unroll
        for (int u = 0; u < 3; ++u) {
          const int kl = l1[h] + u, kr = r1[h] + u, kt = jt[h] - 1 - u;
          cl += kl < Lo && __dsub_rn(dO[min(kl, Lo - 1)], d) < e_lo[h];
          cr += kr < Lo && __dsub_rn(dO[min(kr, Lo - 1)], d) < e_hi[h];
          ct += kt >= 0 && __dadd_rn(dO[max(kt, 0)], d) >= e_t[h];
        }
        l1[h] += cl; r1[h] += cr; jt[h] -= ct;
        far = far || cl == 3 || cr == 3 || ct == 3;
      }
      more = __any_sync(FULL, far);
    }
    // partners [jb, je): within rpmax and rtmax; their rt bins lo .. lo + sp - 1
    const int hb = (np - 1) >> 5, ht = (nt - 1) >> 5;
    const int jb = __shfl_sync(FULL, hb ? l1[1] : l1[0], (np - 1) & 31);
    const int je = min(__shfl_sync(FULL, hb ? r1[1] : r1[0], (np - 1) & 31),
                       __shfl_sync(FULL, ht ? jt[1] : jt[0], (nt - 1) & 31));
    const int lo = __popc(__ballot_sync(FULL, jt[0] <= jb && lane < nt)) +
                   __popc(__ballot_sync(FULL, jt[1] <= jb && lane + 32 < nt));
    const int hi = __popc(__ballot_sync(FULL, jt[0] < je && lane < nt)) +
                   __popc(__ballot_sync(FULL, jt[1] < je && lane + 32 < nt));
    int sp = jb < je ? hi - lo + 1 : 0;
    if (sp > TS) {
      if (lane == 0) atomicAdd(p.err, 1ull);
      sp = 0;
    }
    if (lane == 0) { tlo[m] = lo; span[m] = sp; }
    if (sp > 0) { T0 = min(T0, lo); T1 = max(T1, lo + sp - 1); smax = max(smax, sp); }
    // the lane's ranges [l1, l0) and [r0, r1): bin b - 1 ends where bin b begins
    int l0[2], r0[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      l0[h] = __shfl_up_sync(FULL, l1[h], 1);
      r0[h] = __shfl_up_sync(FULL, r1[h], 1);
    }
    const int l31 = __shfl_sync(FULL, l1[0], 31), r31 = __shfl_sync(FULL, r1[0], 31);
    if (lane == 0) {
      l0[0] = r0[0] = min(l1[0] + 3, r1[0]);   // bin 0: one range
      l0[1] = l31; r0[1] = r31;
    }
    double* rs = cS + (size_t)m * TS * NS;
    double* rl = cL + (size_t)m * TS * NS;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 1 && !two) break;
      const int b = lane + 32 * h;
      const int el = b < np ? min(l0[h], je) : 0, er = b < np ? min(r1[h], je) : 0;
      if (__all_sync(FULL, el - l1[h] <= 3 && er - r0[h] <= 3)) {
        double w[6], l[6];
        int row[6];
#pragma unroll
        for (int u = 0; u < 6; ++u) {
          const int j = u < 3 ? l1[h] + u : r0[h] + u - 3;
          const bool in = j < (u < 3 ? el : er);
          w[u] = in ? wO[j] : 0.0;
          l[u] = in ? lO[j] : 0.0;
          row[u] = in ? 0 : TS;
        }
        for (int q = 0; q + 1 < sp; ++q) {
          const int e = lo + q, jn = __shfl_sync(FULL, e < 32 ? jt[0] : jt[1], e & 31);   // row q ends at jn
#pragma unroll
          for (int u = 0; u < 6; ++u) row[u] += (u < 3 ? l1[h] + u : r0[h] + u - 3) >= jn;
        }
        for (int q = 0; q < sp; ++q) {
          double as = 0.0, al = 0.0;
#pragma unroll
          for (int u = 0; u < 6; ++u) {
            if (row[u] == q) { as += w[u]; al = fma(w[u], l[u], al); }
          }
          if (b < NS) { rs[q * NS + b] = as; rl[q * NS + b] = al; }
        }
      } else {   // more than three partners in a range
        int ja = jb;
        for (int q = 0; q < sp; ++q) {
          const int e = lo + q, jn = q + 1 < sp ? __shfl_sync(FULL, e < 32 ? jt[0] : jt[1], e & 31) : je;
          double as = 0.0, al = 0.0;
          for (int j = max(ja, l1[h]); j < min(jn, el); ++j) { as += wO[j]; al = fma(wO[j], lO[j], al); }
          for (int j = max(ja, r0[h]); j < min(jn, er); ++j) { as += wO[j]; al = fma(wO[j], lO[j], al); }
          if (b < NS) { rs[q * NS + b] = as; rl[q * NS + b] = al; }
          ja = jn;
        }
      }
    }
  }
}

template <int DT, int CH>
__global__ void __launch_bounds__(DT, 1) k_dist(const DistParams p) {
  constexpr int NW = DT / 32;   // warps per CTA
  // 16 x 8 accumulator tiles per warp: NW/4 warps share each of the four tile
  // rows of 16 rp bins (np <= 64), and split its (at most 8) tile columns
  constexpr int CC = NW >= 16 ? 2 : 4;
  extern __shared__ __align__(16) unsigned char smem[];
  const int ML = p.max_len;
  const int np = p.np, nt = p.nt, nb = p.nb, NPAD = p.npad;
  double* sd = reinterpret_cast<double*>(smem);          // [2][ML] dc
  double* sw = sd + 2 * ML;                              // [2][ML] w
  double* sl = sw + 2 * ML;                              // [2][ML] dl
  double* mom = p.moments + (size_t)blockIdx.x * 4 * nt * np;   // [4][nt][np] (CTA-private, L2-resident)
  double* stage = sl + 2 * ML;                           // 2 x [4][CH][NPAD] staged rows, or the column builders
  const int stage_len = stage_doubles(CH, NW, np);
  double* kbuf = stage + stage_len;                      // [2][4][CH] per staged row: k_S, k_L, f1 w, f1 w dl
  int* tlo = reinterpret_cast<int*>(kbuf + 8 * CH);      // [2][ML]
  int* span = tlo + 2 * ML;                              // [2][ML]
  // [2][2*ML] scratch rows of bin t of the pixels of this block and of the next:
  // (side * ML + pixel) * TS + t - tlo
  int* rows_of = span + 2 * ML;
  __shared__ int s_T0, s_T1, s_maxspan, s_cnt[3];
  __shared__ long long s_item;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NS = col_stride(np);
  // staging: this thread copies 16-byte segment cp_seg of rows cp_row, cp_row + cp_step, ...
  const int cp_seg = tid % (NS / 2), cp_step = DT / (NS / 2);
  const int cp_row = tid / (NS / 2) < cp_step ? tid / (NS / 2) : INT_MAX;
  double* colS = p.col + (size_t)blockIdx.x * 2 * 2 * ML * TS * NS;   // [2 sides][ML][TS][NS]
  double* colL = colS + (size_t)2 * ML * TS * NS;
  double* myS = stage + (size_t)warp * 2 * TSB * np;
  double* myL = myS + TSB * np;
  const int ntile = (np + 7) / 8;   // tile rows = tile columns of a 50x50 block (7 for np = 50)
  // warp w: tile row mt = w mod 4 (rp bins 16 mt .. 16 mt + 15) and tile
  // columns ng, ng + nwm, ... (ng = w / 4) of 8 rp bins each
  const int nwm = NW / 4;
  const int mt = warp & 3, ng = warp >> 2;
  const int grp = lane >> 2, kq = lane & 3;
  // Tiles of a diagonal block, which is symmetric: tile rows r and tile columns
  // c >= 2r only, dealt to the warps in turn (16 tiles for 50 rp bins, one per
  // warp, four per SM sub-partition); its columns NS .. NS+3 are the moments.
  const bool moments_in_tiles = NS + 4 <= 64;
  int sym_row[CC], sym_col[CC], sym_tiles = 0;   // sym_tiles: as 8x8 tiles
#pragma unroll
  for (int c = 0; c < CC; ++c) {
    int x = warp + NW * c, r = 0;
    const int ncol = (NS + 4 + 7) / 8, nrow = (np + 15) / 16;
    while (r < nrow && x >= ncol - 2 * r) { x -= ncol - 2 * r; ++r; }
    sym_row[c] = r < nrow ? r : -1;
    sym_col[c] = 2 * r + x;
  }
  for (int r = 0; 16 * r < np; ++r) sym_tiles += ((NS + 4 + 7) / 8 - 2 * r) * min(2, ntile - 2 * r);
  unsigned long long n_mma = 0;     // thread 0: MMAs of this CTA

  for (;;) {
    if (tid == 0) s_item = (long long)atomicAdd(p.next, 1ull);
    __syncthreads();
    const long long t_item = s_item;
    if (t_item >= *p.n_items) break;
    const int a = p.f1[t_item], b = p.f2[t_item];
    const int L1 = p.len[a], L2 = p.len[b];
    if (L1 <= 0 || L2 <= 0) { __syncthreads(); continue; }
    double c = lya_cos12(p.ux[a], p.uy[a], p.uz[a], p.ux[b], p.uy[b], p.uz[b], p.cos_variant);
    c = fmin(1.0, fmax(-1.0, c));
    const double ch = __dsqrt_rn(__dmul_rn(0.5, __dadd_rn(1.0, c)));
    const double sh = __dsqrt_rn(__dmul_rn(0.5, __dsub_rn(1.0, c)));
    const double om1 = p.omega[a], om2 = p.omega[b];
    const double odl2b = p.odl2[b];
    const double io1 = p.odl2[a] > 0.0 ? 1.0 / p.odl2[a] : 0.0;
    const double io2 = p.odl2[b] > 0.0 ? 1.0 / p.odl2[b] : 0.0;
    const bool srt = p.sorted[a] && p.sorted[b];
    const bool edges = nt <= 64 && (p.sorted[a] & p.sorted[b] & LYA_LEAN) && columns_from_edges(L1, L2, np);
    const int64_t A0 = p.pstart[a], B0 = p.pstart[b];
    const double kS1 = 1.0 / om2, kS2 = 1.0 / om1;
    for (int k = tid; k < L1; k += DT) {
      const double4 q = p.pix8[A0 + k];
      sd[k] = q.x; sw[k] = q.y; sl[k] = p.dl[A0 + k];
    }
    for (int k = tid; k < L2; k += DT) {
      const double4 q = p.pix8[B0 + k];
      sd[ML + k] = q.x; sw[ML + k] = q.y; sl[ML + k] = p.dl[B0 + k];
    }
    if (tid == 0) { s_T0 = INT_MAX; s_T1 = -1; s_maxspan = 0; }
    double* ex = stage;          // [np] exact rp edges (the builders' room is free then)
    double* es = stage + np;     // [nt] exact rt edges
    if (edges) {
      for (int k = tid; k < np; k += DT) ex[k] = lya_edge((double)(k + 1), ch, p.binner_rp);
      for (int k = tid; k < nt; k += DT) es[k] = lya_edge((double)(k + 1), sh, p.binner_rt);
    }
    __syncthreads();
    // ---- phase 1: columns.  From edges: each warp takes a contiguous share of
    // the pixels of either side (see build_columns)
    if (edges) {
      int T0 = INT_MAX, T1 = -1, smax = 0;
      for (int side = 0; side < 2; ++side) {
        const int Lm = side == 0 ? L1 : L2, Lo = side == 0 ? L2 : L1, share = (Lm + NW - 1) / NW;
        build_columns(p, sd + side * ML, sd + (1 - side) * ML, sw + (1 - side) * ML, sl + (1 - side) * ML, Lo,
                      min(Lm, warp * share), min(Lm, (warp + 1) * share), ex, es, tlo + side * ML, span + side * ML,
                      colS + (size_t)side * ML * TS * NS, colL + (size_t)side * ML * TS * NS, NS, T0, T1, smax);
      }
      if (lane == 0 && smax > 0) {
        atomicMin(&s_T0, T0);
        atomicMax(&s_T1, T1);
        atomicMax(&s_maxspan, smax);
      }
    }
    // The others: one warp per pixel: side 0 = f1 pixels (partners in
    // f2), side 1 = f2 pixels (partners in f1); built in shared memory with the
    // lanes over the partners, then stored to the CTA's scratch
    for (int side = 0; side < 2 && !edges; ++side) {
      const int Lm = side == 0 ? L1 : L2, Lo = side == 0 ? L2 : L1;
      const double* dm = sd + side * ML;
      const double* dO = sd + (1 - side) * ML;
      const double* wO = sw + (1 - side) * ML;
      const double* lO = sl + (1 - side) * ML;
      double* cS = colS + (size_t)side * ML * TS * NS;
      double* cL = colL + (size_t)side * ML * TS * NS;
      for (int m = warp; m < Lm; m += NW) {
        const double d = dm[m];
        int jlo = 0, jhi = Lo;
        if (srt) {   // partners with |d - d'| ch <= rpmax and (d + d') sh <= rtmax (+ margin)
          const double reach = ch > 0.0 ? ((double)np + 1e-3) / (ch * p.binner_rp) : 1e300;
          const double rt_reach = sh > 0.0 ? ((double)nt + 1e-3) / (sh * p.binner_rt) : 1e300;
          const double tl = d - reach - 1e-6 * fabs(d) - 1e-6;
          const double th = fmin(d + reach, rt_reach - d) + 1e-6 * fabs(d) + 1e-6;
          jlo = warp_first(dO, 0, Lo, [&](double v) { return v > tl; });
          jhi = warp_first(dO, jlo, Lo, [&](double v) { return !(v < th); });
        }
        // window of rt bins the column can touch, and the built rows
        int wlo = 0, nrow = 0;
        int lo = INT_MAX, hi = -1;
        if (srt) {
          // sorted: the rt bin is non-decreasing in the partner index, so the
          // partners at the two ends of the range bound the window; one pass,
          // each lane over a contiguous segment of partners, equal-bin runs
          // merged in registers before the shared-memory add
          if (jlo < jhi) {
            const double f0 = side == 0 ? pair_ft(d, dO[jlo], sh, p) : pair_ft(dO[jlo], d, sh, p);
            const double f1v = side == 0 ? pair_ft(d, dO[jhi - 1], sh, p) : pair_ft(dO[jhi - 1], d, sh, p);
            const double flo = fmax(f0, 0.0), fhi = fmin(f1v, (double)(nt - 1));
            if (flo <= fhi) {
              wlo = (int)flo;
              nrow = (int)fhi - wlo + 1;
            }
          }
          if (nrow > TSB) {
            if (lane == 0) atomicAdd(p.err, 1ull);
            nrow = 0;
          }
          if (nrow > 0) {
            if ((np & 1) == 0) {   // 16-byte stores (both builders start on 16 bytes for even np)
              double2* s2 = reinterpret_cast<double2*>(myS);
              double2* l2 = reinterpret_cast<double2*>(myL);
              for (int q = lane; q < nrow * np / 2; q += 32) { s2[q] = make_double2(0.0, 0.0); l2[q] = make_double2(0.0, 0.0); }
            } else {
              for (int q = lane; q < nrow * np; q += 32) { myS[q] = 0.0; myL[q] = 0.0; }
            }
            __syncwarp();
            const int cnt = jhi - jlo, seg = (cnt + 31) / 32;
            int j = jlo + lane * seg;
            const int je = min(jhi, j + seg);
            int cbp = -1, cbt = -1;
            double as = 0.0, al = 0.0;
            auto merge = [&](bool in, int bp, int bt, double wj, double lj) {
              if (!in) { bp = -1; bt = -1; }
              if (bp != cbp || bt != cbt) {
                if (cbp >= 0) {
                  const int q = (cbt - wlo) * np + cbp;
                  atomicAdd(&myS[q], as);
                  atomicAdd(&myL[q], al);
                }
                cbp = bp; cbt = bt; as = 0.0; al = 0.0;
              }
              if (in) {
                as += wj;
                al = fma(wj, lj, al);
                lo = min(lo, bt);
                hi = max(hi, bt);
              }
            };
            // bins of four partners at a time (independent FP64 chains), then
            // the runs in partner order
            for (; j + 4 <= je; j += 4) {
              int bp[4], bt[4];
              bool in[4];
              double wj[4], lj[4];
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const double dj = dO[j + u];
                wj[u] = wO[j + u];
                lj[u] = lO[j + u];
                in[u] = side == 0 ? pair_bin2(d, dj, ch, sh, p, bp[u], bt[u]) : pair_bin2(dj, d, ch, sh, p, bp[u], bt[u]);
              }
#pragma unroll
              for (int u = 0; u < 4; ++u) merge(in[u], bp[u], bt[u], wj[u], lj[u]);
            }
            for (; j < je; ++j) {
              int bp, bt;
              const bool in = side == 0 ? pair_bin2(d, dO[j], ch, sh, p, bp, bt) : pair_bin2(dO[j], d, ch, sh, p, bp, bt);
              merge(in, bp, bt, wO[j], lO[j]);
            }
            if (cbp >= 0) {
              const int q = (cbt - wlo) * np + cbp;
              atomicAdd(&myS[q], as);
              atomicAdd(&myL[q], al);
            }
          }
          for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
          }
        } else {
          // unsorted: a first pass finds the rt bins the column touches
          for (int o = jlo + lane; o < jhi; o += 32) {
            int bp, bt;
            const bool in = side == 0 ? pair_bin2(d, dO[o], ch, sh, p, bp, bt) : pair_bin2(dO[o], d, ch, sh, p, bp, bt);
            if (in) { lo = min(lo, bt); hi = max(hi, bt); }
          }
          for (int o = 16; o > 0; o >>= 1) {
            lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
          }
          if (hi >= lo && hi - lo + 1 <= TS) {
            wlo = lo;
            nrow = hi - lo + 1;
            for (int q = lane; q < nrow * np; q += 32) { myS[q] = 0.0; myL[q] = 0.0; }
            __syncwarp();
            for (int o = jlo + lane; o < jhi; o += 32) {
              int bp, bt;
              const bool in = side == 0 ? pair_bin2(d, dO[o], ch, sh, p, bp, bt) : pair_bin2(dO[o], d, ch, sh, p, bp, bt);
              if (in) {
                const int q = (bt - wlo) * np + bp;
                atomicAdd(&myS[q], wO[o]);
                atomicAdd(&myL[q], wO[o] * lO[o]);
              }
            }
          }
        }
        int sp = hi >= lo ? hi - lo + 1 : 0;
        if (sp > TS) {
          if (lane == 0) atomicAdd(p.err, 1ull);
          sp = 0;
        }
        if (lane == 0) {
          tlo[side * ML + m] = lo;
          span[side * ML + m] = sp;
        }
        __syncwarp();
        if (sp > 0) {
          // rows lo..hi of the built window go to the CTA's scratch
          double* rs = cS + (size_t)m * TS * NS;
          double* rl = cL + (size_t)m * TS * NS;
          const int off = (lo - wlo) * np;
          if ((np & 1) == 0) {   // NS == np: 16-byte copies, every row start on 16 bytes
            const int h = np / 2;
            for (int row = 0; row < sp; ++row) {
              const double2* ss = reinterpret_cast<const double2*>(myS + off + row * np);
              const double2* sl2 = reinterpret_cast<const double2*>(myL + off + row * np);
              double2* ds = reinterpret_cast<double2*>(rs + row * NS);
              double2* dl = reinterpret_cast<double2*>(rl + row * NS);
              for (int c2 = lane; c2 < h; c2 += 32) { ds[c2] = ss[c2]; dl[c2] = sl2[c2]; }
            }
          } else {
            for (int row = 0; row < sp; ++row) {
              for (int col = lane; col < NS; col += 32) {
                rs[row * NS + col] = col < np ? myS[off + row * np + col] : 0.0;
                rl[row * NS + col] = col < np ? myL[off + row * np + col] : 0.0;
              }
            }
          }
          if (lane == 0) {
            atomicMin(&s_T0, lo);
            atomicMax(&s_T1, lo + sp - 1);
            atomicMax(&s_maxspan, sp);
          }
        }
        __syncwarp();
      }
    }
    __syncthreads();
    const int T0 = s_T0, T1 = s_T1, maxspan = s_maxspan;
    if (T1 < T0) {   // no pixel pair in range
      __syncthreads();
      continue;
    }
    if (!moments_in_tiles) {
      for (int e = tid; e < 4 * nt * np; e += DT) {
        const int tb = (e / np) % nt;
        if (tb >= T0 && tb <= T1) mom[e] = 0.0;
      }
    }
    // coefficient of this lane's moment in the rank-4 part (0: M0, 1: Mi, 2: Mj, 3: Mij)
    const double cq = kq == 0 ? 1.0 / (om1 * om2) : kq == 1 ? io1 / om2 : kq == 2 ? io2 / om1 : io1 * io2;
    // ---- phase 2: blocks (t, u = t + d) of the window, d = 0 (the diagonal) first.
    // The rows of a chunk of pixels are copied from the column scratch into
    // shared memory asynchronously (16-byte cp.async, no registers), one chunk
    // ahead of the chunk the MMA warps multiply (double buffering); the row
    // weights k_S, k_L scale the A fragments as the MMA warps read them.  The
    // chunks of successive blocks form one sequence: the list of the next block's
    // pixels is built in this block's first chunk, its first chunk is copied
    // beside this block's last, and there is one barrier per chunk: 142.3 -> 137.0
    // ms (72,415 forest pairs) against a list, an exposed first chunk and two
    // barriers a chunk for each block.  Blocks with d >= maxspan have no column
    // products and come last, without barriers.
    // Bound: the FP64 MMAs of the blocks (27 of the 137 ms at their peak rate) and
    // the column build, which follow each other in a CTA, issue 46% busy on the
    // whole; two CTAs of 256 threads per SM, which would overlap them, take 157.8
    // ms (chunks of 16, shared loads per MMA).
    const int SET = CH * NPAD;   // doubles of one row set
    // pixels whose column spans both t and u = t + d, into list l
    auto build_list = [&](int t, int d, int l, int* cnt) {
      for (int side = 0; side < 2; ++side) {
        const int Lm = side == 0 ? L1 : L2;
        for (int m = tid; m < Lm; m += DT) {
          const int lo = tlo[side * ML + m], sp = span[side * ML + m];
          if (sp > 0 && lo <= t && t + d < lo + sp) {
            rows_of[l * 2 * ML + atomicAdd(cnt, 1)] = (side * ML + m) * TS + t - lo;   // row u is d further
          }
        }
      }
    };
    // a diagonal block stages the rows of t only: twice the pixels per chunk
    auto chunk_rows = [&](int d) { return d == 0 && moments_in_tiles ? 2 * CH : CH; };
    // Issues the copies of chunk ci of the block at distance d whose n pixels
    // are in list l, into buffer gb (rows beyond the chunk are zeroed with plain
    // stores).  Columns NS .. NPAD-1 are not copied: they keep older contents,
    // which reach only accumulator entries that are never flushed (tile columns
    // >= np), except the moment columns NS .. NS+3 written below, tile columns of
    // a diagonal block.
    auto issue = [&](int d, int l, int n, int ci, int gb) {
      const bool diag = d == 0, wide = diag && moments_in_tiles;
      const int CB = chunk_rows(d), BSET = CB * NPAD;
      double* buf = stage + (size_t)gb * 4 * SET;
      double* kb2 = kbuf + (size_t)gb * 4 * CH;
      const int c0 = ci * CB, rows = min(CB, n - c0), rows8 = (rows + 7) & ~7;
      const int* lr = rows_of + l * 2 * ML + c0;
      // up to four copies per row offset read; a division by the segments of a
      // row for every copy takes 147.3 ms instead of 142.3 (72,415 forest pairs)
      for (int r = cp_row; r < rows; r += cp_step) {
        int off = lr[r] * NS + 2 * cp_seg;
        double* dst = buf + r * NPAD + 2 * cp_seg;
        __pipeline_memcpy_async(dst, colS + off, 16);
        __pipeline_memcpy_async(dst + BSET, colL + off, 16);
        if (!diag) {   // rows of u
          off += d * NS;
          __pipeline_memcpy_async(dst + 2 * BSET, colS + off, 16);
          __pipeline_memcpy_async(dst + 3 * BSET, colL + off, 16);
        }
      }
      for (int q = tid; q < (diag ? 2 : 4) * (rows8 - rows) * NPAD; q += DT) {
        const int set = q / ((rows8 - rows) * NPAD), rem = q - set * (rows8 - rows) * NPAD;
        buf[(size_t)set * BSET + (size_t)rows * NPAD + rem] = 0.0;
      }
      for (int r = tid - (DT - 32); r >= 0 && r < rows8; r += 32) {   // the last warp
        const bool in = r < rows;
        const int m = in ? lr[r] / TS : 0, side = m >= ML;   // pixel of both sides' arrays
        const double wm = sw[m], dlm = sl[m];
        // weights of the column products: an f1 pixel i enters with w_i/Om2 (S)
        // and w_i/O2 (L), an f2 pixel j with w_j/Om1 and w_j/O1
        kb2[r] = in ? wm * (side == 0 ? kS1 : kS2) : 0.0;
        kb2[CB + r] = in ? wm * (side == 0 ? io2 : io1) : 0.0;
        const bool f1r = in && side == 0;
        if (!wide) {
          kb2[2 * CH + r] = f1r ? wm : 0.0;
          kb2[3 * CH + r] = f1r ? wm * dlm : 0.0;
        } else {   // moment columns of the S and L rows of bin t
          double* rs = buf + (size_t)r * NPAD + NS;
          double* rl = buf + BSET + (size_t)r * NPAD + NS;
          rs[0] = f1r ? om2 : 0.0; rs[1] = f1r ? om2 * dlm : 0.0; rs[2] = 0.0; rs[3] = 0.0;
          rl[0] = 0.0; rl[1] = 0.0; rl[2] = f1r ? odl2b : 0.0; rl[3] = f1r ? odl2b * dlm : 0.0;
        }
      }
      __pipeline_commit();
    };
    const int dprod = min(maxspan, T1 - T0 + 1);   // blocks at d < dprod have column products
    if (tid < 3) s_cnt[tid] = 0;
    __syncthreads();
    build_list(T0, 0, 0, &s_cnt[0]);
    __syncthreads();
    int gb = 0;                // buffer of the next chunk to multiply
    int ls = 0;                // counter of the current block's list
    int l = 0;                 // the current block's list
    if (s_cnt[0] > 0) issue(0, 0, s_cnt[0], 0, 0);
    for (int t = T0, d = 0; t + d <= T1;) {
      const bool diag = d == 0;
      const int u = t + d;
      const int tn = t + d < T1 ? t + 1 : T0, dn = t + d < T1 ? d : d + 1;   // the next block
      double acc[CC][4];
#pragma unroll
      for (int c = 0; c < CC; ++c) { acc[c][0] = 0.0; acc[c][1] = 0.0; acc[c][2] = 0.0; acc[c][3] = 0.0; }
      const bool sym = diag && moments_in_tiles;   // tiles of the upper triangle only
      // The rank-4 part, subtracted from the tiles as one MMA each with the four
      // moments as k (lane kq: moment kq; k 4 .. 7 are zero).  Formed per entry in
      // the flush it read eight moments per pair of entries after the last
      // barrier: 149.7 against 147.3 ms (72,415 forest pairs).
      auto rank4 = [&]() {
        const double* mq = mom + (size_t)kq * nt * np;
        const double* mt_ = mq + (size_t)t * np;
        const double* mu_ = mq + (size_t)u * np;
#pragma unroll
        for (int c = 0; c < CC; ++c) {
          const int row = sym ? sym_row[c] : mt, col = sym ? sym_col[c] : ng + nwm * c;
          if (row < 0 || col >= ntile) continue;
          const int bp0 = 16 * row + grp, bp1 = bp0 + 8, bq = 8 * col + grp;
          lya_dmma_16x8x8(acc[c], bp0 < np ? -cq * mt_[bp0] : 0.0, bp1 < np ? -cq * mt_[bp1] : 0.0, 0.0, 0.0,
                          bq < np ? mu_[bq] : 0.0, 0.0);
        }
      };
      if (!diag) rank4();   // the diagonal blocks have completed the moments
      if (d < dprod) {
        const bool more = dn < dprod && tn + dn <= T1;   // the next block has column products
        const int ln = l ^ 1, lsn = ls == 2 ? 0 : ls + 1, lsz = lsn == 2 ? 0 : lsn + 1;
        const int n = s_cnt[ls], CB = chunk_rows(d), BSET = CB * NPAD;
        const int nch = max((n + CB - 1) / CB, 1);   // an empty list: one step, no rows
        for (int ci = 0; ci < nch; ++ci) {
          __pipeline_wait_prior(0);   // this thread's copies of chunk ci have landed
          __syncthreads();            // everyone's have; the other buffer and the other list are free
          if (ci == 0) {
            if (more) build_list(tn, dn, ln, &s_cnt[lsn]);
            if (tid == 0) s_cnt[lsz] = 0;   // read by everyone in the block before, used in the next
          }
          if (ci + 1 < nch) {
            issue(d, l, n, ci + 1, gb ^ 1);
          } else if (more) {
            if (nch == 1) __syncthreads();   // the next list is complete
            const int nn = s_cnt[lsn];
            if (nn > 0) issue(dn, ln, nn, 0, gb ^ 1);
          }
          const double* buf = stage + (size_t)gb * 4 * SET;
          const double* kb2 = kbuf + (size_t)gb * 4 * CH;
          const double* SA = buf;                      // rows of bin t: S, L (unscaled)
          const double* LA = buf + BSET;
          const double* SB = diag ? SA : buf + 2 * SET;   // rows of bin u
          const double* LB = diag ? LA : buf + 3 * SET;
          const int c0 = ci * CB, rows = min(CB, n - c0), rows8 = (rows + 7) & ~7;
          if (tid == 0) n_mma += (unsigned long long)((rows + 3) / 4) * (sym ? sym_tiles : ntile * ntile) * 2;
          if (diag && !sym) {   // moments of bin t from the rows of the f1 pixels
            for (int e = tid; e < 4 * np; e += DT) {
              const int q = e / np, bq = e - q * np;
              const double* src = (q < 2 ? SA : LA) + bq;   // 0: M0, 1: Mi from S; 2: Mj, 3: Mij from L
              const double* cw = kb2 + ((q == 0 || q == 2) ? 2 : 3) * CH;   // f1 w or w dl, 0 for f2 rows
              double sacc = 0.0;
#pragma unroll 4
              for (int r = 0; r < rows; ++r) sacc = fma(cw[r], src[r * NPAD], sacc);
              mom[(q * nt + t) * np + bq] += sacc;
            }
          }
          if (sym) {
#pragma unroll
            for (int c = 0; c < CC; ++c) {
              if (sym_row[c] < 0) continue;
              const int bp0 = 16 * sym_row[c] + grp, bp1 = bp0 + 8, bq = 8 * sym_col[c] + grp;
              const bool v0 = bp0 < np, v1 = bp1 < np;
              for (int r0 = 0; r0 < rows8; r0 += 8) {
                const int ra = (r0 + kq) * NPAD, rb = ra + 4 * NPAD;
                const double ks0 = kb2[r0 + kq], ks1 = kb2[r0 + kq + 4];
                const double kl0 = kb2[CB + r0 + kq], kl1 = kb2[CB + r0 + kq + 4];
                lya_dmma_16x8x8(acc[c], v0 ? SA[ra + bp0] * ks0 : 0.0, v1 ? SA[ra + bp1] * ks0 : 0.0,
                                v0 ? SA[rb + bp0] * ks1 : 0.0, v1 ? SA[rb + bp1] * ks1 : 0.0, SA[ra + bq], SA[rb + bq]);
                lya_dmma_16x8x8(acc[c], v0 ? LA[ra + bp0] * kl0 : 0.0, v1 ? LA[ra + bp1] * kl0 : 0.0,
                                v0 ? LA[rb + bp0] * kl1 : 0.0, v1 ? LA[rb + bp1] * kl1 : 0.0, LA[ra + bq], LA[rb + bq]);
              }
            }
          } else {
            const int bp0 = 16 * mt + grp, bp1 = bp0 + 8;
            const bool v0 = bp0 < np, v1 = bp1 < np;
            for (int r0 = 0; r0 < rows8; r0 += 8) {
              const int ra = (r0 + kq) * NPAD, rb = ra + 4 * NPAD;
              const double ks0 = kb2[r0 + kq], ks1 = kb2[r0 + kq + 4];
              const double kl0 = kb2[CH + r0 + kq], kl1 = kb2[CH + r0 + kq + 4];
              const double as0 = v0 ? SA[ra + bp0] * ks0 : 0.0, as1 = v1 ? SA[ra + bp1] * ks0 : 0.0;
              const double as2 = v0 ? SA[rb + bp0] * ks1 : 0.0, as3 = v1 ? SA[rb + bp1] * ks1 : 0.0;
              const double al0 = v0 ? LA[ra + bp0] * kl0 : 0.0, al1 = v1 ? LA[ra + bp1] * kl0 : 0.0;
              const double al2 = v0 ? LA[rb + bp0] * kl1 : 0.0, al3 = v1 ? LA[rb + bp1] * kl1 : 0.0;
#pragma unroll
              for (int c = 0; c < CC; ++c) {
                const int nt8 = ng + nwm * c;
                if (nt8 < ntile) {
                  lya_dmma_16x8x8(acc[c], as0, as1, as2, as3, SB[ra + 8 * nt8 + grp], SB[rb + 8 * nt8 + grp]);
                  lya_dmma_16x8x8(acc[c], al0, al1, al2, al3, LB[ra + 8 * nt8 + grp], LB[rb + 8 * nt8 + grp]);
                }
              }
            }
          }
          gb ^= 1;
        }
        l = ln;
        ls = lsn;
        if (sym) {   // accumulator columns NS..NS+3: the moments of bin t
#pragma unroll
          for (int c = 0; c < CC; ++c) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int bp = 16 * sym_row[c] + grp + 8 * (i >> 1), q = 8 * sym_col[c] + 2 * kq + (i & 1) - NS;
              if (sym_row[c] >= 0 && bp < np && q >= 0 && q < 4) mom[(q * nt + t) * np + bp] = acc[c][i];
            }
          }
        }
        if (diag) __syncthreads();   // the moments of bin t are complete
      }
      if (diag) rank4();
      // flush: the tiles (column products less the rank-4 part) subtracted, the
      // diagonal added.  A diagonal block from its upper triangle, both halves
      // from one value.
#pragma unroll
      for (int c = 0; c < CC; ++c) {
        const int row = sym ? sym_row[c] : mt, col = sym ? sym_col[c] : ng + nwm * c;
        if (row < 0 || col >= ntile) continue;
#pragma unroll
        for (int h2 = 0; h2 < 2; ++h2) {
          const int bp = 16 * row + grp + 8 * h2;
          if (bp >= np) continue;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int bq = 8 * col + 2 * kq + i;
            if (bq >= np || (sym && bq < bp)) continue;
            double v = -acc[c][2 * h2 + i];
            const int A = bp * nt + t, B = bq * nt + u;
            if (A == B) {
              const double m0a = mom[(size_t)t * np + bp];
              v += m0a;
              if (m0a != 0.0) atomicAdd(&p.W[A], m0a);
            }
            if (v != 0.0) {   // nb * nb < 2^24
              atomicAdd(&p.D[A * nb + B], v);
              if (t != u || (sym && A != B)) atomicAdd(&p.D[B * nb + A], v);
            }
          }
        }
      }
      t = tn;
      d = dn;
    }
    __syncthreads();
  }
  if (tid == 0 && n_mma) atomicAdd(p.mma, n_mma);
}

template <int V>
cudaError_t set_dist_smem_v(int smem) {
  return cudaFuncSetAttribute(k_dist<DIST_SHAPES[V].dt, DIST_SHAPES[V].ch>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              smem);
}

cudaError_t set_dist_smem(int shape, int smem) {
  switch (shape) {
    case 1: return set_dist_smem_v<1>(smem);
    case 2: return set_dist_smem_v<2>(smem);
    case 3: return set_dist_smem_v<3>(smem);
    case 4: return set_dist_smem_v<4>(smem);
    default: return set_dist_smem_v<0>(smem);
  }
}

template <int V>
cudaError_t launch_dist_v(int grid, size_t smem, cudaStream_t s, const DistParams& p) {
  k_dist<DIST_SHAPES[V].dt, DIST_SHAPES[V].ch><<<grid, DIST_SHAPES[V].dt, smem, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_dist(int shape, int grid, size_t smem, cudaStream_t s, const DistParams& p) {
  switch (shape) {
    case 1: return launch_dist_v<1>(grid, smem, s, p);
    case 2: return launch_dist_v<2>(grid, smem, s, p);
    case 3: return launch_dist_v<3>(grid, smem, s, p);
    case 4: return launch_dist_v<4>(grid, smem, s, p);
    default: return launch_dist_v<0>(grid, smem, s, p);
  }
}
static_assert(N_DIST_SHAPES == 5, "the launch tables above cover every shape");
static_assert(DIST_SHAPES[0].ch % 8 == 0 && DIST_SHAPES[1].ch % 8 == 0 && DIST_SHAPES[2].ch % 8 == 0 &&
                  DIST_SHAPES[3].ch % 8 == 0 && DIST_SHAPES[4].ch % 8 == 0 && DIST_SHAPES[3].dt % 128 == 0,
              "chunks hold whole MMA K steps; the warps cover the four tile rows");

}  // namespace

extern "C" int lya_dist_config(lya_ctx* ctx, int32_t shape, int64_t max_items) {
  if (!ctx) return lya_fail(nullptr, LYA_ERR_ARG, "lya_dist_config: ctx is NULL");
  if (shape < 0 || shape >= N_DIST_SHAPES)
    return lya_fail(ctx, LYA_ERR_ARG, "lya_dist_config: shape %d outside [0,%d)", shape, N_DIST_SHAPES);
  if (max_items < 0) return lya_fail(ctx, LYA_ERR_ARG, "lya_dist_config: max_items < 0");
  ctx->dist_shape = shape;
  ctx->dist_max_items = max_items;
  return LYA_OK;
}

extern "C" int lya_dist_run(lya_ctx* ctx, double* D, double* W) {
  if (!ctx) return lya_fail(nullptr, LYA_ERR_ARG, "lya_dist_run: ctx is NULL");
  if (!ctx->bins_set) return lya_fail(ctx, LYA_ERR_STATE, "lya_dist_run: call lya_set_bins first");
  if (ctx->cat.n == 0) return lya_fail(ctx, LYA_ERR_STATE, "lya_dist_run: no forests uploaded");
  if (!ctx->cat.has_dl || !ctx->cat.has_moments)
    return lya_fail(ctx, LYA_ERR_STATE, "lya_dist_run: upload dl, omega and odl2 with the forests");
  const int np = ctx->np, nt = ctx->nt, nb = np * nt;
  if (np > NP_MAX) return lya_fail(ctx, LYA_ERR_ARG, "lya_dist_run: np = %d above %d r_par bins", np, NP_MAX);
  LYA_CHECK_CUDA(ctx, cudaSetDevice(ctx->device));
  int max_len = 1;
  for (int64_t f = 0; f < ctx->cat.n; ++f)
    max_len = std::max<int>(max_len, (int)(ctx->h_start[f + 1] - ctx->h_start[f]));
  if (max_len > 65535) return lya_fail(ctx, LYA_ERR_DATA, "lya_dist_run: forests longer than 65535 pixels");
  const int npad = stage_npad(np);
  const int shape = ctx->dist_shape;
  const int DT = DIST_SHAPES[shape].dt, CH = DIST_SHAPES[shape].ch, NW = DT / 32;
  const size_t stage_len = (size_t)stage_doubles(CH, NW, np);
  // the longest forest a shape takes (the layout launched below needs 24 bytes per pixel less)
  constexpr size_t SMEM_MAX = 227 * 1024;
  const size_t smem = sizeof(double) * (10 * (size_t)max_len + stage_len + 8 * (size_t)CH) +
                      sizeof(int) * (6 * (size_t)max_len);
  if (smem > SMEM_MAX)
    return lya_fail(ctx, LYA_ERR_DATA, "lya_dist_run: forests of %d pixels need %zu B of shared memory (shape %d)",
                    max_len, smem, shape);
  const int grid = ctx->num_sms;
  // scratch and outputs kept in the context, so later calls (one per healpix
  // pixel in the drop-in driver) allocate nothing and replay the captured graph
  DistScratch& ds = ctx->dist;
  // (binnings of equal nb differ in np, and so in the length of a column's rows)
  const int stride = col_stride(np);
  if (!ds.D || ds.nb != nb || ds.max_len < max_len || ds.stride < stride || ds.grid != grid) {
    lya_free(ds.D); lya_free(ds.W); lya_free(ds.col); lya_free(ds.mom); lya_free(ds.err);
    if (ds.graph) { cudaGraphExecDestroy(ds.graph); ds.graph = nullptr; }
    ds = DistScratch{};
    cudaError_t e = lya_alloc(&ds.D, (size_t)nb * nb);
    if (e == cudaSuccess) e = lya_alloc(&ds.W, nb);
    if (e == cudaSuccess) e = lya_alloc(&ds.col, (size_t)grid * 2 * 2 * max_len * TS * stride);
    if (e == cudaSuccess) e = lya_alloc(&ds.mom, (size_t)grid * 4 * nt * np);
    if (e == cudaSuccess) e = lya_alloc(&ds.err, 4);
    if (e != cudaSuccess) {
      lya_free(ds.D); lya_free(ds.W); lya_free(ds.col); lya_free(ds.mom); lya_free(ds.err);
      ds = DistScratch{};
      return lya_fail(ctx, LYA_ERR_ALLOC, "lya_dist_run: device allocation failed");
    }
    ds.nb = nb; ds.max_len = max_len; ds.stride = stride; ds.grid = grid;
  }
  cudaStream_t s = ctx->stream;
  const long long n_items = ctx->dist_max_items > 0 ? std::min<long long>(ctx->wq.n_pairs, ctx->dist_max_items)
                                                    : ctx->wq.n_pairs;
  // Pixels per forest of the kernel's layout: the scratch's, so that the captured
  // graph serves any catalogue, unless that is more than this shape holds (a
  // catalogue of longer forests ran before it, with a shape of smaller chunks).
  auto layout_bytes = [&](int pixels) {
    return sizeof(double) * (6 * (size_t)pixels + stage_len + 8 * (size_t)CH) + sizeof(int) * (8 * (size_t)pixels);
  };
  const int ml = layout_bytes(ds.max_len) <= SMEM_MAX ? ds.max_len : max_len;
  const size_t smem_run = layout_bytes(ml);
  DistParams p;
  memset(&p, 0, sizeof(p));   // padding bytes take part in the graph key
  p.pix8 = ctx->cat.pix8; p.dl = ctx->cat.dl; p.pstart = ctx->cat.pstart; p.len = ctx->cat.len;
  p.sorted = ctx->cat.sorted; p.ux = ctx->cat.ux; p.uy = ctx->cat.uy; p.uz = ctx->cat.uz;
  p.omega = ctx->cat.omega; p.odl2 = ctx->cat.odl2; p.f1 = ctx->wq.f1; p.f2 = ctx->wq.f2;
  p.n_items = reinterpret_cast<const long long*>(ds.err + 2); p.max_len = ml;
  p.binner_rp = (double)np / ctx->rpmax; p.binner_rt = (double)nt / ctx->rtmax;
  p.np = np; p.nt = nt; p.nb = nb; p.cos_variant = ctx->cos_variant; p.npad = npad;
  p.col = ds.col; p.moments = ds.mom; p.D = ds.D; p.W = ds.W; p.err = ds.err; p.next = ds.err + 1;
  p.mma = ds.err + 3;
  p.shape = shape;
  static_assert(sizeof(DistParams) <= sizeof(ds.key), "graph key does not fit");
  cudaError_t e = cudaSuccess;
  if (!ds.graph || memcmp(ds.key, &p, sizeof(p)) != 0) {
    if (ds.graph) { cudaGraphExecDestroy(ds.graph); ds.graph = nullptr; }
    e = set_dist_smem(shape, (int)smem_run);
    cudaGraph_t g = nullptr;
    if (e == cudaSuccess) e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
    if (e == cudaSuccess) {
      cudaError_t eq = cudaMemsetAsync(ds.D, 0, sizeof(double) * (size_t)nb * nb, s);
      if (eq == cudaSuccess) eq = cudaMemsetAsync(ds.W, 0, sizeof(double) * nb, s);
      if (eq == cudaSuccess) eq = cudaMemsetAsync(ds.err, 0, 2 * sizeof(unsigned long long), s);
      if (eq == cudaSuccess) eq = cudaMemsetAsync(ds.err + 3, 0, sizeof(unsigned long long), s);
      if (eq == cudaSuccess) {
        eq = launch_dist(shape, grid, smem_run, s, p);
      }
      const cudaError_t ec = cudaStreamEndCapture(s, &g);
      e = eq != cudaSuccess ? eq : ec;
    }
    if (e == cudaSuccess) e = cudaGraphInstantiate(&ds.graph, g, 0);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess) {
      ds.graph = nullptr;
      return lya_fail(ctx, LYA_ERR_CUDA, "lya_dist_run: capture: %s", cudaGetErrorString(e));
    }
    memcpy(ds.key, &p, sizeof(p));
  }
  e = cudaMemcpyAsync(ds.err + 2, &n_items, sizeof(n_items), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->ev0, s);
  if (e == cudaSuccess) e = cudaGraphLaunch(ds.graph, s);
  if (e == cudaSuccess) {
    ctx->launches++;
    e = cudaEventRecord(ctx->ev1, s);
  }
  unsigned long long nerr = 0, nmma = 0;
  if (e == cudaSuccess) e = lya_touch_pages(D, sizeof(double) * (size_t)nb * nb);   // beside the kernel
  if (e == cudaSuccess) e = cudaMemcpyAsync(&nerr, ds.err, sizeof(nerr), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&nmma, ds.err + 3, sizeof(nmma), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && D) e = cudaMemcpyAsync(D, ds.D, sizeof(double) * (size_t)nb * nb, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess && W) e = cudaMemcpyAsync(W, ds.W, sizeof(double) * nb, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  float ms = 0.f;
  if (e == cudaSuccess) cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  if (e != cudaSuccess) return lya_fail(ctx, LYA_ERR_CUDA, "lya_dist_run: %s", cudaGetErrorString(e));
  ctx->last.kernel_ms = ms;
  ctx->last.dist_mma_flops = (double)nmma * 2.0 * 8 * 8 * 4;   // m8n8k4: 256 FMA per MMA
  if (nerr) return lya_fail(ctx, LYA_ERR_DATA, "lya_dist_run: %llu pixels pair into more than %d rt bins", nerr, TS);
  return LYA_OK;
}
