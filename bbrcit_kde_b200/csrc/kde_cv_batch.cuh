// Batched cross-validation over a bandwidth grid and many datasets in one
// persistent launch (Epanechnikov product kernel).
//
// The reference evaluates one bandwidth at a time: likelihood_cross_validate
// (KernelDensityImpl.h:215-252) and lsq_convolution_cross_validate (:142-209),
// each an all-pairs self-evaluation, called in a host loop over the grid
// (grid_search/grid_search.cc:370-402). Here every (hx_a, hy_b) of the grid comes
// out of one pass over the point pairs:
//
//   Epanechnikov product: K_ab(dx, dy) = (1 - dx^2/hx_a^2)(1 - dy^2/hy_b^2) on
//   |dx| < hx_a, |dy| < hy_b. A pair with p = #{a: hx_a <= |dx|} and
//   q = #{b: hy_b <= |dy|} contributes to exactly the bandwidths a >= p, b >= q,
//   with a polynomial in (1/hx_a^2, 1/hy_b^2). So for one query i the moments
//   M_kl[p][q] = sum_j m_j dx^k dy^l (k, l in {0, 2}) binned by (p, q), then 2-D
//   inclusive prefix sums over (p, q), give
//     S_i[a][b] = P00 - P20/hx_a^2 - P02/hy_b^2 + P22/(hx_a^2 hy_b^2)
//   = sum_{j != i} m_j K_ab for all 4096 (a, b) at once; the likelihood needs
//   log(C_ab S_i[a][b]) per query, so this is done per query.
//
//   Convolution kernel (KernelTraits.h:353-357): P(u) = (2-u)^3 (u^2+6u+4)/32
//   = 1 - 5/4 u^2 + 5/8 u^3 - 1/32 u^5 on u < 2, so the same binning with the
//   16 moments {1, x^2, x^3, x^5} x {1, y^2, y^3, y^5} and cells p = #{a: 2 hx_a <= |dx|}
//   gives sum_{i,j} w_i m_j Kc_ab for all (a, b); it is linear, so it is
//   accumulated over all pairs (i < j, doubled) rather than per query.
//
// Pairs are enumerated from a uniform grid over each dataset (points sorted by
// grid cell on the host, in Morton order inside each cell), visiting only cells
// within the largest support. All arithmetic of the final scores is FP64; the
// moments are exact 64-bit fixed point.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace bbkde {

constexpr int kCvMaxH = 64;                   // bandwidths per axis
constexpr int kCvCells = kCvMaxH * kCvMaxH;   // (p, q) cells
constexpr int kCvLut = 1024;                  // log2 bins of the cell lookup
constexpr int kCvMaxRanges = 2 * 8 + 1;       // candidate cell rows per query
constexpr int kCvRow = kCvMaxH + 1;           // histogram row stride (bank spread)
constexpr int kCvHist = kCvMaxH * kCvRow;     // padded (p, q) histogram size

struct CvSet {
  int64_t begin, n;          // point range in the concatenated arrays
  int64_t cell_begin;        // offset of this set's cell_start[gx * gy + 1]
  double x0, y0, inv_cell;   // grid origin and 1 / cell size
  int gx, gy;
  double diag_wm;            // sum_i w_i m_i (the i == j convolution terms)
  int uniform;               // every point has the same weight, and the bandwidths are
                             // within 1e-60 .. 1e60, so that a density is 0 or normal
                             // (nonzero sums are above 2^-120)
  int pad;
};

// Work item: queries [q0, q1) of one set; kind 0 = likelihood / leave-one-out
// pass (part = its row in the partial buffer), kind 1..4 = convolution pass for
// x-power group kind - 1 over queries of the grid cells (cx .. cx1, cy).
struct CvItem {
  int set, kind, part, cx;
  int cy, cx1;
  int64_t q0, q1;
};

struct CvArgs {
  const double *x, *y, *w, *m;      // points sorted by grid cell, concatenated
  const int64_t *cell_start;        // per set: gx * gy + 1 offsets (set-relative)
  const CvSet *sets;
  const CvItem *items;
  int n_items;
  int *counter;                     // dynamic work counter (zeroed before launch)
  int nhx, nhy;
  const double *hx, *hy;            // ascending
  const unsigned char *lutx, *luty; // lower-bound cell counts per bin of the key
  long long lut_basex, lut_basey;   // key of the first bin (see cv_cell)
  int lut_shift;                    // key = double bits >> lut_shift
  int r_epan, r_conv;               // candidate half-widths in grid cells
  double *epan_part;                // [part][2][kCvCells]: sum w log f, sum w f
  double *conv_hist;                // [set][16][kCvCells]
  unsigned long long *pairs;        // [0] likelihood pairs in support (4 atomics each),
                                    // [1] convolution pairs in support (4 per x-group)
};

// #{h[a] <= v} for v >= 0. The key (the double's bits shifted right: exponent
// and leading mantissa bits) is monotone in v; the table holds, per key bin, the
// count at the bin's lower edge, so it is a lower bound that a short exact
// correction finishes (at most one grid boundary per bin).
__device__ __forceinline__ int cv_cell(double v, const double *h, int n,
                                       const unsigned char *lut, long long base, int shift) {
  long long idx = (__double_as_longlong(v) >> shift) - base;
  idx = idx < 0 ? 0 : (idx >= kCvLut ? kCvLut - 1 : idx);
  int p = lut[idx];
  while (p < n && h[p] <= v) ++p;
  return p;
}

__device__ __forceinline__ void cv_cell_of(const CvSet &s, double x, double y, int &cx, int &cy) {
  cx = (int)floor((x - s.x0) * s.inv_cell);
  cy = (int)floor((y - s.y0) * s.inv_cell);
  cx = cx < 0 ? 0 : (cx >= s.gx ? s.gx - 1 : cx);
  cy = cy < 0 ? 0 : (cy >= s.gy ? s.gy - 1 : cy);
}

// Candidate ranges (set-relative point indices) of the grid rows within `r`
// cells of the cells (cx .. cx1, cy), one row per lane of warp 0, keeping only
// indices >= min_j. Empty rows stay as empty ranges. Returns through shared memory.
__device__ __forceinline__ void cv_ranges(const CvSet &s, const int64_t *cs, int cx, int cx1,
                                          int cy, int r, int64_t min_j, int *rb, int *pre,
                                          int *nr) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int clo = cx - r < 0 ? 0 : cx - r;
    const int chi = cx1 + r >= s.gx ? s.gx - 1 : cx1 + r;
    const int rlo = cy - r < 0 ? 0 : cy - r;
    const int rhi = cy + r >= s.gy ? s.gy - 1 : cy + r;
    const int rows = rhi - rlo + 1;   // <= 2 r + 1 <= kCvMaxRanges <= 32
    int b = 0, len = 0;   // a set has fewer than 2^31 points
    if (lane < rows) {
      const int row = rlo + lane;
      b = (int)cs[(int64_t)row * s.gx + clo];
      const int e = (int)cs[(int64_t)row * s.gx + chi + 1];
      if (b < min_j) b = (int)min_j;
      len = e > b ? e - b : 0;
    }
    int incl = len;   // inclusive warp scan of the lengths
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane < rows) {
      rb[lane] = b;
      pre[lane] = incl - len;
    }
    if (lane == rows - 1) {
      pre[rows] = incl;
      *nr = rows;
    }
  }
}

// Moments are accumulated per cell in 64-bit fixed point, normalised by the
// cell's bandwidth so every contribution lies in [0, m]: for cell p the x-part is
// x~ = |dx| / h_p (likelihood pass, |dx| < h_p) or |dx| / (2 h_p) (convolution
// pass), both < 1. Integer atomics are exact and order-independent, so results
// are bitwise reproducible; cells are converted to FP64 (times h_p^k) before the
// FP64 prefix sums.
constexpr double kCvFixLik = 4611686018427387904.0;   // 2^62: sum of masses <= 1
constexpr double kCvFixConv = 2305843009213693952.0;  // 2^61: sum of 2 w_i m_j <= 2

// Run accumulation: a thread keeps the four fixed-point moments of its latest
// cell in registers while consecutive pairs fall into the same (p, q) cell, and
// adds them to the histograms when the cell changes (and at the end of its
// pairs). Points are Morton-ordered within each grid cell, so consecutive pairs
// of a thread are spatial neighbours and share a cell wherever the bandwidth
// bins are wider than the point spacing. The sums are the same integers in
// another order: exact, and the histograms identical.
struct CvRun {
  int c = -1;
  unsigned long long a0 = 0, a1 = 0, a2 = 0, a3 = 0;
};

// Fire-and-forget shared-memory reduction (no returned value, so the warp does
// not wait for it); exact 64-bit integer addition.
__device__ __forceinline__ void cv_red(unsigned long long *h, unsigned long long iv) {
  const unsigned addr = (unsigned)__cvta_generic_to_shared(h);
  asm volatile("red.shared.add.u64 [%0], %1;" ::"r"(addr), "l"(iv) : "memory");
}

__device__ __forceinline__ void cv_run_flush(unsigned long long *H, CvRun &r) {
  if (r.c >= 0) {
    cv_red(&H[r.c], r.a0);
    cv_red(&H[kCvHist + r.c], r.a1);
    cv_red(&H[2 * kCvHist + r.c], r.a2);
    cv_red(&H[3 * kCvHist + r.c], r.a3);
    r.c = -1;
  }
}

__device__ __forceinline__ void cv_run_add(unsigned long long *H, CvRun &r, int c, double v0,
                                           double v1, double v2, double v3) {
  const unsigned long long i0 = (unsigned long long)__double2ll_rn(v0);
  const unsigned long long i1 = (unsigned long long)__double2ll_rn(v1);
  const unsigned long long i2 = (unsigned long long)__double2ll_rn(v2);
  const unsigned long long i3 = (unsigned long long)__double2ll_rn(v3);
  if (c != r.c) {
    cv_run_flush(H, r);
    r.c = c;
    r.a0 = i0; r.a1 = i1; r.a2 = i2; r.a3 = i3;
  } else {
    r.a0 += i0; r.a1 += i1; r.a2 += i2; r.a3 += i3;
  }
}

constexpr int kCvQBlock = 256;   // queries of one convolution item (staged in smem)
constexpr int kCvUnroll = 2;     // consecutive candidates per thread and step
constexpr int kCvThreads = 1024;
constexpr int kCvSegs1 = 8;      // segments of a row in the likelihood's first prefix ...
constexpr int kCvSegs2 = 16;     // ... and of a column in its second

// Shared memory: H[4][kCvHist] (fixed point) | likelihood prefix rows [2][kCvHist]
// (the convolution's query block x, y, 2 w) | segment totals | hx | hy | 1/hx | 1/hy
// | 1/hx^2 | 1/hy^2 | ranges | misc | LUTs.
constexpr size_t kCvTotals = 4 * kCvSegs1 * kCvMaxH;
static_assert(kCvTotals >= 2 * kCvSegs2 * kCvMaxH && 2 * kCvHist >= 3 * kCvQBlock, "shared areas");
static_assert(kCvMaxH * kCvSegs1 * 2 == kCvThreads && kCvMaxH * kCvSegs2 == kCvThreads,
              "one thread per (row, segment, moment pair) and per (column, segment)");

__host__ __device__ constexpr size_t cv_smem_bytes() {
  return sizeof(double) * (6 * kCvHist + kCvTotals + 6 * kCvMaxH) +
         sizeof(int) * (2 * kCvMaxRanges + 1 + 4) + 2 * kCvLut;
}

// What bounds the likelihood items: per query the 4 x 64 x 64 fixed-point moments
// are read and cleared once (2 x 133 KB of shared memory, ~2,100 clocks) and one
// logarithm per bandwidth pair runs on the FP64 pipe (~2,600 clocks at 64 x 64);
// both prefix directions are therefore split over all 1,024 threads (8 or 4 cells
// in registers, segment totals exchanged once), and the next query's pairs are
// counted in the same interval as this query's logarithms. Measured,
// four sets of 1,500-9,000 points at 64 x 48 bandwidths: 4.0 ms (17.2 ms with one
// serial 64-step prefix per row and column and items of 1,024 queries); 16 sets of
// 20,000 points at 64 x 64: 167 ms (176 ms), where the pairs are the bound.
__global__ void __launch_bounds__(kCvThreads, 1) k_cv_batch(CvArgs a) {
  extern __shared__ __align__(16) double sh[];
  unsigned long long *H = reinterpret_cast<unsigned long long *>(sh);   // 4 * kCvHist
  double *PA = sh + 4 * kCvHist;       // row prefixes of {1, y^2} and ...
  double *PB = PA + kCvHist;           // ... {x^2, x^2 y^2}, combined per bandwidth b
  double *bqx = PA;                    // kCvQBlock each
  double *bqy = bqx + kCvQBlock;
  double *bqw = bqy + kCvQBlock;
  double *tot = PA + 2 * kCvHist;      // kCvTotals
  double *shx = tot + kCvTotals;
  double *shy = shx + kCvMaxH;
  double *ihx = shy + kCvMaxH;
  double *ihy = ihx + kCvMaxH;
  double *ihx2 = ihy + kCvMaxH;
  double *ihy2 = ihx2 + kCvMaxH;
  int *rb = reinterpret_cast<int *>(ihy2 + kCvMaxH);   // kCvMaxRanges
  int *pre = rb + kCvMaxRanges;                        // kCvMaxRanges + 1
  int *misc = pre + kCvMaxRanges + 1;                  // [0] item, [1] nr
  unsigned char *slutx = reinterpret_cast<unsigned char *>(misc + 4);
  unsigned char *sluty = slutx + kCvLut;

  const int tid = threadIdx.x;
  const int nt = blockDim.x;
  const int lane = tid & 31;
  for (int i = tid; i < kCvMaxH; i += nt) {
    double hx = i < a.nhx ? a.hx[i] : 1e300;
    double hy = i < a.nhy ? a.hy[i] : 1e300;
    shx[i] = hx;
    shy[i] = hy;
    ihx[i] = 1.0 / hx;
    ihy[i] = 1.0 / hy;
    ihx2[i] = 1.0 / (hx * hx);
    ihy2[i] = 1.0 / (hy * hy);
  }
  for (int i = tid; i < kCvLut; i += nt) {
    slutx[i] = a.lutx[i];
    sluty[i] = a.luty[i];
  }
  const double hxmax = a.hx[a.nhx - 1], hymax = a.hy[a.nhy - 1];
  unsigned long long n_lik = 0, n_conv = 0;   // in-support pairs of this thread
  __syncthreads();

  for (;;) {
    if (tid == 0) misc[0] = atomicAdd(a.counter, 1);
    __syncthreads();
    const int it = misc[0];
    __syncthreads();
    if (it >= a.n_items) break;
    const CvItem item = a.items[it];
    const CvSet s = a.sets[item.set];
    const int64_t *cs = a.cell_start + s.cell_begin;
    const double *X = a.x + s.begin, *Y = a.y + s.begin, *Wt = a.w + s.begin,
                 *M = a.m + s.begin;

    if (item.kind == 0) {
      // ---- likelihood / leave-one-out pass, one query at a time ----------
      for (int c = tid; c < 4 * kCvHist; c += nt) H[c] = 0ull;
      // First prefix (along q): thread (row p1, segment s1 of 8 columns, moment pair
      // mp). Second (along p) and scores: thread (column b2, segment s2 of 4 rows),
      // whose four scores stay in registers for all queries of the item.
      constexpr int C1 = kCvMaxH / kCvSegs1, C2 = kCvMaxH / kCvSegs2;
      const int p1 = tid % kCvMaxH, s1 = (tid / kCvMaxH) % kCvSegs1, mp = tid / (kCvMaxH * kCvSegs1);
      const int b2 = tid % kCvMaxH, s2 = tid / kCvMaxH;
      // With equal weights sum w log f = w log prod f: lik holds the product's
      // mantissa in [1, 2) (0 once a factor is 0), lexp its exponent.
      double lik[C2], llo[C2];
      int lexp[C2];
      const bool uniform = s.uniform != 0;
#pragma unroll
      for (int k = 0; k < C2; ++k) { lik[k] = uniform ? 1.0 : 0.0; llo[k] = 0.0; lexp[k] = 0; }
      int pcx = -1, pcy = -1;
      for (int64_t i = item.q0; i < item.q1; ++i) {
        const double qx = X[i], qy = Y[i];
        int cx, cy;
        cv_cell_of(s, qx, qy, cx, cy);
        if (cx != pcx || cy != pcy) {   // the same for every thread
          __syncthreads();              // the former ranges are no longer read
          cv_ranges(s, cs, cx, cx, cy, a.r_epan, 0, rb, pre, misc + 1);
          __syncthreads();
          pcx = cx;
          pcy = cy;
        }
        const int nr = misc[1];
        const int total = pre[nr], self = (int)i;
        int r = 0;
        CvRun run;
        for (int base = tid * kCvUnroll; base < total; base += nt * kCvUnroll) {
          int js[kCvUnroll];
          double xs[kCvUnroll], ys[kCvUnroll], ws[kCvUnroll];
#pragma unroll
          for (int u = 0; u < kCvUnroll; ++u) {
            const int k = base + u;
            js[u] = -1;
            if (k < total) {
              while (k >= pre[r + 1]) ++r;
              js[u] = rb[r] + (k - pre[r]);
            }
          }
#pragma unroll
          for (int u = 0; u < kCvUnroll; ++u) {
            if (js[u] >= 0) {
              xs[u] = X[js[u]];
              ys[u] = Y[js[u]];
              ws[u] = M[js[u]];
            }
          }
#pragma unroll
          for (int u = 0; u < kCvUnroll; ++u) {
            if (js[u] < 0) continue;
            const double dx = qx - xs[u], dy = qy - ys[u];
            const double ax = fabs(dx), ay = fabs(dy);
            if (ax >= hxmax || ay >= hymax || js[u] == self) continue;
            ++n_lik;
            const int p = cv_cell(ax, shx, a.nhx, slutx, a.lut_basex, a.lut_shift);
            const int q = cv_cell(ay, shy, a.nhy, sluty, a.lut_basey, a.lut_shift);
            const int c = p * kCvRow + q;
            const double ms = ws[u] * kCvFixLik;
            const double xt = ax * ihx[p], yt = ay * ihy[q];
            const double x2 = xt * xt, y2 = yt * yt;
            cv_run_add(H, run, c, ms, ms * x2, ms * y2, ms * x2 * y2);
          }
        }
        cv_run_flush(H, run);
        __syncthreads();
        // Fixed point -> FP64 moments sum m dx^k dy^l (k, l in {0, 2}); the histogram
        // is left cleared for the next query. mp = 0: {1, y^2}, 1: {x^2, x^2 y^2}.
        double u0[C1], u1[C1];
        {
          unsigned long long *h0 = H + mp * kCvHist + p1 * kCvRow + s1 * C1, *h1 = h0 + 2 * kCvHist;
          const bool on = p1 < a.nhx && s1 * C1 < a.nhy;
          const double hp2 = mp == 0 ? 1.0 : shx[p1] * shx[p1];
          double r0 = 0.0, r1 = 0.0;
#pragma unroll
          for (int k = 0; k < C1; ++k) {
            if (on) {
              const double hq = shy[s1 * C1 + k];
              r0 += (double)(long long)h0[k] * (1.0 / kCvFixLik) * hp2;
              r1 += s1 * C1 + k < a.nhy
                        ? (double)(long long)h1[k] * (1.0 / kCvFixLik) * hp2 * (hq * hq)
                        : 0.0;
              h0[k] = 0ull;
              h1[k] = 0ull;
            }
            u0[k] = r0;
            u1[k] = r1;
          }
          double *t = tot + (2 * mp * kCvSegs1 + s1) * kCvMaxH + p1;
          t[0] = r0;
          t[kCvSegs1 * kCvMaxH] = r1;
        }
        __syncthreads();
        {
          const double *t = tot + 2 * mp * kCvSegs1 * kCvMaxH + p1;
          double o0 = 0.0, o1 = 0.0;
          for (int sg = 0; sg < s1; ++sg) {
            o0 += t[sg * kCvMaxH];
            o1 += t[(kCvSegs1 + sg) * kCvMaxH];
          }
          double *dst = (mp == 0 ? PA : PB) + p1 * kCvRow + s1 * C1;
#pragma unroll
          for (int k = 0; k < C1; ++k)
            dst[k] = (o0 + u0[k]) - (o1 + u1[k]) * ihy2[s1 * C1 + k];
        }
        __syncthreads();
        double va[C2], vb[C2];
        {
          const double *ra = PA + s2 * C2 * kCvRow + b2, *rb2 = PB + s2 * C2 * kCvRow + b2;
          double r0 = 0.0, r1 = 0.0;
#pragma unroll
          for (int k = 0; k < C2; ++k) {
            r0 += ra[k * kCvRow];
            r1 += rb2[k * kCvRow];
            va[k] = r0;
            vb[k] = r1;
          }
          tot[s2 * kCvMaxH + b2] = r0;
          tot[(kCvSegs2 + s2) * kCvMaxH + b2] = r1;
        }
        __syncthreads();
        if (s2 * C2 < a.nhx && b2 < a.nhy) {
          double o0 = 0.0, o1 = 0.0;
          for (int sg = 0; sg < s2; ++sg) {
            o0 += tot[sg * kCvMaxH + b2];
            o1 += tot[(kCvSegs2 + sg) * kCvMaxH + b2];
          }
          const double wi = Wt[i];
          const double cb = 0.5625 * ihy[b2];   // KernelTraits.h:250-252
#pragma unroll
          for (int k = 0; k < C2; ++k) {
            const int ia = s2 * C2 + k;
            if (ia >= a.nhx) break;
            double S = (o0 + va[k]) - (o1 + vb[k]) * ihx2[ia];
            S = S > 0.0 ? S : 0.0;
            const double f = cb * ihx[ia] * S;
            llo[k] += wi * f;
            if (uniform) {
              const double t = lik[k] * f;   // normal or 0: see CvSet::uniform
              const int hi = __double2hiint(t);
              lexp[k] += (hi >> 20) - 1023;
              lik[k] = t > 0.0 ? __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(t))
                               : 0.0;
            } else {
              lik[k] += wi * log(f);
            }
          }
        }
      }
      if (uniform) {
        const double w = Wt[item.q0];
#pragma unroll
        for (int k = 0; k < C2; ++k)
          lik[k] = w * (log(lik[k]) + (double)lexp[k] * 0.69314718055994530942);
      }
      double *dst = a.epan_part + (int64_t)item.part * 2 * kCvCells;
#pragma unroll
      for (int k = 0; k < C2; ++k) {
        const int c = (s2 * C2 + k) * kCvMaxH + b2;
        dst[c] = lik[k];
        dst[kCvCells + c] = llo[k];
      }
      __syncthreads();
    } else {
      // ---- convolution pass, x-power group g, one block of queries of a run of
      // grid cells against every candidate j > i within 2 h_max (pairs are
      // symmetric, so each unordered pair is counted once and doubled) ------
      const int g = item.kind - 1;
      const int nq = (int)(item.q1 - item.q0);
      for (int c = tid; c < 4 * kCvHist; c += nt) H[c] = 0ull;
      for (int t = tid; t < nq; t += nt) {
        bqx[t] = X[item.q0 + t];
        bqy[t] = Y[item.q0 + t];
        bqw[t] = 2.0 * Wt[item.q0 + t] * kCvFixConv;
      }
      cv_ranges(s, cs, item.cx, item.cx1, item.cy, a.r_conv, item.q0 + 1, rb, pre, misc + 1);
      __syncthreads();
      const int nr = misc[1];
      const int total = pre[nr], q0 = (int)item.q0;
      const double hx2 = 2.0 * hxmax, hy2 = 2.0 * hymax;
      int r = 0;
      CvRun run;
      for (int k = tid; k < total; k += nt) {
        while (k >= pre[r + 1]) ++r;
        const int j = rb[r] + (k - pre[r]);
        const double xj = X[j], yj = Y[j], mj = M[j];
        const int lim = min(j - q0, nq);                        // queries i < j
        int t = lane % (lim > 0 ? lim : 1);                    // decorrelate lanes
        for (int s2 = 0; s2 < lim; ++s2) {
          const double ax = fabs(bqx[t] - xj), ay = fabs(bqy[t] - yj);
          const double v0 = bqw[t] * mj;
          if (++t == lim) t = 0;
          if (ax >= hx2 || ay >= hy2) continue;
          ++n_conv;
          const double hax = 0.5 * ax, hay = 0.5 * ay;
          const int p = cv_cell(hax, shx, a.nhx, slutx, a.lut_basex, a.lut_shift);
          const int q = cv_cell(hay, shy, a.nhy, sluty, a.lut_basey, a.lut_shift);
          const int c = p * kCvRow + q;
          const double xt = hax * ihx[p], yt = hay * ihy[q];   // in [0, 1)
          const double x2 = xt * xt;
          double xk = 1.0;
          if (g == 1) xk = x2;
          else if (g == 2) xk = x2 * xt;
          else if (g == 3) xk = x2 * x2 * xt;
          const double v = v0 * xk;
          const double y2 = yt * yt;
          cv_run_add(H, run, c, v, v * y2, v * y2 * yt, v * y2 * y2 * yt);
        }
      }
      cv_run_flush(H, run);
      __syncthreads();
      unsigned long long *dst = reinterpret_cast<unsigned long long *>(a.conv_hist) +
                                ((int64_t)item.set * 16 + 4 * g) * kCvCells;
      for (int e = tid; e < 4 * kCvCells; e += nt) {
        const int m4 = e / kCvCells, c = e % kCvCells;
        const unsigned long long v = H[m4 * kCvHist + (c / kCvMaxH) * kCvRow + c % kCvMaxH];
        if (v != 0ull) atomicAdd(&dst[e], v);
      }
      __syncthreads();
    }
  }
  if (a.pairs) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      n_lik += __shfl_xor_sync(0xffffffffu, n_lik, o);
      n_conv += __shfl_xor_sync(0xffffffffu, n_conv, o);
    }
    if (lane == 0) {
      atomicAdd(&a.pairs[0], n_lik);
      atomicAdd(&a.pairs[1], n_conv);
    }
  }
}

// Finalisation, first step, one block per (moment, set): the fixed-point
// convolution moment -> FP64 sum 2 w_i m_j |dx|^e_k |dy|^e_l (times (2 h_p)^e_k
// (2 h_q)^e_l), 2-D inclusive prefix, in place.
__device__ __forceinline__ double cv_power(double v, int group) {   // v^{0, 2, 3, 5}
  const double v2 = v * v;
  return group == 0 ? 1.0 : group == 1 ? v2 : group == 2 ? v2 * v : v2 * v2 * v;
}

__global__ void __launch_bounds__(kCvThreads) k_cv_prefix(CvArgs a) {
  __shared__ double m[kCvHist];
  const int kx = blockIdx.y / 4, ky = blockIdx.y % 4, tid = threadIdx.x;
  double *hist = a.conv_hist + ((int64_t)blockIdx.x * 16 + blockIdx.y) * kCvCells;
  const unsigned long long *ihist = reinterpret_cast<const unsigned long long *>(hist);
  for (int c = tid; c < kCvCells; c += kCvThreads) {
    const int p = c / kCvMaxH, q = c % kCvMaxH;
    const double sx = p < a.nhx ? cv_power(2.0 * a.hx[p], kx) : 0.0;
    const double sy = q < a.nhy ? cv_power(2.0 * a.hy[q], ky) : 0.0;
    m[p * kCvRow + q] = (double)(long long)ihist[c] / kCvFixConv * sx * sy;
  }
  __syncthreads();
  if (tid < kCvMaxH) {
    double run = 0.0;
#pragma unroll 8
    for (int q = 0; q < kCvMaxH; ++q) { run += m[tid * kCvRow + q]; m[tid * kCvRow + q] = run; }
  }
  __syncthreads();
  if (tid < kCvMaxH) {
    double run = 0.0;
#pragma unroll 8
    for (int p = 0; p < kCvMaxH; ++p) { run += m[p * kCvRow + tid]; m[p * kCvRow + tid] = run; }
  }
  __syncthreads();
  for (int c = tid; c < kCvCells; c += kCvThreads)
    hist[c] = m[(c / kCvMaxH) * kCvRow + c % kCvMaxH];
}

// Second step, one block per (row a of the grid, set): sq = C'_ab (T_ab + sum w m),
// lik and llo = sums over the set's likelihood items in a fixed order (kCvPartSplit
// runs of items per cell, then the runs), lsq = sq - 2 llo.
constexpr int kCvPartSplit = 16;
__global__ void __launch_bounds__(kCvThreads) k_cv_scores(CvArgs a, const int *part_begin,
                                                          const int *part_count, double *lik_out,
                                                          double *lsq_out) {
  __shared__ double s_lik[kCvPartSplit][kCvMaxH], s_llo[kCvPartSplit][kCvMaxH];
  static_assert(kCvPartSplit * kCvMaxH == kCvThreads, "one thread per (run, cell)");
  const int set = blockIdx.x, ia = blockIdx.y;
  const int ib = threadIdx.x % kCvMaxH, run = threadIdx.x / kCvMaxH;
  const int pb = part_begin[set], pc = part_count[set];
  const int per = (pc + kCvPartSplit - 1) / kCvPartSplit;
  const int c = ia * kCvMaxH + ib;
  double lik = 0.0, llo = 0.0;
#pragma unroll 4
  for (int k = run * per; k < min((run + 1) * per, pc); ++k) {
    const double *pp = a.epan_part + (int64_t)(pb + k) * 2 * kCvCells;
    lik += pp[c];
    llo += pp[kCvCells + c];
  }
  s_lik[run][ib] = lik;
  s_llo[run][ib] = llo;
  __syncthreads();
  if (run != 0 || ib >= a.nhy) return;
  for (int k = 1; k < kCvPartSplit; ++k) {
    lik += s_lik[k][ib];
    llo += s_llo[k][ib];
  }
  // P(u) = sum_k c_k u^{e_k}: (c, e) = (1, 0), (-5/4, 2), (5/8, 3), (-1/32, 5).
  const double ck[4] = {1.0, -1.25, 0.625, -0.03125};
  const double *hist = a.conv_hist + (int64_t)set * 16 * kCvCells;
  const double hxa = a.hx[ia], hyb = a.hy[ib];
  double T = 0.0;
  for (int kx = 0; kx < 4; ++kx) {
    const double fx = ck[kx] / cv_power(hxa, kx);
    for (int ky = 0; ky < 4; ++ky) {
      const double fy = ck[ky] / cv_power(hyb, ky);
      T += fx * fy * hist[(kx * 4 + ky) * kCvCells + c];
    }
  }
  const double sq = 0.36 / (hxa * hyb) * (T + a.sets[set].diag_wm);   // KernelTraits.h:349-351
  const int64_t o = ((int64_t)set * a.nhx + ia) * a.nhy + ib;
  lik_out[o] = lik;
  lsq_out[o] = sq - 2.0 * llo;
}

}  // namespace bbkde
