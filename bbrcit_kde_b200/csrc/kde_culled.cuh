// Culled direct sum: the pair sum over the reference tiles that can contribute,
// with a rigorous bound on the part that is skipped.
//
// References are sorted along a Hilbert curve (host code) and packed exactly as
// for k_pair_sum_f32x2; every run of consecutive sorted references (kCullUnit of
// them here, kRefTile in the factored grid kernels) is a "reference tile" with a
// bounding box, its widest kernel scale and its mass. The queries of a block
// (kCullQpb neighbours: consecutive queries in curve order, or an 8 x 8 piece of a
// grid tile) have a bounding box too. For a reference tile and a box, the largest
// value any pair can reach is, for the Gaussians, 2^e with
// e = log2(mass) + s_max * d_min^2 (d_min the distance between the boxes); for
// the Epanechnikov kernels the question is whether any pair lies inside the
// support.
//
// Every run of kGroupTiles consecutive tiles is a "tile group" with the union of
// their boxes, their widest scales and their summed mass: a group bound is at
// least the bound of each member tile, so each scan tests the groups first and
// only opens the members of groups that can matter (two-level scan; a skipped
// group counts as one skipped unit with its group bound).
//
// Gaussian blocks run three scans over the tiles:
//   1. M = the largest e over the block's box;
//   2. sum every tile with e >= M - cut (the near field);
//   3. with S = the smallest near-field sum of the block's queries and the allowance
//      A = max(rel * S, abs), also sum every remaining tile that reaches e >= T =
//      log2(A / n_tiles) - kFarMargin: all the tiles left out hold at most A / 64. (The
//      factored grid kernels count the bounds instead: cull_far_level, at most 9/32.)
// So the skipped part of every query q of the block is below A / 2 <= max(rel * S_q,
// abs) / 2:
// every culled sum is within rel of the full sum, or within abs of it, whichever
// is larger (plus the FP32 arithmetic error of the full sum). abs = 0 gives the
// purely relative bound. This is the reference's combined criterion: its tree
// stops refining a query once the bounds are within rel_err relative or
// abs_err absolute (KernelDensityImpl.h:1071-1095). Tiles whose largest pair exponent s_max d_min^2 is below -128
// are skipped without a bound: ex2.approx.ftz flushes every such kernel value
// to zero, so they add exactly nothing to the FP32 sum either. The per-block
// worst ratio (skipped bound / A) is written for the host to verify.
// Epanechnikov blocks sum every tile that intersects the support of the box;
// the skipped part is exactly zero.
//
// Summation: the warps of a block share its queries and take the listed tiles in
// turn (warp w the entries w, w + warps, ...); FP32 partial sums of kChunk pairs
// are folded into per-query Kahan accumulators of the warp, and the warps' sums
// are added in FP64 in warp order, so results are deterministic.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "kde_device.cuh"

namespace bbkde {

constexpr int kRefTile = 256;      // references per culling tile of the factored grid kernels
constexpr int kCullChunk = 1024;   // capacity of the per-batch list of needed tiles
constexpr int kGroupTiles = 16;    // tiles per tile group (two-level scan)

// Shape of the pair-form kernel: queries and warps per block, references per tile.
// The bound is MUFU (16 ex2 per clock per SM) on the listed pairs; what a shape
// decides is how many pairs are listed beyond the needed ones and whether a call of
// 10^4 queries fills the chip. Measured, 60,001 queries x 100,003 adaptive
// references at rel 1e-6, device ms (pairs listed): 64 queries x 64 references, 8
// warps 0.19 (3.3e8); 32 references 0.23 (2.7e8: staging per pair); 128
// references 0.22 (4.1e8); 128 queries 0.29 (3.7e8); 4 warps 0.23. The former
// shape, 1,024 queries in eight strips x 256 references, 128 threads: 2.86
// (1.35e9), on 59 blocks. 300,000 x 300,000 (h = 0.2, 1e-5): 4.23 ms, 3.4e12 pairs/s
// (74% of the bound); 17.7 ms before.
constexpr int kCullQpb = 64;
constexpr int kCullWarps = 8;
constexpr int kCullUnit = 64;
constexpr int kCullPiece = 8;      // a block's piece of a grid tile: 8 x 8 points

struct RefTile {
  float x0, x1, y0, y1;   // bounding box (y unused in 1-D)
  float sx, sy;           // widest (largest, i.e. least negative) scales
  float lm;               // log2 of 1.01 * sum |mass| (-inf for an empty tile)
  float pad;
};

// Where the queries of a block come from and where its results go.
//   mode 0: explicit FP32 coordinates: block b owns the queries perm[i], i in
//           [b * kCullQpb, (b + 1) * kCullQpb), of the count at qx/qy[p * stride];
//           the result of query p -> out[p].
//   mode 1: tiles of a regular grid: tile_list holds tiles of tile x tile points
//           (tiles numbered ty * ntx + tx); point (i, j) is at (gx0 + i gdx,
//           gy0 + j gdy) and its result goes to out[j * gnx + i]. A pair-form
//           block owns an 8 x 8 piece of a tile (block b: piece b % (tile / 8)^2 of
//           tile tile_list[b / (tile / 8)^2]), a factored block a whole tile.
struct CullQueries {
  int mode;
  const float *qx, *qy;
  int stride;
  const int *perm;
  int64_t count;
  const int *tile_list;
  int tile, ntx;
  int64_t gnx, gny;
  double gx0, gdx, gy0, gdy;
  double *out;
  double scale;
};

struct CullArgs {
  const float4 *refs;     // curve-sorted packed records
  const float *extra;     // second scale column of the product kernels (or null)
  const RefTile *tiles;
  const RefTile *groups;  // one per kGroupTiles consecutive tiles (bounds of the union)
  int n_tiles;
  int n_groups;
  int64_t n_ref;
  float cut;              // near-field width in log2 units
  double rel;             // bound of the skipped part relative to the block minimum
  double abs_n;           // absolute allowance of the skipped part (unnormalised units)
  CullQueries q;
  double *blk_bound;      // per block: worst (skipped bound / allowance)
  double *blk_smin;       // per block: smallest unnormalised sum of its queries
  int *blk_tiles;         // per block: reference tiles summed
  int *status;            // tensor-core form: set to 1 if a wait expired (or null)
};

__device__ __forceinline__ float grid_coord(double x0, double dx, int64_t i) {
  return (float)(x0 + (double)i * dx);
}

// Largest kernel value of tile t for any query in the box: log2 of it for the
// Gaussians (without the mass), the linear value for the Epanechnikov kernels.
template <int OP, int D>
__device__ __forceinline__ float tile_peak(const RefTile &t, float qx0, float qx1, float qy0,
                                           float qy1) {
  const float dx = fmaxf(0.f, fmaxf(t.x0 - qx1, qx0 - t.x1));
  const float dy = D == 2 ? fmaxf(0.f, fmaxf(t.y0 - qy1, qy0 - t.y1)) : 0.f;
  if (OP == OP_GAUSS_ISO) return t.sx * (dx * dx + dy * dy);
  if (OP == OP_GAUSS_PROD) return t.sx * dx * dx + t.sy * dy * dy;
  if (OP == OP_EPAN_ISO) return 1.f + t.sx * (dx * dx + dy * dy);
  return fminf(1.f + t.sx * dx * dx, 1.f + t.sy * dy * dy);   // both factors must be > 0
}

__host__ __device__ constexpr bool op_gauss(int op) {
  return op == OP_GAUSS_ISO || op == OP_GAUSS_PROD;
}

// Query lq of a pair-form block -> coordinates and output index; false if empty.
template <int D>
__device__ __forceinline__ bool cull_query(const CullQueries &q, int lq, float &x, float &y,
                                           int64_t &o) {
  if (q.mode == 0) {
    const int64_t i = (int64_t)blockIdx.x * kCullQpb + lq;
    if (i >= q.count) return false;
    o = q.perm[i];
    x = q.qx[o * q.stride];
    y = D == 2 ? q.qy[o * q.stride] : 0.f;
    return true;
  }
  const int pe = q.tile / kCullPiece, pieces = pe * pe;   // pieces per tile edge, per tile
  const int t = q.tile_list[blockIdx.x / pieces], p = blockIdx.x % pieces;
  const int64_t i = (int64_t)(t % q.ntx) * q.tile + (p % pe) * kCullPiece + lq % kCullPiece;
  const int64_t j = (int64_t)(t / q.ntx) * q.tile + (p / pe) * kCullPiece + lq / kCullPiece;
  if (i >= q.gnx || j >= q.gny) return false;
  x = grid_coord(q.gx0, q.gdx, i);
  y = grid_coord(q.gy0, q.gdy, j);
  o = j * q.gnx + i;
  return true;
}

// Exponent below which every FP32 kernel value is flushed to zero.
constexpr float kFlushExp = -128.0f;

// The groups that a block's scans go through: all of them (list null), or the listed ones.
struct CullGroups {
  const int *list;
  int n;
  __device__ __forceinline__ int operator[](int i) const { return list ? list[i] : i; }
};

// The groups that can reach the block, in order, in s_cand (up to kCullCand of them; all
// groups where there are more, or few enough for one test per thread). A block's three or
// four scans, with barriers every 64 groups, then go over its neighbourhood and not over
// every reference. 10^7 references, 10^6 queries, ms without / with the list: 1-D Gaussian
// h = 0.0005 23.7 / 4.0, h = 0.002 30.8 / 15.1, product Gaussian h = 0.005 16.0 / 2.6,
// Epanechnikov h = 0.01 2.9 / 1.5. can(group): false if no pair of it adds anything. A
// warp tests up to 1,024 consecutive groups per turn, so a turn of 8,192 groups has two
// barriers.
constexpr int kCullCand = 1024;
template <int BLOCK, class Can>
__device__ __forceinline__ CullGroups cull_candidates(const CullArgs &a, int *s_cand, int *s_wc,
                                                      Can can) {
  constexpr int NW = BLOCK / 32;
  const CullGroups all = {nullptr, a.n_groups};
  if (a.n_groups <= BLOCK) return all;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int n = 0;
  for (int r0 = 0; r0 < a.n_groups; r0 += 32 * BLOCK) {
    const int left = min(a.n_groups - r0, 32 * BLOCK), steps = (left + BLOCK - 1) / BLOCK;
    const int g0 = r0 + warp * 32 * steps;   // the warp's groups: 32 * steps from here
    unsigned mask = 0;                       // lane k: the groups g0 + 32 k + bit
#pragma unroll 4
    for (int k = 0; k < steps; ++k) {
      const int g = g0 + 32 * k + lane;
      const unsigned b = __ballot_sync(0xffffffffu, g < r0 + left && can(a.groups[g]));
      if (lane == k) mask = b;
    }
    const int mine = __popc(mask);
    int at = mine;   // inclusive scan over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, at, o);
      if (lane >= o) at += v;
    }
    if (lane == 31) s_wc[warp] = at;
    __syncthreads();
    int total = 0;
    at += n - mine;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      at += w < warp ? s_wc[w] : 0;
      total += s_wc[w];
    }
    n += total;
    if (n <= kCullCand)
      for (; mask; mask &= mask - 1) s_cand[at++] = g0 + 32 * lane + __ffs(mask) - 1;
    __syncthreads();
    if (n > kCullCand) return all;
  }
  return CullGroups{s_cand, n};
}

// Largest bound(t) over all tiles (block-wide; every thread gets the result).
// Thread-per-group: a group whose bound does not exceed the thread's running
// maximum cannot hold a tile that does, so only the others are opened.
template <int BLOCK, class Bound>
__device__ __forceinline__ float cull_max(const CullArgs &a, const CullGroups &groups,
                                          float *s_red, Bound bound) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float e = -INFINITY;
  for (int i = tid; i < groups.n; i += BLOCK) {
    const int gi = groups[i];
    if (bound(a.groups[gi]) > e) {
      const int t1 = min((gi + 1) * kGroupTiles, a.n_tiles);
      for (int ti = gi * kGroupTiles; ti < t1; ++ti) e = fmaxf(e, bound(a.tiles[ti]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e = fmaxf(e, __shfl_xor_sync(0xffffffffu, e, o));
  if (lane == 0) s_red[warp] = e;
  __syncthreads();
  e = -INFINITY;
#pragma unroll
  for (int w = 0; w < BLOCK / 32; ++w) e = fmaxf(e, s_red[w]);
  __syncthreads();
  return e;
}

// Groups tested per batch of cull_pass and the length of its tile list.
__host__ __device__ constexpr int cull_groups_per_batch(int block) {
  return block < kCullChunk / kGroupTiles ? block : kCullChunk / kGroupTiles;
}
__host__ __device__ constexpr int cull_list_len(int block) {
  return cull_groups_per_batch(block) * kGroupTiles;
}

// Block-wide ordered append: the threads with pred write value to dst[rank], rank
// = the number of such threads before them; returns how many wrote (every thread).
template <int BLOCK>
__device__ __forceinline__ int block_append(bool pred, int value, int *dst, int *s_wc) {
  constexpr int NW = BLOCK / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned b = __ballot_sync(0xffffffffu, pred);
  const int rank = __popc(b & ((1u << lane) - 1u));
  if (NW == 1) {
    if (pred) dst[rank] = value;
    __syncwarp();
    return __popc(b);
  }
  if (lane == 0) s_wc[warp] = __popc(b);
  __syncthreads();
  int base = 0, total = 0;
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    base += w < warp ? s_wc[w] : 0;
    total += s_wc[w];
  }
  if (pred) dst[base + rank] = value;
  __syncthreads();
  return total;
}

// One culling pass over the tiles, two levels. Each batch, thread tid < GR tests
// one group (group_needed(group, own); it also books the bound of a group it skips, if
// the group is its own); the needed groups are listed in order (s_glist, GR entries),
// and the block then tests their members in parallel (tile_needed), BLOCK at a time.
// The needed tiles of the batch are listed in ascending order in s_list[0, total)
// (capacity cull_list_len(BLOCK)) and handed to sum_list(total), which every thread
// calls. With parts > 1 (a divisor of kGroupTiles) the blocks of one tile share its
// references: part `part` tests the members ti with ti % parts == part of every needed
// group, and owns the groups gi with gi % parts == part, so that neighbouring tiles,
// which tend to be needed together, go to different parts. Returns the number of tiles
// listed.
template <int BLOCK, class GroupNeeded, class TileNeeded, class SumList>
__device__ __forceinline__ int cull_pass(const CullArgs &a, const CullGroups &groups, int *s_list,
                                         int *s_glist, int *s_wc, GroupNeeded group_needed,
                                         TileNeeded tile_needed, SumList sum_list, int part = 0,
                                         int parts = 1) {
  constexpr int GR = cull_groups_per_batch(BLOCK);
  const int tid = threadIdx.x;
  const int members = kGroupTiles / parts;   // of a group, tested here
  int summed = 0;
  for (int g0 = 0; g0 < groups.n; g0 += GR) {
    const bool in = tid < GR && g0 + tid < groups.n;
    const int gi = in ? groups[g0 + tid] : 0;
    const bool gneed = in && group_needed(a.groups[gi], gi % parts == part);
    const int ng = block_append<BLOCK>(gneed, gi, s_glist, s_wc);
    int total = 0;
    for (int m0 = 0; m0 < ng * members; m0 += BLOCK) {
      const int m = m0 + tid;
      int ti = -1;
      if (m < ng * members) {
        ti = s_glist[m / members] * kGroupTiles + (m % members) * parts + part;
        if (ti >= a.n_tiles || !tile_needed(a.tiles[ti])) ti = -1;
      }
      total += block_append<BLOCK>(ti >= 0, ti, s_list + total, s_wc);
    }
    if (total > 0) sum_list(total);
    summed += total;
    __syncthreads();
  }
  return summed;
}

// Far-field threshold of a block, relative to its allowance (log2): the tiles whose
// bound stays below it, all together, hold at most half of the allowance.
//   * Tiles below t0 = -log2(n_tiles) - 2 hold at most a quarter, however many.
//   * The tiles from t0 up to -2 are counted per bit; the threshold is the highest bit at
//     which the counted bounds below it (each taken at its bit's upper edge) still hold
//     at most kFarShare (with parts > 1 that share of it, each part for its own tiles).
//     A quarter would keep the guarantee too; what is left out is always missing on the
//     same side, so the nearer tiles, whose bounds are the sharper ones, are given less
//     (a 1-D likelihood to 1e-6: off by 4.7e-7 with a quarter, 6.8e-8 with this).
//   Together at most 1/4 + 1/32 = 9/32 of the allowance.
// A threshold of -log2(n_tiles) - 1 for every tile, which needs no count, charges each of
// them as much as the nearest one left out and lies two to three bits lower: the flagged
// tiles of a 4,096^2 pipeline at 1e-5 take 7.8 ms instead of 7.0.
// level(t): the largest bound of t over the block's slots relative to their allowances,
// -inf for a tile that is summed already or flushes to zero; a group's is at least its
// members'. Every thread calls it and gets the result.
constexpr int kFarBins = 32;
constexpr float kFarShare = 1.0f / 32.0f;
template <int BLOCK, class Level>
__device__ __forceinline__ float cull_far_level(const CullArgs &a, const CullGroups &groups,
                                                int *s_bins, float t0, Level level, int part = 0,
                                                int parts = 1) {
  const int tid = threadIdx.x;
  for (int b = tid; b < kFarBins; b += BLOCK) s_bins[b] = 0;
  __syncthreads();
  const int members = kGroupTiles / parts;
  for (int i = tid; i < groups.n; i += BLOCK) {
    const int gi = groups[i];
    if (!(level(a.groups[gi], true) >= t0)) continue;
    for (int m = 0; m < members; ++m) {
      const int ti = gi * kGroupTiles + m * parts + part;
      if (ti >= a.n_tiles) break;
      const float e = level(a.tiles[ti], false);
      if (e >= t0 && e < -2.0f) atomicAdd(&s_bins[min((int)(e - t0), kFarBins - 1)], 1);
    }
  }
  __syncthreads();
  float t = t0, held = 0.f;
  for (int b = 0; b < kFarBins && t < -2.0f; ++b) {
    held += (float)s_bins[b] * exp2f(t + 1.0f);
    if (held > kFarShare / (float)parts) break;
    t += 1.0f;
  }
  return fminf(t, -2.0f);
}

// Far threshold of the pair form: bits below the allowance's share of one tile. What is
// left out is always missing on the same side, so it adds up over a likelihood's points,
// and blocks of 64 queries have few tiles beyond the needed ones to make up for it. Error
// of a 1-D likelihood (51,330 points) and an adaptive density (123,398 references) to 1e-6:
// 5.5e-8 and 9.1e-8 with the counted threshold, 5.9e-9 and 7.7e-8 with 3 bits, 3.4e-9 and
// 7.7e-8 with 6 (256-reference tiles in blocks of 1,024 queries: 3.8e-9 and 7.7e-8); 0.93,
// 0.95 and 0.93 ms, 2.03, 2.13 and 2.23 ms.
constexpr float kFarMargin = 6.0f;

template <int OP, int D>
__global__ void __launch_bounds__(32 * kCullWarps, 4) k_pair_sum_culled(CullArgs a) {
  constexpr int BLOCK = 32 * kCullWarps;
  constexpr int NW = kCullWarps;
  constexpr int QPT = kCullQpb / 32;       // queries per thread: 32 k + lane
  constexpr int U = kCullUnit;
  constexpr int PER = U / 32;              // references a lane stages per tile
  constexpr bool kExt = op_has_extra(OP) && D == 2;
  constexpr bool kGauss = op_gauss(OP);
  constexpr int COLS = (D == 2 ? 4 : 3) + (kExt ? 1 : 0);   // -x, m, s (, -y (, second s))
  static_assert(U % kChunk == 0 && kCullQpb == kCullPiece * kCullPiece, "shape");
  __shared__ __align__(16) float s_ref[NW][COLS][U];
  __shared__ int s_list[cull_list_len(BLOCK)];
  __shared__ int s_glist[cull_groups_per_batch(BLOCK)];
  __shared__ int s_cand[kCullCand];
  __shared__ int s_wc[NW];
  __shared__ float s_red[NW];
  __shared__ double s_sum[NW][kCullQpb];
  __shared__ double s_min[kCullQpb / 32];
  __shared__ double s_skip[NW];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float2 qx[QPT], qy[QPT];   // (x, x), (y, y): two references per packed operation
  float sum[QPT], comp[QPT];
  float qx0 = 3e38f, qx1 = -3e38f, qy0 = 3e38f, qy1 = -3e38f;
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    float x = 0.f, y = 0.f;
    int64_t o = 0;
    if (cull_query<D>(a.q, 32 * k + lane, x, y, o)) {
      qx0 = fminf(qx0, x); qx1 = fmaxf(qx1, x);
      qy0 = fminf(qy0, y); qy1 = fmaxf(qy1, y);
    }
    qx[k] = f2(x);
    qy[k] = f2(y);
    sum[k] = 0.f;
    comp[k] = 0.f;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    qx0 = fminf(qx0, __shfl_xor_sync(0xffffffffu, qx0, o));
    qx1 = fmaxf(qx1, __shfl_xor_sync(0xffffffffu, qx1, o));
    qy0 = fminf(qy0, __shfl_xor_sync(0xffffffffu, qy0, o));
    qy1 = fmaxf(qy1, __shfl_xor_sync(0xffffffffu, qy1, o));
  }

  // No box: a piece outside the grid, or no query is a number. Nothing is summed.
  const bool boxed = qx0 <= qx1 && qy0 <= qy1;

  CullGroups groups = {nullptr, 0};
  if (boxed)   // beyond the support, or all flushed to zero: nothing to sum and no bound
    groups = cull_candidates<BLOCK>(a, s_cand, s_wc, [&](const RefTile &g) {
      const float pb = tile_peak<OP, D>(g, qx0, qx1, qy0, qy1);
      return kGauss ? !(pb < kFlushExp) : pb > 0.f;
    });

  // Scan 1 (Gaussians): largest tile bound over the block's box.
  float e_max = -INFINITY;
  if (kGauss && boxed)
    e_max = cull_max<BLOCK>(a, groups, s_red, [&](const RefTile &t) {
      return t.lm + tile_peak<OP, D>(t, qx0, qx1, qy0, qy1);
    });
  const float t_a = e_max - a.cut;

  // Skipped bound relative to the threshold: 2^(e - T) < 1 per skipped unit (terms below
  // 2^-126 of the threshold flush; they are negligible). ex2.approx errs by ~2^-22
  // relative, inside the 1% mass slack.
  float skipped = 0.f, la = 0.f;   // log2 A
  const float tn = -log2f((float)a.n_tiles) - kFarMargin;   // threshold relative to A
  int summed = 0;

  // Is tile (or group) t needed? phase 0: Epanechnikov (support of the box);
  // phase 1: Gaussian near field; phase 2: Gaussian far field (a unit that is not
  // needed books its bound). For a group the near-field test of phase 2 is left
  // out: a skipped group may hold tiles summed in phase 1, whose bound is then
  // booked as well (an over-estimate).
  auto needed = [&](const RefTile &t, int phase, bool group) -> bool {
    const float pb = tile_peak<OP, D>(t, qx0, qx1, qy0, qy1);
    if (!kGauss) return pb > 0.f;
    if (pb < kFlushExp) return false;   // every pair flushes to zero
    const float e = t.lm + pb;
    const bool near = e >= t_a;
    if (phase == 1) return near;
    if (near && !group) return false;   // already summed
    if (e - la >= tn) return true;
    skipped += ex2_approx(e - la - tn);
    return false;
  };

  // Sum the listed tiles: each warp stages its next tile's records while it sums
  // the current one.
  float (&st)[COLS][U] = s_ref[warp];
  float4 rec[PER];
  float ext[PER];
  auto fetch = [&](int unit) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int64_t rr = (int64_t)unit * U + 32 * u + lane;
      const bool in = rr < a.n_ref;
      rec[u] = in ? __ldg(a.refs + rr) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (kExt) ext[u] = in ? __ldg(a.extra + rr) : 0.f;
    }
  };
  auto sum_list = [&](int total) {
    if (warp < total) fetch(s_list[warp]);
    for (int li = warp; li < total; li += NW) {
#pragma unroll
      for (int u = 0; u < PER; ++u) {
        const int i = 32 * u + lane;
        st[0][i] = -rec[u].x;
        st[1][i] = D == 2 ? rec[u].z : rec[u].y;
        st[2][i] = D == 2 ? rec[u].w : rec[u].z;
        if (D == 2) st[3][i] = -rec[u].y;
        if (kExt) st[COLS - 1][i] = ext[u];
      }
      __syncwarp();
      if (li + NW < total) fetch(s_list[li + NW]);
#pragma unroll 1
      for (int j0 = 0; j0 < U; j0 += kChunk) {
        float2 acc[QPT];
#pragma unroll
        for (int k = 0; k < QPT; ++k) acc[k] = f2(0.0f);
#pragma unroll 4
        for (int j = 0; j < kChunk; j += 4) {
          auto col = [&](int cidx) {
            return *reinterpret_cast<const float4 *>(&st[cidx][j0 + j]);
          };
          const float4 x4 = col(0), m4 = col(1), s4 = col(2);
          const float4 y4 = D == 2 ? col(D == 2 ? 3 : 0) : x4, e4 = kExt ? col(COLS - 1) : s4;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            auto half = [&](const float4 &v) {
              return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
            };
            const float2 m = half(m4);
#pragma unroll
            for (int k = 0; k < QPT; ++k)
              acc[k] = __ffma2_rn(
                  m, pair_u2r<OP, D>(qx[k], qy[k], half(x4), half(y4), half(s4), half(e4)),
                  acc[k]);
          }
        }
        // Kahan fold of the chunk partial (even + odd references).
#pragma unroll
        for (int k = 0; k < QPT; ++k) {
          const float y = (acc[k].x + acc[k].y) - comp[k];
          const float t = sum[k] + y;
          comp[k] = (t - sum[k]) - y;
          sum[k] = t;
        }
      }
      __syncwarp();
    }
  };

  auto pass = [&](int phase) {
    summed += cull_pass<BLOCK>(
        a, groups, s_list, s_glist, s_wc,
        [&](const RefTile &g, bool) { return needed(g, phase, true); },
        [&](const RefTile &t) { return needed(t, phase, false); }, sum_list);
  };
  // The warps' sums of query tid (tid < kCullQpb) added in warp order.
  auto total_of = [&]() {
#pragma unroll
    for (int k = 0; k < QPT; ++k)
      s_sum[warp][32 * k + lane] = (double)sum[k] - (double)comp[k];
    __syncthreads();
    double v = 0.0;
    if (tid < kCullQpb) {
#pragma unroll
      for (int w = 0; w < NW; ++w) v += s_sum[w][tid];
    }
    return v;
  };

  float fx = 0.f, fy = 0.f;   // query tid, its output
  int64_t fo = 0;
  const bool mine = tid < kCullQpb && cull_query<D>(a.q, tid, fx, fy, fo);
  double smin = 0.0, ratio = 0.0;
  if (kGauss && boxed) {
    pass(1);   // scan 2: near field
    double m = total_of();
    if (tid < kCullQpb) {   // whole warps
      if (!mine) m = INFINITY;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) s_min[warp] = m;
    }
    __syncthreads();
    smin = INFINITY;
#pragma unroll
    for (int w = 0; w < kCullQpb / 32; ++w) smin = fmin(smin, s_min[w]);
    // allowance 0 (smin <= 0 and no abs): every tile that does not flush to zero
    const double allow = fmax(a.rel * smin, a.abs_n);
    la = allow > 0.0 ? (float)log2(allow) : -INFINITY;
    pass(2);   // scan 3: far field, bound of the rest
    // Bound of the skipped part (fixed-order reduction) over the allowance.
    double sk = skipped;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sk += __shfl_xor_sync(0xffffffffu, sk, o);
    if (lane == 0) s_skip[warp] = sk;
    __syncthreads();
    double b = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) b += s_skip[w];
    if (b > 0.0) ratio = b * exp2((double)tn);
  } else if (boxed) {
    pass(0);
  }
  const double v = total_of();
  if (tid == 0) {
    a.blk_bound[blockIdx.x] = ratio;
    a.blk_smin[blockIdx.x] = smin;
    a.blk_tiles[blockIdx.x] = summed;
  }
  // A query that is not a number reaches no tile; its Gaussian sum is not a number.
  if (mine) a.q.out[fo] = kGauss && (fx != fx || fy != fy) ? (double)NAN : a.q.scale * v;
}

// ---------------------------------------------------------------------------
// Building the sorted references and their tiles.
// ---------------------------------------------------------------------------

// Order-preserving map of a float to an unsigned integer (for atomic min/max).
__device__ __forceinline__ unsigned ordered_bits(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_ordered(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Bounding box of n points x[i * stride], y[i * stride] -> box[0..3] as ordered
// bits {min x, min y, max x, max y}; box must start as {~0, ~0, 0, 0}.
__global__ void k_bbox(const float *x, const float *y, int stride, int64_t n, unsigned *box) {
  float x0 = 3e38f, x1 = -3e38f, y0 = 3e38f, y1 = -3e38f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float xv = x[i * stride], yv = y ? y[i * stride] : 0.f;
    x0 = fminf(x0, xv); x1 = fmaxf(x1, xv);
    y0 = fminf(y0, yv); y1 = fmaxf(y1, yv);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&box[0], ordered_bits(x0));
    atomicMin(&box[1], ordered_bits(y0));
    atomicMax(&box[2], ordered_bits(x1));
    atomicMax(&box[3], ordered_bits(y1));
  }
}

// Position of (x, y), 16 bits each, along a Hilbert curve: per level the quadrant
// (rx, ry) is digit (3 rx) ^ ry, and the lower levels are reflected / transposed
// into the quadrant's own orientation. Unlike Morton order it has no jumps, so a
// run of consecutive points never spans two distant quadrants.
__device__ __forceinline__ unsigned hilbert16(unsigned x, unsigned y) {
  unsigned key = 0;
#pragma unroll
  for (int b = 15; b >= 0; --b) {
    const unsigned rx = (x >> b) & 1u, ry = (y >> b) & 1u;
    key = (key << 2) | ((3u * rx) ^ ry);
    if (ry == 0u) {
      if (rx) { x = ~x; y = ~y; }   // only the bits below b are read from here on
      const unsigned t = x;
      x = y;
      y = t;
    }
  }
  return key;
}

__device__ __forceinline__ unsigned quantize(float v, float lo, float hi, float levels) {
  const float span = hi - lo;
  const float u = span > 0.f ? (v - lo) / span : 0.f;
  return (unsigned)fminf(fmaxf(u * levels, 0.f), levels - 1.f);
}

// Curve key (2-D: Hilbert order of 16 bits per axis; 1-D: 32-bit quantised x) and
// the identity permutation.
__global__ void k_curve_keys(const float *x, const float *y, int stride, int64_t n,
                         const unsigned *box, unsigned *keys, int *idx) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float xlo = from_ordered(box[0]), ylo = from_ordered(box[1]);
  const float xhi = from_ordered(box[2]), yhi = from_ordered(box[3]);
  unsigned key;
  if (y) {
    key = hilbert16(quantize(x[i * stride], xlo, xhi, 65536.f),
                    quantize(y[i * stride], ylo, yhi, 65536.f));
  } else {
    const float span = xhi - xlo;
    const double u = span > 0.f ? ((double)x[i * stride] - xlo) / span : 0.0;
    key = (unsigned)fmin(fmax(u * 4294967296.0, 0.0), 4294967295.0);
  }
  keys[i] = key;
  idx[i] = (int)i;
}

__global__ void k_gather_rec(const float4 *rec, const float *ext, const int *perm, int64_t n,
                             float4 *rec_out, float *ext_out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int p = perm[i];
  rec_out[i] = rec[p];
  if (ext) ext_out[i] = ext[p];
}

// One warp per tile of `size` sorted records.
template <int D>
__global__ void k_ref_tiles(const float4 *rec, const float *ext, int64_t n, int size,
                            int n_tiles, RefTile *tiles) {
  const int t = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (t >= n_tiles) return;
  float x0 = 3e38f, x1 = -3e38f, y0 = 3e38f, y1 = -3e38f, sx = -3e38f, sy = -3e38f;
  double m = 0.0;
  for (int i = lane; i < size; i += 32) {
    const int64_t r = (int64_t)t * size + i;
    if (r >= n) break;
    const float4 v = rec[r];
    const float px = v.x, py = D == 2 ? v.y : 0.f;
    const float pm = D == 2 ? v.z : v.y, ps = D == 2 ? v.w : v.z;
    x0 = fminf(x0, px); x1 = fmaxf(x1, px);
    y0 = fminf(y0, py); y1 = fmaxf(y1, py);
    sx = fmaxf(sx, ps);
    sy = fmaxf(sy, ext ? ext[r] : ps);
    m += fabs((double)pm);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
    sx = fmaxf(sx, __shfl_xor_sync(0xffffffffu, sx, o));
    sy = fmaxf(sy, __shfl_xor_sync(0xffffffffu, sy, o));
    m += __shfl_xor_sync(0xffffffffu, m, o);
  }
  if (lane == 0) {
    RefTile rt;
    rt.x0 = x0; rt.x1 = x1; rt.y0 = y0; rt.y1 = y1;
    rt.sx = sx; rt.sy = sy;
    rt.lm = m > 0.0 ? (float)log2(1.01 * m) : -INFINITY;
    rt.pad = 0.f;
    tiles[t] = rt;
  }
}

// kGroupTiles lanes per group of as many consecutive tiles: union of the boxes,
// widest scales, log2 of the summed (already 1%-padded) masses, rounded up.
__global__ void k_ref_groups(const RefTile *tiles, int n_tiles, int n_groups,
                             RefTile *groups) {
  static_assert(kGroupTiles == 16, "half a warp per group");
  const int ti = blockIdx.x * blockDim.x + threadIdx.x;   // group ti / 16
  RefTile u;
  u.x0 = 3e38f; u.x1 = -3e38f; u.y0 = 3e38f; u.y1 = -3e38f;
  u.sx = -3e38f; u.sy = -3e38f;
  double m = 0.0;
  if (ti < n_tiles) {
    u = tiles[ti];
    if (u.lm > -INFINITY) m = exp2((double)u.lm);
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    u.x0 = fminf(u.x0, __shfl_xor_sync(0xffffffffu, u.x0, o));
    u.x1 = fmaxf(u.x1, __shfl_xor_sync(0xffffffffu, u.x1, o));
    u.y0 = fminf(u.y0, __shfl_xor_sync(0xffffffffu, u.y0, o));
    u.y1 = fmaxf(u.y1, __shfl_xor_sync(0xffffffffu, u.y1, o));
    u.sx = fmaxf(u.sx, __shfl_xor_sync(0xffffffffu, u.sx, o));
    u.sy = fmaxf(u.sy, __shfl_xor_sync(0xffffffffu, u.sy, o));
    m += __shfl_xor_sync(0xffffffffu, m, o);
  }
  if (ti % kGroupTiles == 0 && ti / kGroupTiles < n_groups) {
    u.lm = m > 0.0 ? nextafterf((float)log2(m), INFINITY) : -INFINITY;
    u.pad = 0.f;
    groups[ti / kGroupTiles] = u;
  }
}

// Largest skipped-bound ratio over the blocks, summed tiles.
__global__ void k_cull_stats(const double *bound, const double *smin, const int *tiles,
                             int nblk, double *out2) {
  __shared__ double s_r[1024], s_t[1024];   // blockDim.x <= 1024, a power of two
  double r = 0.0, tsum = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    r = fmax(r, bound[b]);
    tsum += (double)tiles[b];
  }
  s_r[threadIdx.x] = r;
  s_t[threadIdx.x] = tsum;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      s_r[threadIdx.x] = fmax(s_r[threadIdx.x], s_r[threadIdx.x + s]);
      s_t[threadIdx.x] += s_t[threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out2[0] = s_r[0];
    out2[1] = s_t[0];
  }
}

}  // namespace bbkde
