// Device code of the B200 direct kernel-density library.
//
// The pair sum f(q) = sum_r m_r U(q, x_r; h a_r) is the reference's eval_kernel
// (CudaDirectKde.h:126-173) re-designed for sm_100a:
//   * references are pre-packed once per (kernel, bandwidth) into float4 records
//     {x, y, m, s} (2-D) or {x, m, s, 0} (1-D) whose s folds -log2(e)/2/(h a)^2,
//     so a Gaussian pair costs 2 FADD + FMUL + FFMA + FMUL + MUFU.EX2 + FFMA;
//   * each thread owns QPT queries (register blocking) and reads every staged
//     reference record once from shared memory as a warp-wide broadcast;
//   * per-query partial sums run in FP32 over chunks of CHUNK references and are
//     folded into a Kahan-compensated FP32 pair (sum, comp); the block writes
//     (sum - comp) in FP64; reference segments are combined in FP64 in a fixed
//     order, so results do not depend on block scheduling;
//   * the FP64 variant follows the reference's CPU arithmetic (double exp).
#pragma once

#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

namespace bbkde {

// Device pair operators. kind of the packed record -> U(q, r).
enum Op : int {
  OP_GAUSS_ISO = 0,   // exp2(s * |d|^2)                       Gaussian, Gaussian conv
  OP_GAUSS_PROD = 1,  // exp2(sx dx^2 + sy dy^2)               product Gaussian, hx != hy
  OP_EPAN_ISO = 2,    // max(1 + s |d|^2, 0)                   Epanechnikov
  OP_EPAN_PROD = 3,   // max(1 + sx dx^2, 0) max(1 + sy dy^2, 0)
  OP_EPAN_CONV = 4    // prod_k c_k^3 (v_k^2 + 3 v_k + 1), v_k = |d_k| i_k, c_k = max(1-v_k,0)
};

constexpr int kChunk = 32;   // references per FP32 partial before the Kahan fold

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The Epanechnikov convolution (2 - u)^3 (u^2 + 6u + 4) / 32 on u = |d| / (h a) < 2
// (KernelTraits.h:338-342) in v = u / 2: (1 - v)^3 (v^2 + 3v + 1), the same value with
// every power of two folded into the record's scale 1 / |2 h a|.
__device__ __forceinline__ double epan_conv_d(double d, double inv) {
  const double v = fabs(d) * inv;
  const double c = 1.0 - v > 0.0 ? 1.0 - v : 0.0;
  return c * c * c * (v * v + 3.0 * v + 1.0);
}

// max(a b + c, 0) for a b + c <= 1: the FP32 pipe's saturating multiply-add.
__device__ __forceinline__ float fma_sat(float a, float b, float c) {
  float y;
  asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// 2^kExpBias e^x for x <= 0 (or NaN) on the FP64 pipe, 11 operations: Tang's table-driven
// method (ACM TOMS 15, 1989). x = k ln2 / 16 + r with k rounded by the 1.5 * 2^52 shift,
// ln2 / 16 in two terms, |r| <= ln2 / 32; e^x = 2^(k div 16) 2^(j/16) e^r, j = k mod 16.
// e^r is its Taylor polynomial of degree 7 with the last term economised on the
// Chebyshev polynomial T7 of that interval (relative error 8e-18). `tab` holds
// 2^(j/16), j < 16, with j << 16 taken from the high word and the bias added, so that
// adding k << 16 there leaves the exponent raised by k div 16; 16 doubles are all 32
// banks, so a warp's lookups never conflict.
// The bias keeps every value that the library's exp returns (denormals included) in the
// normal range, without a slow path; the sum is scaled back once per query. x is
// clamped at kExpClamp, where k = -16 (1023 + kExpBias) takes the exponent field of entry
// 0, 1.0, to zero: the value is 0, whatever the mass (the binade above it, 2^-1534, is a
// denormal of too few bits). The clamp works on the high word and lets a NaN of either
// sign pass (plus 0x80000 a negative quiet NaN wraps to a small number). A biased sum that
// overflows (2^512, before the scaling) is taken again without the bias
// (gauss_sum_unbiased).
constexpr int kExpBias = 512;
constexpr unsigned kExpClamp = 0xC0909FECu;   // high word of -1063.98: k = -24560
__device__ constexpr double kExpTab[16] = {
    1.0, 1.0442737824274138, 1.0905077326652577, 1.1387886347566916,
    1.189207115002721, 1.241857812073484, 1.2968395546510096, 1.3542555469368927,
    1.4142135623730951, 1.4768261459394993, 1.5422108254079407, 1.6104903319492543,
    1.681792830507429, 1.7562521603732995, 1.8340080864093424, 1.9152065613971474};

// Entry j of the shared-memory table of exp_neg.
__device__ __forceinline__ double exp_tab_entry(int j) {
  return __hiloint2double(__double2hiint(kExpTab[j]) - (j << 16) + (kExpBias << 20),
                          __double2loint(kExpTab[j]));
}

__device__ __forceinline__ double exp_neg(double x, const double *tab) {
  const unsigned h =
      __viaddmin_u32((unsigned)__double2hiint(x), 0x80000u, kExpClamp + 0x80000u) - 0x80000u;
  x = __hiloint2double((int)h, __double2loint(x));
  const double shift = 6755399441055744.0;   // 1.5 * 2^52
  const double t = fma(x, 23.083120654223414, shift);
  const int k = __double2loint(t);
  const double kd = t - shift;
  const double r = fma(kd, -1.4494042586539372e-18, fma(kd, -0.04332169878499658, x));
  double p = fma(1.0 / 720.0, r, 0.008333496247359863);
  p = fma(p, r, 0.041666666666666664);
  p = fma(p, r, 0.16666666662844765);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0000000000000022);
  const double b = tab[k & 15];
  const double s = __hiloint2double(__double2hiint(b) + (k << 16), __double2loint(b));
  return fma(s, r * p, s);
}

// U of N queries and one FP64 record (scales s and e, natural log for the Gaussians,
// whose values carry the factor 2^kExpBias).
template <int OP, int D, int N>
__device__ __forceinline__ void pair_u64(const double (&qx)[N], const double (&qy)[N], double x,
                                         double y, double s, double e, const double *tab,
                                         double (&u)[N]) {
  auto pos = [](double v) { return v > 0.0 ? v : 0.0; };
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double dx = qx[k] - x, dy = D == 2 ? qy[k] - y : 0.0;
    if (OP == OP_GAUSS_ISO || (OP == OP_GAUSS_PROD && D == 1))
      u[k] = exp_neg((D == 2 ? dx * dx + dy * dy : dx * dx) * s, tab);
    else if (OP == OP_GAUSS_PROD)
      u[k] = exp_neg(dx * dx * s + dy * dy * e, tab);
    else if (OP == OP_EPAN_ISO)
      u[k] = pos(1.0 + (D == 2 ? dx * dx + dy * dy : dx * dx) * s);
    else if (OP == OP_EPAN_PROD)
      u[k] = D == 2 ? pos(1.0 + dx * dx * s) * pos(1.0 + dy * dy * e) : pos(1.0 + dx * dx * s);
    else
      u[k] = D == 2 ? epan_conv_d(dx, s) * epan_conv_d(dy, e) : epan_conv_d(dx, s);
  }
}

__host__ __device__ constexpr bool op_has_extra(int op) {
  return op == OP_GAUSS_PROD || op == OP_EPAN_PROD || op == OP_EPAN_CONV;
}

// Arguments of one pair-sum launch. Reference records and query coordinates are
// indexed globally; the launch covers references [r_begin, r_end) split into
// gridDim.y segments of seg_len and queries [q_begin, q_begin + q_count).
struct SumArgs {
  const void *refs;        // float4* or double4*
  const void *extra;       // float* or double* (product kernels), may be null
  const void *qx;          // float* / double*
  const void *qy;          // float* / double* (unused for D = 1)
  int64_t r_begin, r_end;
  int64_t seg_len;
  int64_t q_begin, q_count;
  int exclude_self;        // self-evaluation: skip the pair r == q (same global index)
  double scale;            // multiplies each written partial
  double *out;             // [gridDim.y][q_count] partials (or final values)
  int *status;             // device error flag (0 = ok)
};

// ---------------------------------------------------------------------------
// FP32-compensated pair sum on packed f32x2 arithmetic (sm_100 FADD2 / FMUL2 /
// FFMA2): each instruction evaluates the same operation for two queries, so a
// Gaussian pair costs 3 packed-FP32 issue slots + 1 MUFU.EX2 instead of 6 + 1.
//
// Shared-memory records are pre-duplicated so every operand is a ready
// register pair: r0 = {-x, -x, -y, -y}, r1 = {m, m, s, s}, r2 = {e, e, _, _}
// (2-D) and r0 = {-x, -x, 0, 0}, r1 = {m, m, s, s} (1-D); q - x is evaluated as
// q + (-x), which IEEE defines identically.
// All operators.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

// 2^x on the FP32 pipe for two lanes, x <= 0 -- the alternative to MUFU.EX2 that
// lets the pair sum spread its exponentials over two pipes. Range reduction by the
// 1.5 * 2^23 shift (t = x + 1.5 * 2^23 holds n = round(x) in its low mantissa bits,
// f = x - n in [-1/2, 1/2] exactly), 2^f by a degree-5 polynomial (coefficients
// fitted for minimum relative error on [-1/2, 1/2] by Lawson's iteratively
// reweighted least squares: 7.5e-8 in exact arithmetic, 2.1e-7 evaluated with FP32
// FMAs), times 2^n, whose bits are t << 23 (the shift carries the exponent bias 127; its
// 0x4B400000 leaves the 32-bit word). As ex2.approx.ftz does, it gives 0 for x < -126 --
// 2^-127 is 0 here and the product flushes -- and NaN for NaN, so that a sum does not
// depend on which of its exponentials run here: with every far pair at 2^-125 instead, an
// isolated point's leave-one-out density was 1e-38 and its likelihood finite.
__device__ __forceinline__ float2 exp2_poly2(float2 x) {
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x.x));   // -127
  asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x.y));
  const float2 t = __fadd2_rn(x, f2(12583039.0f));   // 1.5 * 2^23 + 127
  const float2 n = __fadd2_rn(t, f2(-12583039.0f));
  const float2 f = __ffma2_rn(n, f2(-1.0f), x);
  float2 p = __ffma2_rn(f2(1.327644451521337e-3f), f, f2(9.67553723603487e-3f));
  p = __ffma2_rn(p, f, f2(5.550713464617729e-2f));
  p = __ffma2_rn(p, f, f2(2.4022120237350464e-1f));
  p = __ffma2_rn(p, f, f2(6.931469440460205e-1f));
  p = __ffma2_rn(p, f, f2(1.0000001192092896f));
  float2 u;
  asm("{\n\t.reg .b64 a, b, c;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\t"
      "mul.rn.ftz.f32x2 c, a, b;\n\tmov.b64 {%0, %1}, c;\n\t}"
      : "=f"(u.x), "=f"(u.y)
      : "f"(p.x), "f"(p.y), "f"(__uint_as_float(__float_as_uint(t.x) << 23)),
        "f"(__uint_as_float(__float_as_uint(t.y) << 23)));
  return u;
}

// max(1 + s d2, 0) for two lanes: two saturating multiply-adds (1 + s d2 <= 1) instead
// of a packed one and two maxima, which go to another pipe but cost issue slots.
__device__ __forceinline__ float2 epan_factor2(const float2 d2, const float2 s) {
  return make_float2(fma_sat(d2.x, s.x, 1.0f), fma_sat(d2.y, s.y, 1.0f));
}

// (1 - v)^3 (v^2 + 3v + 1) for two lanes, v = |d| inv, 0 beyond v = 1 (epan_conv_d).
__device__ __forceinline__ float2 epan_conv2(const float2 d, const float2 inv) {
  const float2 v = make_float2(fabsf(d.x) * inv.x, fabsf(d.y) * inv.y);
  const float2 c = make_float2(fma_sat(v.x, -1.0f, 1.0f), fma_sat(v.y, -1.0f, 1.0f));
  const float2 q = __ffma2_rn(v, __fadd2_rn(v, f2(3.0f)), f2(1.0f));
  return __fmul2_rn(__fmul2_rn(c, c), __fmul2_rn(c, q));
}

// U of two pairs, one per packed lane: coordinate differences from q + (-r), the
// reference's scales s (and sy for the product kernels).
template <int OP, int D, bool POLY = false>
__device__ __forceinline__ float2 pair_u2r(const float2 qx, const float2 qy, const float2 nrx,
                                           const float2 nry, const float2 s, const float2 sy) {
  float2 dx = __fadd2_rn(qx, nrx);
  if constexpr (D == 2) {
    float2 dy = __fadd2_rn(qy, nry);
    if constexpr (OP == OP_GAUSS_ISO) {
      float2 d2 = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
      float2 e = __fmul2_rn(d2, s);
      return POLY ? exp2_poly2(e) : make_float2(ex2_approx(e.x), ex2_approx(e.y));
    } else if constexpr (OP == OP_GAUSS_PROD) {
      float2 e = __ffma2_rn(__fmul2_rn(dy, dy), sy, __fmul2_rn(__fmul2_rn(dx, dx), s));
      return POLY ? exp2_poly2(e) : make_float2(ex2_approx(e.x), ex2_approx(e.y));
    } else if constexpr (OP == OP_EPAN_ISO) {
      float2 d2 = __ffma2_rn(dy, dy, __fmul2_rn(dx, dx));
      return epan_factor2(d2, s);
    } else if constexpr (OP == OP_EPAN_PROD) {
      return __fmul2_rn(epan_factor2(__fmul2_rn(dx, dx), s),
                        epan_factor2(__fmul2_rn(dy, dy), sy));
    } else {  // OP_EPAN_CONV
      return __fmul2_rn(epan_conv2(dx, s), epan_conv2(dy, sy));
    }
  } else {
    if constexpr (OP == OP_GAUSS_ISO || OP == OP_GAUSS_PROD) {
      float2 e = __fmul2_rn(__fmul2_rn(dx, dx), s);
      return POLY ? exp2_poly2(e) : make_float2(ex2_approx(e.x), ex2_approx(e.y));
    } else if constexpr (OP == OP_EPAN_ISO || OP == OP_EPAN_PROD) {
      return epan_factor2(__fmul2_rn(dx, dx), s);
    } else {
      return epan_conv2(dx, s);
    }
  }
}

// The same from a pre-duplicated shared-memory record (two queries, one reference).
template <int OP, int D, bool POLY = false>
__device__ __forceinline__ float2 pair_u2(const float2 qx, const float2 qy, const float4 &r0,
                                          const float4 &r1, const float4 &r2) {
  return pair_u2r<OP, D, POLY>(qx, qy, make_float2(r0.x, r0.y), make_float2(r0.z, r0.w),
                               make_float2(r1.z, r1.w), make_float2(r2.x, r2.y));
}

// One reference (shared-memory record j) against this thread's query pairs.
template <int OP, int D, int NP, bool POLY, bool EXT>
__device__ __forceinline__ void ref_pairs(const float4 *s_r0, const float4 *s_r1,
                                          const float4 *s_r2, int j, const float2 (&qx)[NP],
                                          const float2 (&qy)[NP], float2 (&acc)[NP]) {
  const float4 r0 = s_r0[j];
  const float4 r1 = s_r1[j];
  const float4 r2 = EXT ? s_r2[j] : r1;
  const float2 m = make_float2(r1.x, r1.y);
#pragma unroll
  for (int p = 0; p < NP; ++p)
    acc[p] = __ffma2_rn(m, pair_u2<OP, D, POLY>(qx[p], qy[p], r0, r1, r2), acc[p]);
}

// POLY_EVERY > 0: for the Gaussians, every POLY_EVERY-th reference of a chunk takes
// its exponentials from exp2_poly2 (FP32 pipe) instead of MUFU.EX2, so that both
// pipes share the work (1 in 8 balances them: the MUFU bound alone is 16 pairs
// per clock per SM, the joint bound ~18.3).
// kPoly3Of16: three of every 16 (the 1-D Gaussian, whose pair has 4 FP32 operations:
// joint bound 19.7 pairs per clock per SM, 18.3 with 1 in 8 or 1 in 4).
constexpr int kPoly3Of16 = 316;
template <int OP, int D, int QPT, int BLOCK, int TILE, int MINB, int POLY_EVERY = 0>
__global__ void __launch_bounds__(BLOCK, MINB) k_pair_sum_f32x2(SumArgs a) {
  static_assert(QPT % 2 == 0, "queries are processed in pairs");
  static_assert(POLY_EVERY == kPoly3Of16 || kChunk % (POLY_EVERY > 0 ? POLY_EVERY : 1) == 0,
                "poly stride divides a chunk");
  static_assert(TILE % kChunk == 0 && TILE % BLOCK == 0, "tile shape");
  constexpr int NP = QPT / 2;
  constexpr bool kExt = op_has_extra(OP) && D == 2;
  __shared__ float4 s_r0[TILE];
  __shared__ float4 s_r1[TILE];
  __shared__ float4 s_r2[kExt ? TILE : 1];

  const float4 *__restrict__ refs = static_cast<const float4 *>(a.refs);
  const float *__restrict__ ext = static_cast<const float *>(a.extra);
  const float *__restrict__ gqx = static_cast<const float *>(a.qx);
  const float *__restrict__ gqy = static_cast<const float *>(a.qy);

  const int tid = threadIdx.x;
  const int64_t lq0 = (int64_t)blockIdx.x * (BLOCK * QPT);
  const int64_t r_lo = a.r_begin + (int64_t)blockIdx.y * a.seg_len;
  const int64_t r_hi = min(r_lo + a.seg_len, a.r_end);

  // Query pair p of this thread = local queries (2p, 2p+1) -> slots k = 2p, 2p+1.
  float2 qx[NP], qy[NP];
  float sum[QPT], comp[QPT];
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    int64_t lq = lq0 + k * BLOCK + tid;
    bool ok = lq < a.q_count;
    float x = ok ? gqx[a.q_begin + lq] : 0.0f;
    float y = (ok && D == 2) ? gqy[a.q_begin + lq] : 0.0f;
    if (k & 1) { qx[k >> 1].y = x; qy[k >> 1].y = y; }
    else { qx[k >> 1].x = x; qy[k >> 1].x = y; }
    sum[k] = 0.0f;
    comp[k] = 0.0f;
  }
  const int64_t qg_lo = a.q_begin + lq0;
  const int64_t qg_hi = qg_lo + BLOCK * QPT;

  for (int64_t t0 = r_lo; t0 < r_hi; t0 += TILE) {
    __syncthreads();
#pragma unroll
    for (int i = tid; i < TILE; i += BLOCK) {
      int64_t r = t0 + i;
      float4 v = r < r_hi ? refs[r] : make_float4(0.f, 0.f, 0.f, 0.f);  // zero-mass padding
      if (D == 2) {
        s_r0[i] = make_float4(-v.x, -v.x, -v.y, -v.y);
        s_r1[i] = make_float4(v.z, v.z, v.w, v.w);
        if (kExt) {
          float e = r < r_hi ? ext[r] : 0.0f;
          s_r2[i] = make_float4(e, e, 0.f, 0.f);
        }
      } else {
        s_r0[i] = make_float4(-v.x, -v.x, 0.f, 0.f);
        s_r1[i] = make_float4(v.y, v.y, v.z, v.z);
      }
    }
    __syncthreads();
    const bool diag = a.exclude_self && t0 < qg_hi && qg_lo < t0 + TILE;
    for (int j0 = 0; j0 < TILE; j0 += kChunk) {
      float2 acc[NP];
#pragma unroll
      for (int p = 0; p < NP; ++p) acc[p] = f2(0.0f);
      if (!diag) {
        if constexpr (POLY_EVERY == 0 || !(OP == OP_GAUSS_ISO || OP == OP_GAUSS_PROD)) {
#pragma unroll 4
          for (int j = 0; j < kChunk; ++j)
            ref_pairs<OP, D, NP, false, kExt>(s_r0, s_r1, s_r2, j0 + j, qx, qy, acc);
        } else {
          // groups of G references, every S-th of them on the FP32 pipe
          constexpr int G = POLY_EVERY == kPoly3Of16 ? 16 : POLY_EVERY;
          constexpr int S = POLY_EVERY == kPoly3Of16 ? 5 : POLY_EVERY;
#pragma unroll 1
          for (int j = 0; j < kChunk; j += G) {
#pragma unroll
            for (int jj = 0; jj < G; ++jj) {
              if (jj % S == S - 1)
                ref_pairs<OP, D, NP, true, kExt>(s_r0, s_r1, s_r2, j0 + j + jj, qx, qy, acc);
              else
                ref_pairs<OP, D, NP, false, kExt>(s_r0, s_r1, s_r2, j0 + j + jj, qx, qy, acc);
            }
          }
        }
      } else {
        // Diagonal tile of a self-evaluation: zero the mass of the pair r == q.
        for (int j = 0; j < kChunk; ++j) {
          const float4 r0 = s_r0[j0 + j];
          const float4 r1 = s_r1[j0 + j];
          const float4 r2 = kExt ? s_r2[j0 + j] : r1;
          const int64_t rg = t0 + j0 + j;
#pragma unroll
          for (int p = 0; p < NP; ++p) {
            const int64_t q0 = qg_lo + (2 * p) * BLOCK + tid;
            const int64_t q1 = q0 + BLOCK;
            const float2 m = make_float2(rg == q0 ? 0.0f : r1.x, rg == q1 ? 0.0f : r1.y);
            acc[p] = __ffma2_rn(m, pair_u2<OP, D>(qx[p], qy[p], r0, r1, r2), acc[p]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < NP; ++p) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = 2 * p + h;
          const float v = h ? acc[p].y : acc[p].x;
          float y = v - comp[k];
          float t = sum[k] + y;
          comp[k] = (t - sum[k]) - y;
          sum[k] = t;
        }
      }
    }
  }

  double *out = a.out + (int64_t)blockIdx.y * a.q_count;
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    int64_t lq = lq0 + k * BLOCK + tid;
    if (lq < a.q_count) out[lq] = a.scale * ((double)sum[k] - (double)comp[k]);
  }
}

// ---------------------------------------------------------------------------
// FP32-compensated pair sum of small problems: a block owns 64 queries and its eight
// warps take the references of its segment in turn, 64 at a time (two references per
// packed operation, columns in shared memory), so that the sums of a segment meet in
// the block and few segments fill the chip. The warps' Kahan sums are added in FP64
// in warp order. The MUFU bound of 10,000 x 10,000 2-D Gaussian pairs is 21.5 us: 36 us
// measured (launch and ramp about 7), 48 in the 2,048-query blocks of shape 0, which
// left 148 SMs 200 blocks; 500 x 400: 8 us, 28 before. 128 queries, 4 warps or three
// resident blocks per SM measured the same or slower; at 2.5e9 pairs the 4-query
// shape of k_pair_sum_f32x2 is 6% faster.
// ---------------------------------------------------------------------------
constexpr int kSplitQueries = 64;
constexpr int kSplitWarps = 8;
constexpr int kSplitUnit = 64;                          // references a warp stages at a time
constexpr int kSplitStep = kSplitWarps * kSplitUnit;    // references of one turn of the block

template <int OP, int D>
__global__ void __launch_bounds__(32 * kSplitWarps, 4) k_pair_sum_split(SumArgs a) {
  constexpr int NW = kSplitWarps, U = kSplitUnit, QPT = kSplitQueries / 32, PER = U / 32;
  constexpr bool kExt = op_has_extra(OP) && D == 2;
  constexpr int COLS = (D == 2 ? 4 : 3) + (kExt ? 1 : 0);   // -x, m, s (, -y (, second s))
  static_assert(U % kChunk == 0, "whole chunks");
  __shared__ __align__(16) float s_ref[NW][COLS][U];
  __shared__ double s_sum[NW][kSplitQueries];

  const float4 *__restrict__ refs = static_cast<const float4 *>(a.refs);
  const float *__restrict__ ext = static_cast<const float *>(a.extra);
  const float *__restrict__ gqx = static_cast<const float *>(a.qx);
  const float *__restrict__ gqy = static_cast<const float *>(a.qy);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t lq0 = (int64_t)blockIdx.x * kSplitQueries;
  const int64_t qg0 = a.q_begin + lq0;
  const int64_t r_lo = a.r_begin + (int64_t)blockIdx.y * a.seg_len;
  const int64_t r_hi = min(r_lo + a.seg_len, a.r_end);

  float2 qx[QPT], qy[QPT];
  float sum[QPT], comp[QPT];
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    const bool ok = lq0 + 32 * k + lane < a.q_count;
    qx[k] = f2(ok ? gqx[qg0 + 32 * k + lane] : 0.0f);
    qy[k] = f2(ok && D == 2 ? gqy[qg0 + 32 * k + lane] : 0.0f);
    sum[k] = 0.0f;
    comp[k] = 0.0f;
  }
  float (&st)[COLS][U] = s_ref[warp];
  float4 rec[PER];
  float ex[PER];
  auto fetch = [&](int64_t t0) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int64_t r = t0 + 32 * u + lane;
      const bool in = r < r_hi;
      rec[u] = in ? __ldg(refs + r) : make_float4(0.f, 0.f, 0.f, 0.f);   // zero-mass padding
      if (kExt) ex[u] = in ? __ldg(ext + r) : 0.0f;
    }
  };
  int64_t t0 = r_lo + warp * U;
  if (t0 < r_hi) fetch(t0);
  for (; t0 < r_hi; t0 += kSplitStep) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int i = 32 * u + lane;
      st[0][i] = -rec[u].x;
      st[1][i] = D == 2 ? rec[u].z : rec[u].y;
      st[2][i] = D == 2 ? rec[u].w : rec[u].z;
      if (D == 2) st[3][i] = -rec[u].y;
      if (kExt) st[COLS - 1][i] = ex[u];
    }
    __syncwarp();
    if (t0 + kSplitStep < r_hi) fetch(t0 + kSplitStep);
    const bool diag = a.exclude_self && t0 < qg0 + kSplitQueries && qg0 < t0 + U;
#pragma unroll 1
    for (int j0 = 0; j0 < U; j0 += kChunk) {
      float2 acc[QPT];
#pragma unroll
      for (int k = 0; k < QPT; ++k) acc[k] = f2(0.0f);
      auto four = [&](int j, auto diagonal) {
        auto col = [&](int c) { return *reinterpret_cast<const float4 *>(&st[c][j0 + j]); };
        const float4 x4 = col(0), m4 = col(1), s4 = col(2);
        const float4 y4 = D == 2 ? col(D == 2 ? 3 : 0) : x4, e4 = kExt ? col(COLS - 1) : s4;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          auto half = [&](const float4 &v) {
            return h ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
          };
#pragma unroll
          for (int k = 0; k < QPT; ++k) {
            float2 m = half(m4);
            if (decltype(diagonal)::value) {   // zero the mass of the pair r == q
              const int64_t rel = qg0 + 32 * k + lane - (t0 + j0 + j + 2 * h);
              if (rel == 0) m.x = 0.0f;
              if (rel == 1) m.y = 0.0f;
            }
            acc[k] = __ffma2_rn(
                m, pair_u2r<OP, D>(qx[k], qy[k], half(x4), half(y4), half(s4), half(e4)),
                acc[k]);
          }
        }
      };
      if (!diag) {
#pragma unroll 4
        for (int j = 0; j < kChunk; j += 4) four(j, std::false_type{});
      } else {
#pragma unroll 1
        for (int j = 0; j < kChunk; j += 4) four(j, std::true_type{});
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
#pragma unroll
  for (int k = 0; k < QPT; ++k)
    s_sum[warp][32 * k + lane] = (double)sum[k] - (double)comp[k];
  __syncthreads();
  if (tid < kSplitQueries && lq0 + tid < a.q_count) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) v += s_sum[w][tid];
    a.out[(int64_t)blockIdx.y * a.q_count + lq0 + tid] = a.scale * v;
  }
}

// Gaussian sum of one query over [lo, hi) with the library's exp, for sums that overflow
// under exp_neg's bias (masses beyond 2^512, infinities) or are NaN; -1: no self pair.
template <int OP, int D>
__device__ __noinline__ double gauss_sum_unbiased(const double4 *refs, const double *ext,
                                                  int64_t lo, int64_t hi, double qx, double qy,
                                                  int64_t self) {
  double total = 0.0;
  for (int64_t r = lo; r < hi; ++r) {
    const double4 v = refs[r];
    const double dx = qx - v.x, dy = D == 2 ? qy - v.y : 0.0;
    const double m = D == 2 ? v.z : v.y, s = D == 2 ? v.w : v.z;
    const double x = D == 1 ? dx * dx * s
                     : OP == OP_GAUSS_ISO ? (dx * dx + dy * dy) * s
                                          : dx * dx * s + dy * dy * ext[r];
    total += (r == self ? 0.0 : m) * exp(x);
  }
  return total;
}

// ---------------------------------------------------------------------------
// FP64 pair sum (reference arithmetic). Thread t of block b owns the queries
// (b QPT + k) BLOCK + t. The FP64 pipe (64 lanes per clock per SM) is the bound: 18
// operations per product-Gaussian pair, 11 of them exp_neg; four queries per thread
// give it independent chains and share the record loads. 20,011 x 15,013 product-Gaussian
// pairs: 392 us (7.7e11 pairs/s, 74% of the bound), 703 us with the library's exp and one
// query per thread; 2 queries 422, 8 queries 398.
// ---------------------------------------------------------------------------
template <int OP, int D, int QPT, int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_pair_sum_f64(SumArgs a) {
  constexpr bool kExt = op_has_extra(OP) && D == 2;
  constexpr bool kGauss = OP == OP_GAUSS_ISO || OP == OP_GAUSS_PROD;
  __shared__ double2 s_a[BLOCK];                  // {x, y} / {x, m}
  __shared__ double2 s_b[BLOCK];                  // {m, s} / {s, -}
  __shared__ double s_ext[kExt ? BLOCK : 1];
  __shared__ double s_tab[16];
  const double4 *__restrict__ refs = static_cast<const double4 *>(a.refs);
  const double *__restrict__ ext = static_cast<const double *>(a.extra);
  const double *__restrict__ gqx = static_cast<const double *>(a.qx);
  const double *__restrict__ gqy = static_cast<const double *>(a.qy);

  const int tid = threadIdx.x;
  if (tid < 16) s_tab[tid] = exp_tab_entry(tid);
  const int64_t lq0 = (int64_t)blockIdx.x * (BLOCK * QPT);
  const int64_t qg_lo = a.q_begin + lq0, qg_hi = qg_lo + BLOCK * QPT;
  double qx[QPT], qy[QPT], total[QPT];
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    const int64_t lq = lq0 + k * BLOCK + tid;
    const bool ok = lq < a.q_count;
    qx[k] = ok ? gqx[a.q_begin + lq] : 0.0;
    qy[k] = ok && D == 2 ? gqy[a.q_begin + lq] : 0.0;
    total[k] = 0.0;
  }
  const int64_t r_lo = a.r_begin + (int64_t)blockIdx.y * a.seg_len;
  const int64_t r_hi = min(r_lo + a.seg_len, a.r_end);

  for (int64_t t0 = r_lo; t0 < r_hi; t0 += BLOCK) {
    __syncthreads();
    const int64_t r = t0 + tid;
    if (r < r_hi) {
      const double4 v = refs[r];
      s_a[tid] = make_double2(v.x, v.y);
      s_b[tid] = make_double2(v.z, v.w);
      if (kExt) s_ext[tid] = ext[r];
    }
    __syncthreads();
    const int n = (int)min(r_hi - t0, (int64_t)BLOCK);
    const bool diag = a.exclude_self && t0 < qg_hi && qg_lo < t0 + BLOCK;
    auto one = [&](int j, auto diagonal) {
      const double2 ra = s_a[j], rb = s_b[j];
      const double e = kExt ? s_ext[j] : 0.0;
      const double m = D == 2 ? rb.x : ra.y, s = D == 2 ? rb.y : rb.x;
      double u[QPT];
      pair_u64<OP, D>(qx, qy, ra.x, ra.y, s, e, s_tab, u);
#pragma unroll
      for (int k = 0; k < QPT; ++k) {
        const bool self = decltype(diagonal)::value && t0 + j == qg_lo + k * BLOCK + tid;
        total[k] += (self ? 0.0 : m) * u[k];
      }
    };
    if (!diag) {
#pragma unroll 2
      for (int j = 0; j < n; ++j) one(j, std::false_type{});
    } else {
#pragma unroll 1
      for (int j = 0; j < n; ++j) one(j, std::true_type{});
    }
  }
#pragma unroll
  for (int k = 0; k < QPT; ++k) {
    const int64_t lq = lq0 + k * BLOCK + tid;
    if (lq >= a.q_count) continue;
    double v = kGauss ? ldexp(total[k], -kExpBias) : total[k];
    if (kGauss && !isfinite(v))
      v = gauss_sum_unbiased<OP, D>(refs, ext, r_lo, r_hi, qx[k], qy[k],
                                    a.exclude_self ? a.q_begin + lq : -1);
    a.out[(int64_t)blockIdx.y * a.q_count + lq] = a.scale * v;
  }
}

// ---------------------------------------------------------------------------
// Packing: FP64 SoA point attributes -> per-kernel records.
// ---------------------------------------------------------------------------
struct PackArgs {
  const double *x, *y, *mass, *abw;   // SoA (y unused for D = 1; abw may be null)
  int64_t n;
  int op, dim;
  double c1, c2;      // scale numerators: s = c1 / (h1 a)^2 style (see host code)
  double h1, h2;      // bandwidths
};

// The record scales per operator, with a = abw_r:
//   GAUSS_*:  s = c1 / (h1 a)^2 (c1 = -log2(e)/2, or -log2(e)/4 for the
//             Gaussian convolution), e = c2 / (h2 a)^2
//   EPAN_ISO / EPAN_PROD: s = -1 / (h1 a)^2, e = -1 / (h2 a)^2
//   EPAN_CONV: s = 1 / |2 h1 a|, e = 1 / |2 h2 a| (the kernel is one of |u|)
__device__ __forceinline__ void pack_scales(const PackArgs &p, double a, double &s, double &e) {
  if (p.op == OP_EPAN_CONV) {
    s = 0.5 / fabs(p.h1 * a);
    e = 0.5 / fabs(p.h2 * a);
  } else {
    s = p.c1 / (p.h1 * p.h1 * a * a);
    e = p.c2 / (p.h2 * p.h2 * a * a);
  }
}

__global__ void k_pack_f32(PackArgs p, float4 *rec, float *ext) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  double a = p.abw ? p.abw[i] : 1.0;
  double s, e;
  pack_scales(p, a, s, e);
  float m = (float)(p.mass[i]);
  if (p.dim == 2)
    rec[i] = make_float4((float)p.x[i], (float)p.y[i], m, (float)s);
  else
    rec[i] = make_float4((float)p.x[i], m, (float)s, 0.0f);
  if (ext) ext[i] = (float)e;
}

__global__ void k_pack_f64(PackArgs p, double4 *rec, double *ext) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  double a = p.abw ? p.abw[i] : 1.0;
  double s, e;
  pack_scales(p, a, s, e);
  double m = p.mass[i];
  if (p.dim == 2)
    rec[i] = make_double4(p.x[i], p.y[i], m, s);
  else
    rec[i] = make_double4(p.x[i], m, s, 0.0);
  if (ext) ext[i] = e;
}

// FP32 copies of the coordinate columns (y null for D = 1).
__global__ void k_to_f32(const double *x, const double *y, float *fx, float *fy, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  fx[i] = (float)x[i];
  if (y) fy[i] = (float)y[i];
}

// One uploaded point set -> FP64 columns, in one pass: AoS coordinates (stride dim) are
// split, missing masses and local bandwidths are 1, a missing weight is the mass. A
// given column that is its own destination was copied there already. fx / fy (or null)
// get the FP32 coordinates.
struct IngestArgs {
  const double *coords, *mass, *abw, *weight;
  int dim;
  int64_t n;
  double *x, *y, *m, *a, *w;
  float *fx, *fy;
};
__global__ void k_ingest(IngestArgs p) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  const double x = p.coords[i * p.dim], y = p.dim == 2 ? p.coords[i * p.dim + 1] : 0.0;
  p.x[i] = x;
  if (p.dim == 2) p.y[i] = y;
  if (p.fx) {
    p.fx[i] = (float)x;
    if (p.dim == 2) p.fy[i] = (float)y;
  }
  const double m = p.mass ? p.mass[i] : 1.0;
  if (p.mass != p.m) p.m[i] = m;
  if (p.abw != p.a) p.a[i] = p.abw ? p.abw[i] : 1.0;
  if (p.weight != p.w) p.w[i] = p.weight ? p.weight[i] : m;
}

// ---------------------------------------------------------------------------
// Segment combination (+ optional weighted reductions), fixed order.
// ---------------------------------------------------------------------------
enum Epi : int { EPI_NONE = 0, EPI_W_LOG = 1, EPI_W_VALUE = 2 };

constexpr int kRedBlock = 256;

__device__ __forceinline__ double block_reduce_sum(double v, double *sm) {
  const int tid = threadIdx.x;
  sm[tid] = v;
  __syncthreads();
  for (int s = kRedBlock / 2; s > 0; s >>= 1) {
    if (tid < s) sm[tid] += sm[tid + s];
    __syncthreads();
  }
  double r = sm[0];
  __syncthreads();
  return r;
}

// out[q] = scale * sum_s partial[s][q]; with EPI_W_LOG / EPI_W_VALUE also writes
// block_sums[blockIdx.x] = sum over the block's q of w[q] * log(out[q]) / w[q] * out[q].
// G groups of kRedBlock / G threads take the segments in turn (group g the segments g,
// g + G, ...; their sums are added in group order): one thread per query left most SMs
// idle and its loads in one chain (10,000 queries x 40 segments 9.5 us, 8 groups 4).
template <int G>
__global__ void __launch_bounds__(kRedBlock)
k_combine(const double *partial, int nseg, int64_t q_count, double scale, double *out,
          int epi, const double *w, double *block_sums) {
  constexpr int QB = kRedBlock / G;
  __shared__ double sm[kRedBlock];
  const int g = threadIdx.x / QB;
  const int64_t q = (int64_t)blockIdx.x * QB + threadIdx.x % QB;
  double s = 0.0;
  if (q < q_count) {
#pragma unroll 4
    for (int i = g; i < nseg; i += G) s += partial[(int64_t)i * q_count + q];
  }
  if (G > 1) {
    sm[threadIdx.x] = s;
    __syncthreads();
    if (g == 0)
      for (int k = 1; k < G; ++k) s += sm[k * QB + threadIdx.x];
    __syncthreads();
  }
  double v = 0.0;
  if (g == 0 && q < q_count) {
    s *= scale;
    out[q] = s;
    if (epi == EPI_W_LOG) v = w[q] * log(s);
    else if (epi == EPI_W_VALUE) v = w[q] * s;
  }
  if (epi != EPI_NONE) {
    double b = block_reduce_sum(v, sm);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = b;
  }
}

// result[0] = sum of block_sums[0..n) in a fixed order.
__global__ void __launch_bounds__(kRedBlock)
k_sum_blocks(const double *block_sums, int64_t n, double *result) {
  __shared__ double sm[kRedBlock];
  double v = 0.0;
  for (int64_t i = threadIdx.x; i < n; i += kRedBlock) v += block_sums[i];
  double b = block_reduce_sum(v, sm);
  if (threadIdx.x == 0) result[0] = b;
}

// block_sums[b] = sum of v[i]^2 over block b's grid-stride share (fixed order).
__global__ void __launch_bounds__(kRedBlock)
k_sum_sq(const double *v, int64_t n, double *block_sums) {
  __shared__ double sm[kRedBlock];
  double s = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * kRedBlock + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * kRedBlock)
    s += v[i] * v[i];
  const double b = block_reduce_sum(s, sm);
  if (threadIdx.x == 0) block_sums[blockIdx.x] = b;
}

// Adaptive pilot finish (KernelDensityImpl.h:330-353):
// g = exp(logsum), abw_i = (pilot_i / g)^-alpha, mass_i = w_i abw_i^-dim.
__global__ void k_pilot_finalize(const double *pilot, const double *w, const double *logsum,
                                 double alpha, int dim, int64_t n, double *abw, double *mass,
                                 double *g_out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double g = exp(logsum[0]);
  if (i == 0 && g_out) g_out[0] = g;
  if (i >= n) return;
  double bw = pow(pilot[i] / g, -alpha);
  abw[i] = bw;
  mass[i] = w[i] * pow(bw, (double)-dim);
}

// sum_i w_i log(v_i) (mode 0) or sum_i w_i v_i (mode 1), v_i = f_i - sub_i C
// with sub_i rounded to FP32 (the mass the FP32 sums used; sub null: v_i = f_i),
// over n values in kWlogBlocks fixed slices: one FP64 partial per block
// (fixed-order tree within the block) -> part[blockIdx.x].
constexpr int kWlogBlocks = 256;
__global__ void k_wsum_partial(const double *f, const double *sub, double C, const double *w,
                               int mode, int64_t n, double *part) {
  __shared__ double s[256];
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = (int64_t)blockIdx.x * per, hi = lo + per < n ? lo + per : n;
  double acc = 0.0;
  for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const double v = sub ? f[i] - (double)(float)sub[i] * C : f[i];
    acc += w[i] * (mode == 0 ? log(v) : v);
  }
  s[threadIdx.x] = acc;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = s[0];
}

// out[0] = sum of part[0, m) (m <= 1024 = blockDim.x, a power of two), fixed order.
__global__ void k_sum_partials(const double *part, int m, double *out) {
  __shared__ double s[1024];
  s[threadIdx.x] = (int)threadIdx.x < m ? part[threadIdx.x] : 0.0;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = s[0];
}

__global__ void k_unadapt(const double *w, int64_t n, double *abw, double *mass) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  abw[i] = 1.0;
  mass[i] = w[i];
}

}  // namespace bbkde
