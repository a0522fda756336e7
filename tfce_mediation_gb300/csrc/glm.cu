// Mass-univariate OLS t-statistics for many designs against one data matrix:
// the GB300 replacement of tval_int / se_of_slope / calc_beta_se
// (tfce_mediation/cynumstats.pyx:28-29, 47-74) and of the per-permutation
// design loop of tfce_mediation/tmanalysis/vertex_tfce_multiple_regression_randomise.py:90-107.
//
// One CTA owns a tile of kTileV vertex columns of Y (all n subjects, held in
// shared memory) and runs every design of the batch over it, so Y is read
// from HBM once per batch.  For design g and column v:
//   beta_j = sum_s pinv[g][j][s] * y[s][v]                (cy_lin_lstsqr_mat)
//   rss    = sum_s (y[s][v] - sum_j X[g][s][j] beta_j)^2  (residuals, never Y'Y)
//   t_j    = beta_j / sqrt(rss / dof_g * invdiag[g][j])   (se_of_slope, tval_int)
// in FP32 with FMA accumulation; the k x k inverse and pseudoinverse are formed
// in FP64, on the device for an engine's batches (glm_design.cu), else on the
// host.
//
// Also: the indirect-effect (Sobel/Aroian/Goodman) combination of two path t
// maps (tfce_mediation/pyfunc.py:146-161).
#include <algorithm>

#include <math_constants.h>

#include "common.cuh"

namespace tfgb {

constexpr int kGlmThreads = 256;
constexpr int kColsPerThread = 4;

// Y tile [n][TV] in shared memory; each thread computes 4 adjacent columns of
// one design; TV/4 threads per design; kGlmThreads/(TV/4) designs in flight.
enum GlmWhat : int32_t { kWhatT = 0, kWhatBeta = 1, kWhatSE = 2, kWhatResid = 3, kWhatF = 4, kWhatRSS = 5 };

template <int KMAX, int TV>
__global__ void __launch_bounds__(kGlmThreads) glm_tstat_kernel(
    const float* __restrict__ Y, int64_t ldy, int32_t n, int64_t V,
    const float* __restrict__ pinv, const float* __restrict__ X,
    const float* __restrict__ invdiag, const float* __restrict__ dof, int32_t G,
    const int32_t* __restrict__ coef, int32_t n_coef, float* __restrict__ t_out, int64_t ldt,
    int32_t what) {
  extern __shared__ float4 smem4[];
  float* ys = reinterpret_cast<float*>(smem4);
  constexpr int kThreadsPerDesign = TV / kColsPerThread;
  constexpr int kDesignsInFlight = kGlmThreads / kThreadsPerDesign;
  const int64_t vbase = (int64_t)blockIdx.x * TV;

  // stage the tile (zero-filled past V)
  for (int i = threadIdx.x; i < n * TV; i += kGlmThreads) {
    const int s = i / TV, c = i % TV;
    const int64_t v = vbase + c;
    ys[i] = (v < V) ? Y[(int64_t)s * ldy + v] : 0.0f;
  }
  __syncthreads();

  const int lane_d = threadIdx.x % kThreadsPerDesign;
  const int slot = threadIdx.x / kThreadsPerDesign;
  const int c0 = lane_d * kColsPerThread;
  const float4* yrow = reinterpret_cast<const float4*>(ys) + lane_d;  // stride TV/4 per subject
  // A design's rows are read four subjects a load where their rows are aligned
  // (n a multiple of 4): one load a weight kept the load pipe busier than the
  // FMAs (32 designs of 60 x 3 over 76k vertices: 104 us, so 83).
  const bool aligned = n % 4 == 0 && ((reinterpret_cast<uintptr_t>(pinv) | reinterpret_cast<uintptr_t>(X)) & 15) == 0;
  const int n4 = aligned ? n : 0;

  for (int g = slot; g < G; g += kDesignsInFlight) {
    const float* pg = pinv + (int64_t)g * KMAX * n;
    const float* xg = X + (int64_t)g * n * KMAX;
    float b[KMAX][kColsPerThread];
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
#pragma unroll
      for (int c = 0; c < kColsPerThread; ++c) b[j][c] = 0.0f;
    auto add = [&](float4 y, int j, float w) {
      b[j][0] = fmaf(w, y.x, b[j][0]);
      b[j][1] = fmaf(w, y.y, b[j][1]);
      b[j][2] = fmaf(w, y.z, b[j][2]);
      b[j][3] = fmaf(w, y.w, b[j][3]);
    };
    int s = 0;
    for (; s < n4; s += 4) {
      float4 w[KMAX];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) w[j] = __ldg(reinterpret_cast<const float4*>(pg + (int64_t)j * n + s));
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 y = yrow[(s + q) * (TV / 4)];
#pragma unroll
        for (int j = 0; j < KMAX; ++j) add(y, j, q == 0 ? w[j].x : q == 1 ? w[j].y : q == 2 ? w[j].z : w[j].w);
      }
    }
    for (; s < n; ++s) {
      const float4 y = yrow[s * (TV / 4)];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) add(y, j, __ldg(pg + (int64_t)j * n + s));
    }
    float rss[kColsPerThread] = {0.0f, 0.0f, 0.0f, 0.0f};
    auto residual = [&](int at, const float* xv) {
      const float4 y = yrow[at * (TV / 4)];
      float r0 = y.x, r1 = y.y, r2 = y.z, r3 = y.w;
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        r0 = fmaf(-xv[j], b[j][0], r0);
        r1 = fmaf(-xv[j], b[j][1], r1);
        r2 = fmaf(-xv[j], b[j][2], r2);
        r3 = fmaf(-xv[j], b[j][3], r3);
      }
      rss[0] = fmaf(r0, r0, rss[0]);
      rss[1] = fmaf(r1, r1, rss[1]);
      rss[2] = fmaf(r2, r2, rss[2]);
      rss[3] = fmaf(r3, r3, rss[3]);
      if (what == kWhatResid) {
        float* dst = t_out + ((int64_t)g * n + at) * ldt + vbase + c0;
        const float rr[4] = {r0, r1, r2, r3};
#pragma unroll
        for (int c = 0; c < kColsPerThread; ++c)
          if (vbase + c0 + c < V) dst[c] = rr[c];
      }
    };
    for (s = 0; s < n4; s += 4) {
      float xv[4 * KMAX];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        const float4 x4 = __ldg(reinterpret_cast<const float4*>(xg + (int64_t)s * KMAX) + j);
        xv[4 * j] = x4.x;
        xv[4 * j + 1] = x4.y;
        xv[4 * j + 2] = x4.z;
        xv[4 * j + 3] = x4.w;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) residual(s + q, xv + q * KMAX);
    }
    for (; s < n; ++s) {
      float xv[KMAX];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) xv[j] = __ldg(xg + (int64_t)s * KMAX + j);
      residual(s, xv);
    }
    if (what == kWhatResid) continue;
    if (what == kWhatRSS || what == kWhatF) {
      float outv[kColsPerThread];
      if (what == kWhatRSS) {
#pragma unroll
        for (int c = 0; c < kColsPerThread; ++c) outv[c] = rss[c];
      } else {
        // F = ((TSS - RSS)/(k-1)) / (RSS/(n-k))   (cynumstats.pyx:31-36).
        // TSS is taken around a supplied centre (the reference uses the grand
        // mean of the whole matrix, np.mean(y)) passed in invdiag[0], or
        // around each column's mean when invdiag is NULL.
        float mean[kColsPerThread] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (invdiag) {
#pragma unroll
          for (int c = 0; c < kColsPerThread; ++c) mean[c] = invdiag[0];
        } else {
          for (int s = 0; s < n; ++s) {
            const float4 y = yrow[s * (TV / 4)];
            mean[0] += y.x; mean[1] += y.y; mean[2] += y.z; mean[3] += y.w;
          }
          const float inv_n = 1.0f / static_cast<float>(n);
#pragma unroll
          for (int c = 0; c < kColsPerThread; ++c) mean[c] *= inv_n;
        }
        float tss[kColsPerThread] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int s = 0; s < n; ++s) {
          const float4 y = yrow[s * (TV / 4)];
          const float d0 = y.x - mean[0], d1 = y.y - mean[1], d2 = y.z - mean[2], d3 = y.w - mean[3];
          tss[0] = fmaf(d0, d0, tss[0]); tss[1] = fmaf(d1, d1, tss[1]);
          tss[2] = fmaf(d2, d2, tss[2]); tss[3] = fmaf(d3, d3, tss[3]);
        }
        const float dg = dof[g];
        const float km1 = static_cast<float>(n) - dg - 1.0f;
#pragma unroll
        for (int c = 0; c < kColsPerThread; ++c) outv[c] = ((tss[c] - rss[c]) / km1) / (rss[c] / dg);
      }
      float* dst = t_out + (int64_t)g * ldt + vbase + c0;
#pragma unroll
      for (int c = 0; c < kColsPerThread; ++c)
        if (vbase + c0 + c < V) dst[c] = outv[c];
      continue;
    }
    const float inv_dof = 1.0f / dof[g];
    for (int ci = 0; ci < n_coef; ++ci) {
      const int j = coef[ci];
      const float d = (what == kWhatBeta) ? 0.0f : invdiag[(int64_t)g * KMAX + j];  // NULL for betas
      float* dst = t_out + ((int64_t)g * n_coef + ci) * ldt + vbase + c0;
#pragma unroll
      for (int c = 0; c < kColsPerThread; ++c) {
        if (vbase + c0 + c < V) {
          float bj = 0.0f;
#pragma unroll
          for (int jj = 0; jj < KMAX; ++jj)
            if (jj == j) bj = b[jj][c];
          const float se = sqrtf(rss[c] * inv_dof * d);
          dst[c] = (what == kWhatT) ? bj / se : (what == kWhatBeta) ? bj : se;
        }
      }
    }
  }
}

template <int KMAX>
int launch_glm_k(int tv, const float* Y, int64_t ldy, int32_t n, int64_t V, const float* pinv,
                 const float* X, const float* invdiag, const float* dof, int32_t G,
                 const int32_t* coef, int32_t n_coef, float* t_out, int64_t ldt, int32_t what,
                 cudaStream_t st) {
  const size_t smem = sizeof(float) * (size_t)n * tv;
  const unsigned grid = static_cast<unsigned>((V + tv - 1) / tv);
#define TFGB_GLM_LAUNCH(TVV)                                                                   \
  do {                                                                                         \
    auto kern = glm_tstat_kernel<KMAX, TVV>;                                                   \
    TFGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                   static_cast<int>(smem)));                                   \
    kern<<<grid, kGlmThreads, smem, st>>>(Y, ldy, n, V, pinv, X, invdiag, dof, G, coef,        \
                                          n_coef, t_out, ldt, what);                           \
  } while (0)
  if (tv == 64) TFGB_GLM_LAUNCH(64);
  else if (tv == 32) TFGB_GLM_LAUNCH(32);
  else TFGB_GLM_LAUNCH(16);
#undef TFGB_GLM_LAUNCH
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

// FP64 form for the observed (unpermuted) statistic and the one-off helpers,
// with the reference's precision: betas and sigma^2 in double from the float32
// data, the SE rounded to float32 (se_of_slope stores it in a float32 array,
// cynumstats.pyx:47-52) and t = double beta / that SE (tval_int, :59-64).
// One thread per vertex, the design's pseudoinverse and rows in shared memory.
//
// Bound by the double pipe (2 FMA per SM and cycle, 64 times fewer than float):
// with residuals in double too and the data converted by it, 200 subjects x
// 305k vertices x 4 columns took 1,213 us.  The betas stay there.  sigma^2 only
// has to decide a float32 rounding, so its residuals are formed in pairs of
// floats, the rounding is taken where the pairs' error bound decides it
// (Ziv 1991), and the vertices where it does not (one in some thousands, data
// out of the float range, a near-perfect fit) redo theirs in double.  The data
// are widened by integer operations.  The results are the same bit for bit, in
// 605 us.

// The double of a float, without the double pipe for normal numbers.
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f), e = u & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return (u << 1) ? (double)f : __hiloint2double((int)u, 0);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}

__device__ __forceinline__ float two_sum(float x, float y, float& err) {  // Knuth
  const float s = __fadd_rn(x, y), t = __fsub_rn(s, x);
  err = __fadd_rn(__fsub_rn(x, __fsub_rn(s, t)), __fsub_rn(y, t));
  return s;
}

template <int KMAX>
__global__ void __launch_bounds__(256) glm_f64_kernel(
    const float* __restrict__ Y, int64_t ldy, int32_t n, int64_t V, const double* __restrict__ pinv,
    const double* __restrict__ X, const double* __restrict__ invdiag, const double* __restrict__ dof,
    const int32_t* __restrict__ coef, int32_t n_coef, int32_t what, double* __restrict__ out, int64_t ldo) {
  extern __shared__ double sm64[];
  double* ps = sm64;                                        // [n][KMAX]
  float2* xs = reinterpret_cast<float2*>(sm64 + KMAX * n);  // [n][KMAX]: X in pairs
  __shared__ uint32_t x_max[KMAX];                          // bits of each column's largest |X|
  const int64_t g = blockIdx.y;
  const double* Xg = X + g * n * KMAX;
  if (threadIdx.x < KMAX) x_max[threadIdx.x] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < KMAX * n; i += blockDim.x) {
    ps[(i % n) * KMAX + i / n] = pinv[g * KMAX * n + i];
    const double x = Xg[i];
    const float hi = (float)x;
    xs[i] = make_float2(hi, (float)(x - (double)hi));
    atomicMax(&x_max[i % KMAX], __float_as_uint(fabsf(hi)));
  }
  __syncthreads();
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  const float* Yv = Y + v;
  double b[KMAX];
#pragma unroll
  for (int j = 0; j < KMAX; ++j) b[j] = 0.0;
#pragma unroll 4
  for (int s = 0; s < n; ++s) {
    const double y = widen(Yv[(int64_t)s * ldy]);
#pragma unroll
    for (int j = 0; j < KMAX; ++j) b[j] = fma(ps[s * KMAX + j], y, b[j]);
  }
  // RSS in pairs of floats, and the bound of its relative error (of its root)
  double rss = 0.0, eps = 1.0;
  if (what != kWhatBeta) {
    float bh[KMAX], bl[KMAX], top = 0.0f, sum = 0.0f, low = 0.0f;
    float reach = 0.0f;  // largest sum of the fit's terms
    bool fits = true;
#pragma unroll
    for (int j = 0; j < KMAX; ++j) {
      bh[j] = -(float)b[j];
      bl[j] = -(float)(b[j] + (double)bh[j]);
      const float xm = __uint_as_float(x_max[j]);
      fits = fits && fabsf(bh[j]) <= 0x1p60f && xm <= 0x1p60f;
      reach = __fmaf_rn(fabsf(bh[j]), xm, reach);
    }
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
      float r = Yv[(int64_t)s * ldy], rl = 0.0f;
      top = fmaxf(top, fabsf(r));
#pragma unroll
      for (int j = 0; j < KMAX; ++j) {
        const float2 x = xs[s * KMAX + j];
        const float p = __fmul_rn(x.x, bh[j]);
        float e;
        r = two_sum(r, p, e);
        rl = __fadd_rn(rl, __fadd_rn(e, __fmaf_rn(x.x, bh[j], -p)));
        rl = __fmaf_rn(x.x, bl[j], __fmaf_rn(x.y, bh[j], rl));
      }
      float e;
      r = two_sum(r, rl, rl);  // the terms may have cancelled down to rl
      const float q = __fmul_rn(r, r);
      sum = two_sum(sum, q, e);
      low = __fadd_rn(low, __fadd_rn(e, __fmaf_rn(__fadd_rn(r, r), rl, __fmaf_rn(r, r, -q))));
      const float t = __fadd_rn(sum, low);  // |low| stays below an ulp of the sum
      low = __fsub_rn(low, __fsub_rn(t, sum));
      sum = t;
    }
    // With u = 2^-24 and M = top + reach, which no partial sum exceeds: x and b as
    // pairs and the product of their low parts left out cost 3 u^2 |x b| a
    // column.  After j columns |rl| <= (j + 3) u M (a two-sum's error is at most u
    // M, the three low products of a column u |x b| each), and a column rounds
    // four times, u times (u M + u |x b|) and three times |rl|: in all
    // u^2 M (1.5 K^2 + 11.5 K + 4), below 0.75 K (K + 8) + 8 times 2^-47 M.  RSS is
    // off by (3 n + 6) u^2 of itself (two roundings of at most u times 2 u of the
    // sum a subject, and those of a square's low part), its root by half of that.
    if (fits && sum >= 0x1p-60f && sum <= 0x1p100f) {
      rss = (double)sum + (double)low;
      const float root = sqrtf(__fdiv_rn(sum, (float)n));
      eps = 0x1p-43 + (double)(0x1p-47f * ((float)n + (0.75f * KMAX * (KMAX + 8) + 8.0f) * ((top + reach) / root)));
    }
  }
  auto rss_double = [&]() {
    double total = 0.0;
    for (int s = 0; s < n; ++s) {
      double r = (double)Yv[(int64_t)s * ldy];
#pragma unroll
      for (int j = 0; j < KMAX; ++j) r = fma(-Xg[s * KMAX + j], b[j], r);
      total = fma(r, r, total);
    }
    return total;
  };
  for (int c = 0; c < n_coef; ++c) {
    const int j = coef[c];
    double bj = 0.0;
#pragma unroll
    for (int jj = 0; jj < KMAX; ++jj)
      if (jj == j) bj = b[jj];
    double* dst = out + (g * n_coef + c) * ldo + v;
    if (j < 0 || j >= KMAX) {
      *dst = CUDART_NAN;
      continue;
    }
    if (what == kWhatBeta) {
      *dst = bj;
      continue;
    }
    double root = sqrt(rss / dof[g] * invdiag[g * KMAX + j]);
    if (eps > 0.0 && !(eps < 0x1p-24 && __double2float_rn(root * (1.0 - eps)) == __double2float_rn(root * (1.0 + eps)))) {
      rss = rss_double();
      eps = 0.0;
      root = sqrt(rss / dof[g] * invdiag[g * KMAX + j]);
    }
    const double se = (double)__double2float_rn(root);
    *dst = (what == kWhatSE) ? se : bj / se;
  }
}

// Aroian (0), Sobel (1), Goodman (2) z from path t values, in double like
// the reference's numpy expression.
__device__ __noinline__ float sobel_double(float fa, float fb, int alg) {
  const double a = fa, b = fb;
  const double ia = 1.0 / (a * a), ib = 1.0 / (b * b), iab = 1.0 / (a * a * b * b);
  double q;
  if (alg == 0) q = ib + ia + iab;
  else if (alg == 1) q = ib + ia;
  else q = ib + ia - iab;
  return (float)(1.0 / sqrt(q));
}

// The same as |ab| / sqrt(a^2 + b^2 + {1, 0, -1}) in pairs of floats.  Products
// are exact by fma (Dekker 1971, with fma), sums carry their rounding error
// (Knuth's two-sum), and one Newton step from rsqrtf squares its error: below
// 2^-42 before the one rounding to float, which is the right one where 2^-40 to
// either side rounds alike (Ziv 1991).  The rest (one value in 2^15), factors
// whose square or product could leave the float range, zeros, NaN and sums that
// cancel go to the double expression.  Three divisions and a root in double
// kept the double pipe busy for 348 us on 64 maps of 82k vertices; this takes 19.
__device__ __forceinline__ float sobel_z(float a, float b, int alg) {
  const float aa = fabsf(a), ab = fabsf(b);
  const float ah = __fmul_rn(a, a), bh = __fmul_rn(b, b);
  const float al = __fmaf_rn(a, a, -ah), bl = __fmaf_rn(b, b, -bh);
  const float one = alg == 0 ? 1.0f : alg == 1 ? 0.0f : -1.0f;
  float e0, e1;
  const float s0 = two_sum(ah, bh, e0);
  const float sh = two_sum(s0, one, e1);
  const float sl = __fadd_rn(__fadd_rn(e0, e1), __fadd_rn(al, bl));
  if (!(fminf(aa, ab) >= 0x1p-40f && fmaxf(aa, ab) <= 0x1p40f && (alg < 2 || sh >= 1.0f))) return sobel_double(a, b, alg);
  const float r = rsqrtf(sh);
  const float rh = __fmul_rn(r, r), rl = __fmaf_rn(r, r, -rh);
  const float h = __fsub_rn(__fmaf_rn(-sh, rh, 1.0f), __fmaf_rn(sh, rl, __fmul_rn(sl, rh)));  // 1 - s r^2
  const float c = __fmul_rn(h, __fmaf_rn(0.375f, h, 0.5f));  // (1 - h)^(-1/2) - 1
  const float ph = __fmul_rn(aa, ab), pl = __fmaf_rn(aa, ab, -ph);
  const float yh = __fmul_rn(ph, r), yl = __fmaf_rn(ph, r, -yh);
  const float lo = __fadd_rn(__fmaf_rn(pl, r, yl), __fmul_rn(yh, c));
  const float z = __fadd_rn(yh, __fmaf_rn(0x1p-40f, yh, lo));
  return z == __fadd_rn(yh, __fmaf_rn(-0x1p-40f, yh, lo)) ? z : sobel_double(a, b, alg);
}

// Grid (vertices / 1024, maps): four strided vertices a thread.
__global__ void __launch_bounds__(256) sobel_combine_kernel(const float* __restrict__ ta, int64_t lda,
                                                            const float* __restrict__ ta_scalar,
                                                            const float* __restrict__ tb, int64_t ldb, int32_t P,
                                                            int64_t V, int32_t alg, float* __restrict__ z,
                                                            int64_t ldz) {
  const int64_t v0 = blockIdx.x * 1024ll + threadIdx.x;
  for (int32_t p = blockIdx.y; p < P; p += gridDim.y) {
    float a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t v = v0 + k * 256;
      if (v < V) {
        a[k] = ta ? ta[p * lda + v] : ta_scalar[p];
        b[k] = tb[p * ldb + v];
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t v = v0 + k * 256;
      if (v < V) z[p * ldz + v] = sobel_z(a[k], b[k], alg);
    }
  }
}

}  // namespace tfgb

extern "C" {

int glm_stat(const float* Y, int64_t ldy, int32_t n, int64_t V, const float* pinv, const float* X,
             const float* invdiag, const float* dof, int32_t G, int32_t kmax, const int32_t* coef,
             int32_t n_coef, int32_t what, float* out, int64_t ldo, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(Y && pinv && X && dof && out, "NULL pointer");
  TFGB_CHECK_ARG(what >= 0 && what <= 5, "what must be in [0, 5]");
  const bool per_coef = (what <= 2);
  TFGB_CHECK_ARG(!per_coef || (coef && n_coef >= 1), "coef list required");
  TFGB_CHECK_ARG(what == 1 || what == 3 || what == 4 || what == 5 || invdiag, "invdiag is NULL");
  if (what != 4 && what != 0 && what != 2) invdiag = nullptr;  // unused
  TFGB_CHECK_ARG(n > 0 && V >= 0 && G >= 0, "bad sizes");
  TFGB_CHECK_ARG(kmax >= 1 && kmax <= 8, "kmax must be in [1, 8]");
  TFGB_CHECK_ARG(ldy >= V && ldo >= V, "leading dimension < V");
  if (V == 0 || G == 0) return TFCE_OK;
  int tv;
  if ((size_t)n * 64 * 4 <= 200 * 1024) tv = 64;
  else if ((size_t)n * 32 * 4 <= 200 * 1024) tv = 32;
  else if ((size_t)n * 16 * 4 <= 200 * 1024) tv = 16;
  else {
    tfgb::set_error("n = %d subjects exceeds the shared-memory tile (max 3200)", n);
    return TFCE_EINVAL;
  }
  if (!per_coef) {
    coef = nullptr;
    n_coef = 0;
  }
  const float* idg = invdiag;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (kmax) {
#define TFGB_K(KK) \
    case KK: return tfgb::launch_glm_k<KK>(tv, Y, ldy, n, V, pinv, X, idg, dof, G, coef, n_coef, out, ldo, what, st);
    TFGB_K(1) TFGB_K(2) TFGB_K(3) TFGB_K(4) TFGB_K(5) TFGB_K(6) TFGB_K(7)
    default: return tfgb::launch_glm_k<8>(tv, Y, ldy, n, V, pinv, X, idg, dof, G, coef, n_coef, out, ldo, what, st);
#undef TFGB_K
  }
}

int glm_tstat(const float* Y, int64_t ldy, int32_t n, int64_t V, const float* pinv, const float* X,
              const float* invdiag, const float* dof, int32_t G, int32_t kmax,
              const int32_t* coef, int32_t n_coef, float* t_out, int64_t ldt, void* stream) {
  return glm_stat(Y, ldy, n, V, pinv, X, invdiag, dof, G, kmax, coef, n_coef, 0, t_out, ldt, stream);
}

int glm_fstat(const float* Y, int64_t ldy, int32_t n, int64_t V, const float* pinv, const float* X,
              const float* dof, int32_t G, int32_t kmax, const float* centre, float* f_out,
              int64_t ldf, void* stream) {
  return glm_stat(Y, ldy, n, V, pinv, X, centre, dof, G, kmax, nullptr, 0, 4, f_out, ldf, stream);
}

int glm_stat_f64(const float* Y, int64_t ldy, int32_t n, int64_t V, const double* pinv, const double* X,
                 const double* invdiag, const double* dof, int32_t G, int32_t kmax, const int32_t* coef,
                 int32_t n_coef, int32_t what, double* out, int64_t ldo, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(Y && pinv && X && dof && out && coef, "NULL pointer");
  TFGB_CHECK_ARG(what >= 0 && what <= 2, "what must be 0 (t), 1 (beta) or 2 (se)");
  TFGB_CHECK_ARG(what == 1 || invdiag, "invdiag is NULL");
  TFGB_CHECK_ARG(n > 0 && V >= 0 && G >= 0 && n_coef >= 1, "bad sizes");
  TFGB_CHECK_ARG(kmax >= 1 && kmax <= 8, "kmax must be in [1, 8]");
  TFGB_CHECK_ARG(ldy >= V && ldo >= V, "leading dimension < V");
  TFGB_CHECK_ARG(G < 65536, "at most 65535 designs per launch");
  const size_t smem = sizeof(double) * 2 * (size_t)kmax * n;
  if (smem > 200 * 1024) {
    tfgb::set_error("n = %d subjects x %d columns exceeds the shared-memory design tile", n, kmax);
    return TFCE_EINVAL;
  }
  if (V == 0 || G == 0) return TFCE_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const dim3 grid(static_cast<unsigned>((V + 255) / 256), static_cast<unsigned>(G));
  switch (kmax) {
#define TFGB_K64(KK)                                                                                   \
    case KK: {                                                                                         \
      const size_t sm = sizeof(double) * 2 * KK * (size_t)n;                                           \
      TFGB_CUDA(cudaFuncSetAttribute(tfgb::glm_f64_kernel<KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     static_cast<int>(sm)));                                           \
      tfgb::glm_f64_kernel<KK><<<grid, 256, sm, st>>>(Y, ldy, n, V, pinv, X, invdiag, dof, coef, n_coef, \
                                                      what, out, ldo);                                 \
      break;                                                                                           \
    }
    TFGB_K64(1) TFGB_K64(2) TFGB_K64(3) TFGB_K64(4) TFGB_K64(5) TFGB_K64(6) TFGB_K64(7) TFGB_K64(8)
#undef TFGB_K64
    default: break;
  }
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

int sobel_combine(const float* ta, int64_t lda, const float* ta_scalar, const float* tb,
                  int64_t ldb, int32_t P, int64_t V, int32_t alg, float* z, int64_t ldz,
                  void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG((ta || ta_scalar) && tb && z, "NULL pointer");
  TFGB_CHECK_ARG(alg >= 0 && alg <= 2, "alg must be 0 (aroian), 1 (sobel) or 2 (goodman)");
  TFGB_CHECK_ARG(P >= 0 && V >= 0, "bad sizes");
  if (P == 0 || V == 0) return TFCE_OK;
  const dim3 grid(static_cast<unsigned>((V + 1023) / 1024), static_cast<unsigned>(std::min(P, 65535)));
  tfgb::sobel_combine_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      ta, lda, ta_scalar, tb, ldb, P, V, alg, z, ldz);
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

}  // extern "C"
