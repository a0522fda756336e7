// Design operators of the quadratic-form GLM (glm_tstat_tc_qf), formed on the
// device: for every design [1, x_1 .. x_k-1] the centred columns as split-BF16
// tiles and inv(Xc'Xc), which the permutation loops of
// tfce_mediation/tmanalysis/vertex_tfce_multiple_regression_randomise.py:90-107
// and vertex_tfce_mediation_randomise.py:79-91 form with numpy for one design at
// a time (cynumstats.pyx:28-29, pyfunc.py:131-145).
//
// A design is named by where its columns come from: a base matrix in FP64, the
// base columns, and an index row that permutes the subjects of some of them.
// So a batch of P permutations sends P x n indices (4 bytes each) to the device
// instead of the centred designs, and no FP64 work is left to the host.
//
// One CTA per design.  Means, cross products and the (k-1) x (k-1) inverse
// are FP64, as the host's were; the columns are rounded to float32 after
// centring and split into BF16 hi/lo.  Bound by latency: 350 subjects x 4
// columns are 11 KB a design, and the inverse is a serial chain; 128 threads
// hold a ragged n without many idle lanes, and a batch has CTAs for every SM.
// Forming them on the host took 6.9 ms per 256 designs of 350 x 5 (numpy) and
// the upload of 1.4 MB; t maps of 64 such designs over 163,842 vertices went
// from 2.03 to 0.52 ms, 64 Aroian mediation permutations from 4.66 to 2.04 ms.
#include <cuda_bf16.h>

#include "common.cuh"

namespace tfgb {

constexpr int kDesignThreads = 128;
constexpr int kDesignCols = 7;     // columns after the intercept
constexpr int32_t kPermuted = 256; // flag of a column entry

struct DesignArgs {
  const double* base;  // [n][ld], or one such matrix per design (stride > 0)
  int64_t ld, stride;
  const int32_t* rows;  // [ceil(G / share)][n] subject of each design row, or NULL
  const int32_t* cols;  // [kmax] or [share][kmax]: base column (| kPermuted) of a design column, -1: none
  int32_t share, n, n_pad, G, kmax, R;
  __nv_bfloat16* tiles;
  float* ginv;     // [G_pad][R][R]
  float* invdiag;  // [G][kmax]
  float* dof;      // [G]
  int32_t* err;
};

constexpr int kDesignSums = kDesignCols * (kDesignCols + 1) / 2;

struct DesignShared {
  double mean[kDesignCols], gram[kDesignCols][2 * kDesignCols];
  double part[kDesignSums][kDesignThreads];  // the threads' sums
};

// Sum q of the threads' n_sums sums, in the first of each four threads.
__device__ inline double gather_sums(const DesignShared& S, int n_sums) {
  const int q = threadIdx.x >> 2, i0 = threadIdx.x & 3;
  double v = 0.0;
  if (q < n_sums)
    for (int i = i0; i < kDesignThreads; i += 4) v += S.part[q][i];
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// Means and centred cross products of the columns entry(s, 0 .. kc), each all
// at once: sum by sum, their 14 reductions (5 columns) took most of a design's
// time.
template <typename Entry>
__device__ void centred_products(const Entry& entry, int kc, int n, DesignShared& S) {
  static_assert(4 * kDesignSums <= kDesignThreads, "four threads add a sum up");
  const int tid = threadIdx.x;
  double sum[kDesignSums] = {};
  for (int i = tid; i < n; i += kDesignThreads)
#pragma unroll
    for (int j = 0; j < kDesignCols; ++j)
      if (j < kc) sum[j] += entry(i, j);
#pragma unroll
  for (int j = 0; j < kDesignCols; ++j)
    if (j < kc) S.part[j][tid] = sum[j];
  __syncthreads();
  const double total = gather_sums(S, kc);
  if (tid % 4 == 0 && tid / 4 < kc) S.mean[tid / 4] = total / n;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kDesignSums; ++q) sum[q] = 0.0;
  for (int i = tid; i < n; i += kDesignThreads) {
    double c[kDesignCols];
#pragma unroll
    for (int j = 0; j < kDesignCols; ++j)
      if (j < kc) c[j] = entry(i, j) - S.mean[j];
#pragma unroll
    for (int j = 0; j < kDesignCols; ++j)
#pragma unroll
      for (int l = 0; l <= j; ++l)
        if (j < kc) sum[j * (j + 1) / 2 + l] += c[j] * c[l];
  }
#pragma unroll
  for (int j = 0; j < kDesignCols; ++j)
#pragma unroll
    for (int l = 0; l <= j; ++l)
      if (j < kc) S.part[j * (j + 1) / 2 + l][tid] = sum[j * (j + 1) / 2 + l];
  __syncthreads();
  const double product = gather_sums(S, kc * (kc + 1) / 2);
  const int q = tid / 4;
  if (tid % 4 == 0 && q < kc * (kc + 1) / 2) {
    int j = 0;
    while ((j + 1) * (j + 2) / 2 <= q) ++j;
    const int l = q - j * (j + 1) / 2;
    S.gram[j][l] = S.gram[l][j] = product;
  }
  __syncthreads();
}

// Inverse of the w x w block at the left of g's rows of `ld` into the block
// beside it, by Gauss-Jordan with row pivots.  One warp, a lane per column.
__device__ void invert(double* g, int ld, int w, int32_t* err) {
  constexpr int kMost = kDesignCols + 1;
  const int lane = threadIdx.x & 31;
  double c[kMost];
#pragma unroll
  for (int r = 0; r < kMost; ++r) {
    c[r] = 0.0;
    if (r < w && lane < w) c[r] = g[r * ld + lane];
    else if (r < w && lane == w + r) c[r] = 1.0;
  }
#pragma unroll
  for (int j = 0; j < kMost; ++j) {
    if (j >= w) break;
    double f[kMost];  // the pivot's column
#pragma unroll
    for (int r = 0; r < kMost; ++r) f[r] = __shfl_sync(0xffffffffu, c[r], j);
    int p = j;
    double top = fabs(f[j]);
#pragma unroll
    for (int r = j + 1; r < kMost; ++r)
      if (r < w && fabs(f[r]) > top) {
        p = r;
        top = fabs(f[r]);
      }
#pragma unroll
    for (int r = j + 1; r < kMost; ++r)
      if (r == p) {
        const double x = c[j], y = f[j];
        c[j] = c[r];
        c[r] = x;
        f[j] = f[r];
        f[r] = y;
      }
    if (f[j] == 0.0 && lane == 0) atomicCAS(err, 0, kDevSingular);
    c[j] = c[j] / f[j];  // divided, so that equal columns leave an exact zero
#pragma unroll
    for (int r = 0; r < kMost; ++r)
      if (r != j && f[r] != 0.0) c[r] = fma(-f[r], c[j], c[r]);
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < kMost; ++r)
    if (r < w && lane >= w && lane < 2 * w) g[r * ld + lane] = c[r];
  __syncwarp();
}

__global__ void __launch_bounds__(kDesignThreads) design_kernel(DesignArgs a) {
  __shared__ DesignShared S;
  __shared__ int32_t sCol[kDesignCols];
  auto& mean = S.mean;
  auto& gram = S.gram;
  const int d = blockIdx.x, tid = threadIdx.x;
  const int kc = a.kmax - 1, R = a.R;
  const bool live = d < a.G;
  const double* X = a.base + (live ? d * a.stride : 0);
  const int32_t* rows = (a.rows && live) ? a.rows + (int64_t)(d / a.share) * a.n : nullptr;
  if (tid < kc) sCol[tid] = live ? a.cols[(d % a.share) * a.kmax + tid + 1] : -1;
  __syncthreads();
  // design entry (s, j); a row index outside [0, n) is recorded and reads row s
  auto entry = [&](int s, int j) -> double {
    const int32_t c = sCol[j];
    if (c < 0) return 0.0;
    int r = s;
    if ((c & kPermuted) && rows) {
      const int p = rows[s];
      if (static_cast<unsigned>(p) < static_cast<unsigned>(a.n)) r = p;
      else atomicCAS(a.err, 0, kDevBadIndex);
    }
    return X[(int64_t)r * a.ld + (c & (kPermuted - 1))];
  };
  if (live) centred_products(entry, kc, a.n, S);
  // a missing column keeps a zero row and column
  if (tid < 32 && live) {
    if (tid == 0) {
      int k = 1;
      for (int j = 0; j < kc; ++j) {
        if (sCol[j] >= 0) ++k;
        else gram[j][j] = 1.0;
      }
      a.dof[d] = static_cast<float>(a.n - k);
    }
    __syncwarp();
    invert(&gram[0][0], 2 * kDesignCols, kc, a.err);
  }
  // the split-BF16 tiles of glm_tile_split: 256-row blocks, 16-column steps of
  // [hi|lo][8-column block][row][8]
  const int ks_count = a.n_pad / 16;
  for (int t = tid; t < R * (a.n_pad / 8); t += kDesignThreads) {
    const int j = t % R, c0 = (t / R) * 8;
    __align__(16) __nv_bfloat16 h[8];
    __align__(16) __nv_bfloat16 l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = c0 + e;
      const float x = (live && j < kc && c < a.n && sCol[j] >= 0) ? static_cast<float>(entry(c, j) - mean[j]) : 0.0f;
      h[e] = __float2bfloat16_rn(x);
      l[e] = __float2bfloat16_rn(x - __bfloat162float(h[e]));
    }
    const int64_t row = (int64_t)d * R + j;
    const int64_t blk = row / 256, r = row % 256;
    const int ks = c0 / 16, kb = (c0 % 16) / 8;
    __nv_bfloat16* at = a.tiles + (blk * ks_count + ks) * 2 * 256 * 16 + kb * 256 * 8 + r * 8;
    *reinterpret_cast<uint4*>(at) = *reinterpret_cast<const uint4*>(h);
    *reinterpret_cast<uint4*>(at + 256 * 16) = *reinterpret_cast<const uint4*>(l);
  }
  __syncthreads();
  for (int t = tid; t < R * R; t += kDesignThreads) {
    const int j = t / R, l = t % R;
    const bool in = live && j < kc && l < kc && sCol[j] >= 0 && sCol[l] >= 0;
    a.ginv[(int64_t)d * R * R + t] = in ? static_cast<float>(gram[j][kc + l]) : 0.0f;
  }
  if (live && tid < a.kmax)
    a.invdiag[(int64_t)d * a.kmax + tid] =
        (tid > 0 && sCol[tid - 1] >= 0) ? static_cast<float>(gram[tid - 1][kc + tid - 1]) : 0.0f;
}

// Operands of the residual-epilogue GLM (glm_stat_tc) for permuted intercept
// designs [1, x_1 .. x_kmax-1], all columns permuted alike: tiles of the
// pseudoinverse rows, their sums, the negated design rows, inv(X'X)'s diagonal
// and the weights of an output program.  The host formed and uploaded them
// batch by batch: 1.1 of the 1.9 ms that 32 permutations of a rhythm model
// over 82k vertices took; this takes 47 us.  The FP32 GLM's (glm_tstat) come
// from here too: 32 weighted permutations 1.00 -> 0.81 ms.
struct ResidualDesignArgs {
  const double* base;   // [n][ld]
  int64_t ld;
  const int32_t* rows;  // [G][n], or NULL
  int32_t n, n_pad, n_sc, G, kmax, DB, centred;
  const int32_t* program;  // [n_rows] {kind, column, width, weight offset}
  int32_t n_rows, w_stride;
  __nv_bfloat16* tiles;    // row blocks of DB * 8
  float* u;                // [G_pad][kmax]
  float* x;                // [G_pad / DB][n_sc][kmax][DB]
  float* invdiag;          // [G][kmax]
  float* dof;              // [G]
  float* weights;          // [G][w_stride]
  // for the FP32 kernel (glm_tstat) instead of tiles, u and x
  float* pinv;             // [G][kmax][n]
  float* rows32;           // [G][n][kmax]
  int32_t* err;
};

__global__ void __launch_bounds__(kDesignThreads) residual_design_kernel(ResidualDesignArgs a) {
  constexpr int kAll = kDesignCols + 1;
  __shared__ DesignShared S;
  __shared__ double full[kAll][kAll];       // inv(X'X)
  __shared__ double block[kAll][2 * kAll];  // a program row's block of it, and its inverse
  const int d = blockIdx.x, tid = threadIdx.x;
  const int kmax = a.kmax, kc = kmax - 1;
  const bool live = d < a.G;
  const int32_t* rows = (a.rows && live) ? a.rows + (int64_t)d * a.n : nullptr;
  auto entry = [&](int s, int j) -> double {  // column j + 1
    int r = s;
    if (rows) {
      const int p = rows[s];
      if (static_cast<unsigned>(p) < static_cast<unsigned>(a.n)) r = p;
      else atomicCAS(a.err, 0, kDevBadIndex);
    }
    return a.base[(int64_t)r * a.ld + j + 1];
  };
  if (live) {
    centred_products(entry, kc, a.n, S);
    if (tid < 32) {
      invert(&S.gram[0][0], 2 * kDesignCols, kc, a.err);
      if (tid < kc) {
        double gm = 0.0;
        for (int l = 0; l < kc; ++l) {
          full[tid + 1][l + 1] = S.gram[tid][kc + l];
          gm = fma(S.gram[tid][kc + l], S.mean[l], gm);
        }
        full[0][tid + 1] = full[tid + 1][0] = -gm;
      }
      __syncwarp();
      if (tid == 0) {
        double m0 = 1.0 / a.n;
        for (int j = 0; j < kc; ++j) m0 = fma(-S.mean[j], full[0][j + 1], m0);
        full[0][0] = m0;
        a.dof[d] = static_cast<float>(a.n - kmax);
      }
      __syncwarp();
      float* w = a.weights + (int64_t)d * a.w_stride;
      for (int t = 0; t < a.n_rows; ++t) {
        const int kind = a.program[4 * t], j = a.program[4 * t + 1], width = a.program[4 * t + 2], o = a.program[4 * t + 3];
        const bool block_row = kind == kTcOutF || kind == kTcOutEss;
        if (!block_row && kind != kTcOutAmp && kind != kTcOutAcro) continue;
        const int size = block_row ? width * width : 3;
        if (o < 0 || width < 1 || width > kAll || o + size > a.w_stride) continue;
        const bool inside = j >= 0 && j + width <= kmax;  // else the GLM returns NaN for the row
        if (inside && block_row) {
          for (int e = tid; e < size; e += 32) block[e / width][e % width] = full[j + e / width][j + e % width];
          __syncwarp();
          invert(&block[0][0], 2 * kAll, width, a.err);
          for (int e = tid; e < size; e += 32) w[o + e] = static_cast<float>(block[e / width][width + e % width]);
          __syncwarp();
        } else {
          for (int e = tid; e < size; e += 32) w[o + e] = inside ? static_cast<float>(full[j + e / 2][j + (e + 1) / 2]) : 0.0f;
        }
      }
    }
    __syncthreads();
  }
  // pseudoinverse entry (row j, subject s)
  auto pinv = [&](int j, int s) {
    double v = j == 0 ? 1.0 / a.n : 0.0;
    for (int l = 0; l < kc; ++l) v = fma(full[j][l + 1], entry(s, l) - S.mean[l], v);
    return v;
  };
  if (a.pinv) {
    for (int t = tid; t < kmax * a.n; t += kDesignThreads) {
      a.pinv[(int64_t)d * kmax * a.n + t] = static_cast<float>(pinv(t / a.n, t % a.n));
      const int s = t / kmax, j = t % kmax;
      a.rows32[(int64_t)d * kmax * a.n + t] = j == 0 ? 1.0f : static_cast<float>(entry(s, j - 1));
    }
    if (tid < kmax) a.invdiag[(int64_t)d * kmax + tid] = static_cast<float>(full[tid][tid]);
    return;
  }
  const int rb = a.DB * 8, ks_count = a.n_pad / 16;
  for (int t = tid; t < 8 * (a.n_pad / 8); t += kDesignThreads) {
    const int j = t % 8, c0 = (t / 8) * 8;
    __align__(16) __nv_bfloat16 h[8];
    __align__(16) __nv_bfloat16 l[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int c = c0 + e;
      const float x = (live && j < kmax && c < a.n) ? static_cast<float>(pinv(j, c)) : 0.0f;
      h[e] = __float2bfloat16_rn(x);
      l[e] = __float2bfloat16_rn(x - __bfloat162float(h[e]));
    }
    const int64_t row = (int64_t)d * 8 + j;
    const int64_t blk = row / rb, r = row % rb;
    const int ks = c0 / 16, kb = (c0 % 16) / 8;
    __nv_bfloat16* at = a.tiles + ((blk * ks_count + ks) * 2 * rb * 16 + (int64_t)kb * rb * 8 + r * 8);
    *reinterpret_cast<uint4*>(at) = *reinterpret_cast<const uint4*>(h);
    *reinterpret_cast<uint4*>(at + (int64_t)rb * 16) = *reinterpret_cast<const uint4*>(l);
  }
  float* x = a.x + (int64_t)(d / a.DB) * a.n_sc * kmax * a.DB + d % a.DB;
  for (int t = tid; t < a.n_sc * kmax; t += kDesignThreads) {
    const int s = t / kmax, j = t % kmax;
    double v = 0.0;
    if (live && s < a.n) {
      if (j == 0) v = a.centred ? 0.0 : -1.0;
      else v = a.centred ? S.mean[j - 1] - entry(s, j - 1) : -entry(s, j - 1);
    }
    x[(int64_t)t * a.DB] = static_cast<float>(v);
  }
  // the rows sum to those of the identity's first column
  if (tid < kmax) {
    a.u[(int64_t)d * kmax + tid] = (live && tid == 0) ? 1.0f : 0.0f;
    if (live) a.invdiag[(int64_t)d * kmax + tid] = static_cast<float>(full[tid][tid]);
  }
}

}  // namespace tfgb

extern "C" {

int glm_fp32_designs(const double* base, int64_t ld, const int32_t* rows, int32_t n, int32_t G, int32_t kmax,
                     float* pinv, float* X, float* invdiag, float* dof, int32_t* err, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(base && pinv && X && invdiag && dof && err, "NULL pointer");
  TFGB_CHECK_ARG(kmax >= 2 && kmax <= 8, "kmax must be in [2, 8]");
  TFGB_CHECK_ARG(n > 0 && ld >= kmax && G >= 0, "bad sizes");
  if (G == 0) return TFCE_OK;
  tfgb::ResidualDesignArgs a{};
  a.base = base;
  a.ld = ld;
  a.rows = rows;
  a.n = n;
  a.G = G;
  a.kmax = kmax;
  a.DB = 1;
  a.pinv = pinv;
  a.rows32 = X;
  a.invdiag = invdiag;
  a.dof = dof;
  a.err = err;
  tfgb::residual_design_kernel<<<static_cast<unsigned>(G), tfgb::kDesignThreads, 0, static_cast<cudaStream_t>(stream)>>>(a);
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

int glm_tc_designs(const double* base, int64_t ld, const int32_t* rows, int32_t n, int32_t n_pad, int32_t n_sc,
                   int32_t G, int32_t kmax, int32_t design_block, int32_t centred, const int32_t* program,
                   int32_t n_rows, int32_t w_stride, void* p_tiles, float* u_rows, float* x_rows, float* invdiag,
                   float* dof, float* weights, int32_t* err, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(base && p_tiles && u_rows && x_rows && invdiag && dof && err, "NULL pointer");
  TFGB_CHECK_ARG(kmax >= 2 && kmax <= 8, "kmax must be in [2, 8]");
  TFGB_CHECK_ARG(n > 0 && n_pad >= n && n_pad % 16 == 0, "n_pad must be >= n and a multiple of 16");
  TFGB_CHECK_ARG(n_sc >= n && ld >= kmax && G >= 0 && n_rows >= 0 && w_stride >= 0, "bad sizes");
  TFGB_CHECK_ARG(design_block == 16 || (design_block == 32 && kmax <= 5),
                 "design_block must be 32 (kmax <= 5) or 16");
  TFGB_CHECK_ARG((n_rows == 0 || program) && (w_stride == 0 || weights), "program / weights is NULL");
  TFGB_CHECK_ARG(reinterpret_cast<uintptr_t>(p_tiles) % 16 == 0, "tiles must be 16-byte aligned");
  if (G == 0) return TFCE_OK;
  tfgb::ResidualDesignArgs a{};
  a.base = base;
  a.ld = ld;
  a.rows = rows;
  a.n = n;
  a.n_pad = n_pad;
  a.n_sc = n_sc;
  a.G = G;
  a.kmax = kmax;
  a.DB = design_block;
  a.centred = centred;
  a.program = program;
  a.n_rows = w_stride ? n_rows : 0;
  a.w_stride = w_stride;
  a.tiles = static_cast<__nv_bfloat16*>(p_tiles);
  a.u = u_rows;
  a.x = x_rows;
  a.invdiag = invdiag;
  a.dof = dof;
  a.weights = weights;
  a.err = err;
  const unsigned grid = static_cast<unsigned>((G + design_block - 1) / design_block * design_block);
  tfgb::residual_design_kernel<<<grid, tfgb::kDesignThreads, 0, static_cast<cudaStream_t>(stream)>>>(a);
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

int glm_qf_designs(const double* base, int64_t ld, int64_t stride, const int32_t* rows, const int32_t* cols,
                   int32_t share, int32_t n, int32_t n_pad, int32_t G, int32_t kmax, void* x_tiles, float* ginv,
                   float* invdiag, float* dof, int32_t* err, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(base && cols && x_tiles && ginv && invdiag && dof && err, "NULL pointer");
  TFGB_CHECK_ARG(kmax >= 2 && kmax <= 8, "kmax must be in [2, 8]");
  TFGB_CHECK_ARG(n > 0 && n_pad >= n && n_pad % 16 == 0, "n_pad must be >= n and a multiple of 16");
  TFGB_CHECK_ARG(ld > 0 && stride >= 0 && share >= 1 && G >= 0, "bad sizes");
  TFGB_CHECK_ARG(reinterpret_cast<uintptr_t>(x_tiles) % 16 == 0, "tiles must be 16-byte aligned");
  if (G == 0) return TFCE_OK;
  tfgb::DesignArgs a{};
  a.base = base;
  a.ld = ld;
  a.stride = stride;
  a.rows = rows;
  a.cols = cols;
  a.share = share;
  a.n = n;
  a.n_pad = n_pad;
  a.G = G;
  a.kmax = kmax;
  a.R = kmax <= 5 ? 4 : 8;
  a.tiles = static_cast<__nv_bfloat16*>(x_tiles);
  a.ginv = ginv;
  a.invdiag = invdiag;
  a.dof = dof;
  a.err = err;
  const int db = glm_qf_design_block(kmax);
  const unsigned grid = static_cast<unsigned>((G + db - 1) / db * db);  // padding designs are written as zeros
  tfgb::design_kernel<<<grid, tfgb::kDesignThreads, 0, static_cast<cudaStream_t>(stream)>>>(a);
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

}  // extern "C"
