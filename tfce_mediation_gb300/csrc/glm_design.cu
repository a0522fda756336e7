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

__device__ inline double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = 0.0;
  for (int w = 0; w < kDesignThreads / 32; ++w) v += red[w];
  return v;
}

__global__ void __launch_bounds__(kDesignThreads) design_kernel(DesignArgs a) {
  __shared__ double red[kDesignThreads / 32];
  __shared__ double mean[kDesignCols], gram[kDesignCols][2 * kDesignCols];
  __shared__ int32_t sCol[kDesignCols];
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
  if (live) {
    for (int j = 0; j < kc; ++j) {
      double s = 0.0;
      for (int i = tid; i < a.n; i += kDesignThreads) s += entry(i, j);
      s = block_sum(s, red);
      if (tid == 0) mean[j] = s / a.n;
    }
    __syncthreads();
    for (int j = 0; j < kc; ++j)
      for (int l = j; l < kc; ++l) {
        double s = 0.0;
        for (int i = tid; i < a.n; i += kDesignThreads) s += (entry(i, j) - mean[j]) * (entry(i, l) - mean[l]);
        s = block_sum(s, red);
        if (tid == 0) gram[j][l] = gram[l][j] = s;
      }
    __syncthreads();
  }
  // inverse by Gauss-Jordan with row pivots; a missing column keeps a zero
  // row and column
  if (tid == 0) {
    int k = 1;
    if (live) {
      for (int j = 0; j < kc; ++j) {
        const bool has = sCol[j] >= 0;
        k += has;
        for (int l = 0; l < kc; ++l) gram[j][kc + l] = (j == l) ? 1.0 : 0.0;
        if (!has) gram[j][j] = 1.0;
      }
      for (int j = 0; j < kc; ++j) {
        int p = j;
        for (int r = j + 1; r < kc; ++r)
          if (fabs(gram[r][j]) > fabs(gram[p][j])) p = r;
        if (p != j)
          for (int l = 0; l < 2 * kc; ++l) {
            const double t = gram[j][l];
            gram[j][l] = gram[p][l];
            gram[p][l] = t;
          }
        if (gram[j][j] == 0.0) atomicCAS(a.err, 0, kDevSingular);
        const double pivot = gram[j][j];  // divided, so that equal columns leave an exact zero
        for (int l = 0; l < 2 * kc; ++l) gram[j][l] = gram[j][l] / pivot;
        for (int r = 0; r < kc; ++r) {
          if (r == j) continue;
          const double f = gram[r][j];
          if (f != 0.0)
            for (int l = 0; l < 2 * kc; ++l) gram[r][l] = fma(-f, gram[j][l], gram[r][l]);
        }
      }
      a.dof[d] = static_cast<float>(a.n - k);
    }
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

}  // namespace tfgb

extern "C" {

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
