// FWER lookups: sort the permutation maxima and map TFCE images to 1-p(FWER),
// the GB300 replacement of
//   tfce_mediation/tmanalysis/calculate_fweP_vertex.py:37-69 (mode 0),
//   tfce_mediation/tmanalysis/calculate_fweP_voxel.py:23-49   (mode 0),
//   tfce_mediation/tm_func.py:566-573 / pyfunc.py:254-261      (mode 1).
// The sort is a bitonic network in its "mirror first" form: every
// compare-exchange puts the smaller value at the lower index, so lengths that
// are not a power of two are handled by treating missing elements as +inf
// without storing them (no scratch buffer).
#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace tfgb {

// Doubles as integers of the same order, and back (there are 64 integer
// comparisons to one of doubles; -0 comes before 0, NaN at the ends).
__device__ __forceinline__ long long order_key(long long bits) {
  return bits ^ ((bits >> 63) & 0x7fffffffffffffffll);
}

// Stages of the network that stay within 4,096 values run in shared memory, one
// launch for all of them: 20,000 values took 120 launches (2 us each, whatever
// their size) stage by stage, 234 us; 10 so,
// 65 us.
constexpr int kSortBlock = 4096;
constexpr int kSortThreads = 1024;

// kFirst: sorts every block of 4,096; else the last stages (partners below
// 4,096 apart) of a longer merge.
template <bool kFirst>
__global__ void __launch_bounds__(kSortThreads) bitonic_block(long long* __restrict__ a, int64_t n) {
  __shared__ long long s[kSortBlock];
  const int64_t base = blockIdx.x * (int64_t)kSortBlock;
  const int len = static_cast<int>(min(n - base, (int64_t)kSortBlock));
  for (int i = threadIdx.x; i < len; i += kSortThreads) s[i] = order_key(a[base + i]);
  auto stage = [&](int j, bool mirror) {
    __syncthreads();
    for (int t = threadIdx.x; t < kSortBlock / 2; t += kSortThreads) {
      const int i = 2 * t - (t & (j - 1));  // a zero bit inserted at j
      const int l = mirror ? (i ^ (2 * j - 1)) : (i + j);
      if (l >= len) continue;  // partner is padding (+inf): already in order
      const long long x = s[i], y = s[l];
      if (y < x) {
        s[i] = y;
        s[l] = x;
      }
    }
  };
  for (int k = kFirst ? 2 : 2 * kSortBlock; k <= (kFirst ? kSortBlock : 2 * kSortBlock); k <<= 1) {
    if (kFirst) {
      if (k >= 2 * len) break;
      stage(k / 2, true);
    }
    for (int j = k / 4; j >= 1; j >>= 1) stage(j, false);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < len; i += kSortThreads) a[base + i] = order_key(s[i]);
}

__global__ void bitonic_step(long long* __restrict__ a, int64_t n, int64_t half_pairs, int64_t j,
                             int mirror) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < half_pairs;
       t += (int64_t)gridDim.x * blockDim.x) {
    // t enumerates the lower elements of the pairs: insert a zero bit at j
    const int64_t i = ((t / j) * 2 * j) + (t % j);
    const int64_t l = mirror ? (i ^ (2 * j - 1)) : (i + j);
    if (l >= n) continue;  // partner is padding (+inf): already in order
    const long long x = a[i], y = a[l];
    if (order_key(y) < order_key(x)) {
      a[i] = y;
      a[l] = x;
    }
  }
}

constexpr int kSamples = 512;

// The search starts in 512 samples of the null in shared memory (ten of the
// fifteen steps for 20,000 maxima), each step of which is a dependent load, and
// compares integers: 26 -> 18 us for 328k values.
template <typename T>
__global__ void __launch_bounds__(256) fwer_lookup_kernel(const double* __restrict__ srt, int64_t N,
                                                          const T* __restrict__ img, int64_t V, int mode,
                                                          double* __restrict__ out) {
  __shared__ long long sample[kSamples];  // order keys
  const int64_t stride = (N + kSamples - 1) / kSamples;
  const int n_samples = static_cast<int>((N + stride - 1) / stride);
  for (int i = threadIdx.x; i < n_samples; i += blockDim.x) sample[i] = order_key(__double_as_longlong(srt[i * stride]));
  __syncthreads();
  auto below = [&](double x) -> int64_t {  // maxima below x
    const long long k = order_key(__double_as_longlong(x));
    const long long top = 0x7ff0000000000000ll;
    if (k > top || k < order_key(top | (1ll << 63))) return 0;  // NaN
    const long long x_key = k == 0 ? -1 : k;                    // -0 is not below 0
    int lo = 0, hi = n_samples;
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (sample[mid] < x_key) lo = mid + 1;
      else hi = mid;
    }
    int64_t first = lo ? (lo - 1) * stride + 1 : 0, last = min(N, lo * stride);
    while (first < last) {
      const int64_t mid = (first + last) >> 1;
      if (order_key(__double_as_longlong(srt[mid])) < x_key) first = mid + 1;
      else last = mid;
    }
    return first;
  };
  for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < V;
       v += (int64_t)gridDim.x * blockDim.x) {
    const double x = img[v];
    double p = 0.0;
    if (mode == 0) {
      if (x > 0.0) {
        const int64_t idx = below(x);
        p = (idx == 0) ? 0.0 : (double)(idx - 1) / (double)N;
      }
    } else {
      const int64_t idx = below(x);
      if (idx == N) {
        p = (double)(N - 1) / (double)N;
      } else {
        // idx - 1 == -1 wraps to the last element, as numpy indexing does
        const int64_t lo = (idx == 0) ? N - 1 : idx - 1;
        if (fabs(x - srt[lo]) < fabs(x - srt[idx])) p = (double)lo / (double)N;
        else p = (double)idx / (double)N;
      }
    }
    out[v] = p;
  }
}

}  // namespace tfgb

extern "C" {

int fwer_sort(double* values, int64_t n, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(n >= 0, "n < 0");
  TFGB_CHECK_ARG(n == 0 || values != nullptr, "values is NULL");
  if (n < 2) return TFCE_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  long long* bits = reinterpret_cast<long long*>(values);
  int64_t n2 = 1;
  while (n2 < n) n2 <<= 1;
  const int64_t pairs = n2 / 2;
  const int threads = 256;
  const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((pairs + threads - 1) / threads, 4096));
  const unsigned whole = static_cast<unsigned>((n + tfgb::kSortBlock - 1) / tfgb::kSortBlock);
  tfgb::bitonic_block<true><<<whole, tfgb::kSortThreads, 0, st>>>(bits, n);
  for (int64_t k = 2 * tfgb::kSortBlock; k <= n2; k <<= 1) {
    tfgb::bitonic_step<<<blocks, threads, 0, st>>>(bits, n, pairs, k / 2, 1);
    for (int64_t j = k / 4; j >= tfgb::kSortBlock; j >>= 1)
      tfgb::bitonic_step<<<blocks, threads, 0, st>>>(bits, n, pairs, j, 0);
    tfgb::bitonic_block<false><<<whole, tfgb::kSortThreads, 0, st>>>(bits, n);
  }
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

static int fwer_lookup_any(const double* sorted_null, int64_t N, const void* image, bool f32, int64_t V, int32_t mode,
                           double* out, void* stream) {
  tfgb::clear_error();
  TFGB_CHECK_ARG(N >= 1, "empty null distribution");
  TFGB_CHECK_ARG(sorted_null && image && out, "NULL pointer");
  TFGB_CHECK_ARG(mode == 0 || mode == 1, "mode must be 0 or 1");
  if (V <= 0) return TFCE_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned blocks = static_cast<unsigned>(std::min<int64_t>((V + 255) / 256, 152 * 8));
  if (f32)
    tfgb::fwer_lookup_kernel<<<blocks, 256, 0, st>>>(sorted_null, N, static_cast<const float*>(image), V, mode, out);
  else
    tfgb::fwer_lookup_kernel<<<blocks, 256, 0, st>>>(sorted_null, N, static_cast<const double*>(image), V, mode, out);
  TFGB_CUDA(cudaGetLastError());
  return TFCE_OK;
}

int fwer_lookup(const double* sorted_null, int64_t N, const double* image, int64_t V, int32_t mode,
                double* out, void* stream) {
  return fwer_lookup_any(sorted_null, N, image, false, V, mode, out, stream);
}

int fwer_lookup_f32(const double* sorted_null, int64_t N, const float* image, int64_t V, int32_t mode,
                    double* out, void* stream) {
  return fwer_lookup_any(sorted_null, N, image, true, V, mode, out, stream);
}

}  // extern "C"
