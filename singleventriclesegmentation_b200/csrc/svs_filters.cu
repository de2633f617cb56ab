// Pre- and post-filters of the flow path: the Gaussian pre-blur (svs/utils/flow_utils.py:94-112)
// and the 3x3x3 median post-filter (flow_utils.py:115-132), both on the device.
#include <climits>

#include <cuda_runtime.h>

#include "svs_common.cuh"

namespace svs {
namespace {

constexpr int kMaxBlurTaps = 13 * 13 * 13;  // sigma up to 2.6 (kernel size int(5 sigma) made odd)

template <typename T>
struct BlurWeights {
  T w[kMaxBlurTaps];
};

// Zero-padded 3D correlation with a (2r+1)^3 kernel (F.conv3d, padding = r). Accumulates in
// the value type in (z, y, x) tap order.
template <typename T>
__global__ void blur_kernel(const T* __restrict__ in, int nz, int ny, int nx, int r,
                            const __grid_constant__ BlurWeights<T> W, T* __restrict__ out) {
  const int64_t n = (int64_t)nz * ny * nx;
  const int k = 2 * r + 1;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n;
       v += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(v % nx), y = (int)((v / nx) % ny), z = (int)(v / ((int64_t)nx * ny));
    T acc = T(0);
    for (int a = 0; a < k; ++a) {
      const int zz = z + a - r;
      if (zz < 0 || zz >= nz) continue;
      for (int b = 0; b < k; ++b) {
        const int yy = y + b - r;
        if (yy < 0 || yy >= ny) continue;
        const T* row = in + ((size_t)zz * ny + yy) * nx;
        const T* wr = W.w + (a * k + b) * k;
        for (int c = 0; c < k; ++c) {
          const int xx = x + c - r;
          if (xx >= 0 && xx < nx) acc = fma(wr[c], __ldg(row + xx), acc);
        }
      }
    }
    out[v] = acc;
  }
}

// Median of the 27 values around (z, y, x) by rank counting: the element with fewer than 14
// smaller values and at least 14 values not larger than it (exact with ties; with NaNs the
// comparisons leave them out, and the first tap stays if fewer than 14 values are left).
template <typename T>
__device__ __noinline__ T median27_by_rank(const T* __restrict__ in, int nz, int ny, int nx, int C, int z, int y,
                                           int x, int c) {
  T w[27];
  int m = 0;
  for (int a = -1; a <= 1; ++a)
    for (int b = -1; b <= 1; ++b)
      for (int d = -1; d <= 1; ++d)
        w[m++] = __ldg(in + (((size_t)fold(z + a, nz, SVS_BOUNDARY_MIRROR) * ny + fold(y + b, ny, SVS_BOUNDARY_MIRROR)) * nx +
                             fold(x + d, nx, SVS_BOUNDARY_MIRROR)) * C + c);
  T med = w[0];
  for (int i = 0; i < 27; ++i) {
    int lt = 0, le = 0;
    for (int j = 0; j < 27; ++j) {
      lt += w[j] < w[i];
      le += w[j] <= w[i];
    }
    if (lt <= 13 && le > 13) med = w[i];
  }
  return med;
}

__device__ __forceinline__ float tmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float tmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double tmin(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ double tmax(double a, double b) { return fmax(a, b); }
template <typename T> __device__ __forceinline__ void order(T& a, T& b) {
  const T lo = tmin(a, b);
  b = tmax(a, b);
  a = lo;
}
// Sorting network of 9 values: 25 comparators (the least possible) in 7 layers, from B. Dobbelaere's
// published list of sorting networks.
template <typename T> __device__ __forceinline__ void sort9(T (&w)[9]) {
  order(w[0], w[3]); order(w[1], w[7]); order(w[2], w[5]); order(w[4], w[8]);
  order(w[0], w[7]); order(w[2], w[4]); order(w[3], w[8]); order(w[5], w[6]);
  order(w[0], w[2]); order(w[1], w[3]); order(w[4], w[5]); order(w[7], w[8]);
  order(w[1], w[4]); order(w[3], w[6]); order(w[5], w[7]);
  order(w[0], w[1]); order(w[2], w[4]); order(w[3], w[5]); order(w[6], w[8]);
  order(w[2], w[3]); order(w[4], w[5]); order(w[6], w[7]);
  order(w[1], w[2]); order(w[3], w[4]); order(w[5], w[6]);
}
// Median of three sorted lists of 9. Ordering the i-th smallest of the three lists against each
// other leaves 13 of the 27 that can have rank 14: the least of rows 5-8, the middle of rows 2-6,
// the greatest of rows 0-3, three sorted runs whose 7th is the median; the two runs of 4 are
// merged (9 comparators), the 7th of an 8- and a 5-run is a min of maxima.
template <typename T>
__device__ __forceinline__ T median_of_sorted(const T (&a)[9], const T (&b)[9], const T (&c)[9]) {
  T x[8], m[5];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = tmax(tmax(a[i], b[i]), c[i]);
    x[4 + i] = tmin(tmin(a[5 + i], b[5 + i]), c[5 + i]);
  }
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const T lo = tmin(a[2 + i], b[2 + i]), hi = tmax(a[2 + i], b[2 + i]);
    m[i] = tmax(lo, tmin(hi, c[2 + i]));
  }
  order(x[0], x[4]); order(x[1], x[5]); order(x[2], x[6]); order(x[3], x[7]);
  order(x[2], x[4]); order(x[3], x[5]);
  order(x[1], x[2]); order(x[3], x[4]); order(x[5], x[6]);
  const T p = tmin(tmax(x[1], m[4]), tmax(x[2], m[3])), q = tmin(tmax(x[3], m[2]), tmax(x[4], m[1]));
  return tmin(tmin(p, q), tmin(tmax(x[5], m[0]), x[6]));
}

// 3^3 median of each component with scipy 'reflect' (== MIRROR fold) at the faces. A thread owns
// one (x, component) of one row and marches kMedianRun planes along z: each plane's 3 x 3 values
// are loaded and sorted once (25 comparators) and serve the three windows that hold them, whose
// medians take another 26 comparators or so. Bound by the min/max instructions (half rate) and
// their latency at 4 blocks per SM. 80^3 x 3: 275 us by counting ranks (27 x 27 x 2 comparisons,
// indexed local memory), 25 us so; runs of 4 planes 29 us, of 16 25 us, 3 blocks per SM 27 us.
// Windows with a NaN or an infinity (the zero-weighted sum of their values is not zero) are counted.
constexpr int kMedianRun = 8;
template <typename T>
__global__ void __launch_bounds__(128, 4)
median3_kernel(const T* __restrict__ in, int nz, int ny, int nx, int C, T* __restrict__ out) {
  const int64_t row = (int64_t)nx * C;
  const int64_t xb = (row + blockDim.x - 1) / blockDim.x, zb = (nz + kMedianRun - 1) / kMedianRun;
  for (int64_t t = blockIdx.x; t < xb * ny * zb; t += gridDim.x) {
    const int64_t r = (t % xb) * blockDim.x + threadIdx.x;
    if (r >= row) continue;
    const int y = (int)(t / xb % ny), z0 = (int)(t / (xb * ny)) * kMedianRun;
    const int x = (int)(r / C), c = (int)(r - (int64_t)x * C);
    int64_t o[9];
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        o[3 * b + d] = (int64_t)fold(y + b - 1, ny, SVS_BOUNDARY_MIRROR) * row +
                       (int64_t)fold(x + d - 1, nx, SVS_BOUNDARY_MIRROR) * C + c;
    T s[3][9], zero[3];  // the last three planes sorted, and their zero-weighted sums
#pragma unroll
    for (int k = 0; k < kMedianRun + 2; ++k) {
      if (z0 + k - 2 >= nz) break;
      T(&w)[9] = s[k % 3];
      const T* plane = in + (int64_t)fold(min(z0 + k - 1, nz), nz, SVS_BOUNDARY_MIRROR) * ny * row;
      T sum = T(0);
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        w[i] = __ldg(plane + o[i]);
        sum = fma(w[i], T(0), sum);
      }
      zero[k % 3] = sum;
      sort9(w);
      if (k < 2) continue;
      const int z = z0 + k - 2;
      const bool finite = zero[0] + zero[1] + zero[2] == T(0);
      out[(int64_t)z * ny * row + (int64_t)y * row + r] =
          finite ? median_of_sorted(s[0], s[1], s[2]) : median27_by_rank(in, nz, ny, nx, C, z, y, x, c);
    }
  }
}

// Generic odd window (7, and 5 of doubles or of rows beyond 2^31 elements): partial selection sort in local memory up to the median rank.
template <typename T>
__global__ void median_generic_kernel(const T* __restrict__ in, int nz, int ny, int nx, int C,
                                      int ks, T* __restrict__ out) {
  const int64_t n = (int64_t)nz * ny * nx * C;
  const int r = ks / 2, cnt = ks * ks * ks;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(t % C);
    const int64_t v = t / C;
    const int x = (int)(v % nx), y = (int)((v / nx) % ny), z = (int)(v / ((int64_t)nx * ny));
    T w[343];
    int m = 0;
    for (int a = -r; a <= r; ++a)
      for (int b = -r; b <= r; ++b)
        for (int d = -r; d <= r; ++d)
          w[m++] = __ldg(in + (((size_t)fold(z + a, nz, SVS_BOUNDARY_MIRROR) * ny +
                                fold(y + b, ny, SVS_BOUNDARY_MIRROR)) * nx +
                               fold(x + d, nx, SVS_BOUNDARY_MIRROR)) * C + c);
    const int rank = cnt / 2;
    for (int i = 0; i <= rank; ++i) {
      int best = i;
      for (int j = i + 1; j < cnt; ++j)
        if (w[j] < w[best]) best = j;
      const T tmp = w[i]; w[i] = w[best]; w[best] = tmp;
    }
    out[t] = w[rank];
  }
}

// 5^3 median of float values: the 125 values of a window as ordered integers in registers, the
// rank-62 value bracketed by bisection (each step counts the values up to the middle and pulls the
// bracket in to values of the window, about 9 steps). 80^3 x 3: 11.0 ms by selection in local
// memory, 0.41 ms so (bound by the counting instructions). Windows with a NaN are left
// to median_generic_kernel's selection, run here for that voxel.
__device__ __noinline__ float median125_by_selection(const float* __restrict__ in, int nz, int ny, int nx, int C, int z,
                                                     int y, int x, int c) {
  float w[125];
  int m = 0;
  for (int a = -2; a <= 2; ++a)
    for (int b = -2; b <= 2; ++b)
      for (int d = -2; d <= 2; ++d)
        w[m++] = __ldg(in + (((size_t)fold(z + a, nz, SVS_BOUNDARY_MIRROR) * ny + fold(y + b, ny, SVS_BOUNDARY_MIRROR)) * nx +
                             fold(x + d, nx, SVS_BOUNDARY_MIRROR)) * C + c);
  for (int i = 0; i <= 62; ++i) {
    int best = i;
    for (int j = i + 1; j < 125; ++j)
      if (w[j] < w[best]) best = j;
    const float tmp = w[i]; w[i] = w[best]; w[best] = tmp;
  }
  return w[62];
}
// Floats in the order of signed integers (-0 just below +0).
__device__ __forceinline__ int ordered(float v) {
  const int b = __float_as_int(v);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__global__ void __launch_bounds__(128)
median5_kernel(const float* __restrict__ in, int nz, int ny, int nx, int C, float* __restrict__ out) {
  const int64_t row = (int64_t)nx * C, n = row * ny * nz;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t q = t / row;
    const int r = (int)(t - q * row), x = r / C, c = r - x * C, z = (int)(q / ny), y = (int)(q - (int64_t)z * ny);
    int ox[5];
#pragma unroll
    for (int d = 0; d < 5; ++d) ox[d] = fold(x + d - 2, nx, SVS_BOUNDARY_MIRROR) * C + c;
    int w[125];
    int lo = INT_MAX, hi = INT_MIN;
    bool nan = false;
#pragma unroll
    for (int a = 0; a < 5; ++a) {
      const float* plane = in + (int64_t)fold(z + a - 2, nz, SVS_BOUNDARY_MIRROR) * ny * row;
#pragma unroll
      for (int b = 0; b < 5; ++b) {
        const float* line = plane + (int64_t)fold(y + b - 2, ny, SVS_BOUNDARY_MIRROR) * row;
#pragma unroll
        for (int d = 0; d < 5; ++d) {
          const float v = __ldg(line + ox[d]);
          nan |= v != v;
          const int k = ordered(v);
          w[(a * 5 + b) * 5 + d] = k;
          lo = min(lo, k);
          hi = max(hi, k);
        }
      }
    }
    if (nan) {
      out[t] = median125_by_selection(in, nz, ny, nx, C, z, y, x, c);
      continue;
    }
    // the median lies in [lo, hi]; `below` values are less than lo
    while (lo < hi) {
      const int mid = (int)(((long long)lo + hi) >> 1);  // floor: mid < hi
      int cnt = 0, up = INT_MIN, next = INT_MAX;
#pragma unroll
      for (int i = 0; i < 125; ++i) {
        const bool le = w[i] <= mid;
        cnt += le;
        up = max(up, le ? w[i] : INT_MIN);
        next = min(next, le ? INT_MAX : w[i]);
      }
      if (cnt > 62) hi = up;      // the median is at most mid, and no value lies in (up, mid]
      else lo = next;
    }
    out[t] = __int_as_float(lo ^ ((lo >> 31) & 0x7fffffff));
  }
}

// median5_kernel indexes a row (nx voxels of C components) with 32 bits; longer rows take the general kernel.
constexpr bool median5_row_fits(int nx, int C) { return (int64_t)nx * C <= INT_MAX; }
static_assert(median5_row_fits(80, 3) && median5_row_fits(INT_MAX, 1) && !median5_row_fits(1 << 30, 2) &&
                  !median5_row_fits(50000, 50000),
              "no row of more than 2^31 - 1 elements");

unsigned grid_for(int64_t n, int threads) {
  const int64_t blocks = (n + threads - 1) / threads;
  return (unsigned)(blocks < 148 * 64 ? (blocks > 0 ? blocks : 1) : 148 * 64);
}

}  // namespace
}  // namespace svs

using namespace svs;

namespace svs {
namespace {

template <typename T>
svs_status gauss_blur3d(const char* nm, const T* in, int nz, int ny, int nx, const T* weights_host, int r, T* out,
                        cudaStream_t stream) {
  SVS_REQUIRE(in && out && weights_host, std::string(nm) + ": null pointer");
  SVS_REQUIRE(nz > 0 && ny > 0 && nx > 0, std::string(nm) + ": bad sizes");
  SVS_REQUIRE(r >= 0 && (2 * r + 1) * (2 * r + 1) * (2 * r + 1) <= kMaxBlurTaps,
              std::string(nm) + ": kernel radius out of range (max 6)");
  BlurWeights<T> W;
  const int k = 2 * r + 1;
  for (int i = 0; i < k * k * k; ++i) W.w[i] = weights_host[i];
  const int64_t n = (int64_t)nz * ny * nx;
  blur_kernel<T><<<grid_for(n, 256), 256, 0, stream>>>(in, nz, ny, nx, r, W, out);
  return check_launch(nm);
}

template <typename T>
svs_status median3d(const char* nm, const T* in, int nz, int ny, int nx, int C, int ks, T* out, cudaStream_t stream) {
  SVS_REQUIRE(in && out, std::string(nm) + ": null pointer");
  SVS_REQUIRE(nz > 0 && ny > 0 && nx > 0 && C > 0, std::string(nm) + ": bad sizes");
  SVS_REQUIRE(ks == 1 || ks == 3 || ks == 5 || ks == 7, std::string(nm) + ": kernel size must be 1, 3, 5 or 7");
  const int64_t n = (int64_t)nz * ny * nx * C;
  if (ks == 1) return check_cuda(cudaMemcpyAsync(out, in, n * sizeof(T), cudaMemcpyDeviceToDevice, stream), nm);
  if (ks == 3) {
    const int64_t blocks = (((int64_t)nx * C + 127) / 128) * ny * ((nz + kMedianRun - 1) / kMedianRun);
    median3_kernel<T><<<(unsigned)(blocks < (1 << 30) ? blocks : (1 << 30)), 128, 0, stream>>>(in, nz, ny, nx, C, out);
    return check_launch(nm);
  }
  if constexpr (sizeof(T) == 4)
    if (ks == 5 && median5_row_fits(nx, C)) {
      median5_kernel<<<grid_for(n, 128), 128, 0, stream>>>(in, nz, ny, nx, C, out);
      return check_launch(nm);
    }
  median_generic_kernel<T><<<grid_for(n, 128), 128, 0, stream>>>(in, nz, ny, nx, C, ks, out);
  return check_launch(nm);
}

}  // namespace
}  // namespace svs

extern "C" {

svs_status svs_gauss_blur3d(const float* in, int nz, int ny, int nx, const float* weights_host, int r, float* out,
                            svs_stream_t stream) {
  return gauss_blur3d<float>("svs_gauss_blur3d", in, nz, ny, nx, weights_host, r, out, stream);
}
svs_status svs_gauss_blur3d_f64(const double* in, int nz, int ny, int nx, const double* weights_host, int r,
                                double* out, svs_stream_t stream) {
  return gauss_blur3d<double>("svs_gauss_blur3d_f64", in, nz, ny, nx, weights_host, r, out, stream);
}
svs_status svs_median3d(const float* in, int nz, int ny, int nx, int C, int ks, float* out, svs_stream_t stream) {
  return median3d<float>("svs_median3d", in, nz, ny, nx, C, ks, out, stream);
}
svs_status svs_median3d_f64(const double* in, int nz, int ny, int nx, int C, int ks, double* out,
                            svs_stream_t stream) {
  return median3d<double>("svs_median3d_f64", in, nz, ny, nx, C, ks, out, stream);
}

}  // extern "C"
