// Shared device helpers of libsvsflow: boundary folding, 1D Catmull-Rom, 3D sampling in the
// three interpolation modes, and host-side status handling.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "svsflow.h"

namespace svs {

// ------------------------------------------------------------------------------- host status
void set_error(const std::string& msg);
svs_status fail(svs_status code, const std::string& msg);
// Checks the launch that was just issued (cudaGetLastError) and counts it.
svs_status check_launch(const char* what, uint64_t launches = 1);
svs_status check_cuda(cudaError_t e, const char* what);
void count_launches(uint64_t n);

#define SVS_REQUIRE(cond, msg)                                              \
  do {                                                                      \
    if (!(cond)) return ::svs::fail(SVS_ERR_INVALID_ARG, std::string(msg)); \
  } while (0)

inline unsigned ceil_div(int64_t a, int64_t b) { return (unsigned)((a + b - 1) / b); }

// ----------------------------------------------------------------------------- device helpers

// Index folding of boundary.cuh:25-46 (a single fold), followed by a clamp so that no sample is
// ever read outside the array: the reference reads out of bounds when a sample lies more than
// one volume length outside (boundary.cuh:33-46). The fold is a switch, not the reference's
// device function-pointer table (boundary.cuh:54), so it inlines. The arithmetic on i must not
// overflow (safe_index): the compiler orders clamps and additions on the strength of that.
__device__ __forceinline__ int fold(int i, int n, int bdry) {
  int f = i;
  if (bdry != SVS_BOUNDARY_NEAREST) {  // MIRROR repeats the face's node, REFLECT does not
    const int s = bdry == SVS_BOUNDARY_MIRROR ? 1 : 0;
    f = i > n - 1 ? 2 * n - 2 + s - i : max(i, -i - s);
  }
  return min(max(f, 0), n - 1);
}

// The helpers below are templates on the value type T (float, or double for the FP64 forms of
// the per-operator entry points); the float instantiations are the arithmetic of the reference's
// float path.
// Floor of a grid coordinate as a 32-bit index: saturated beyond the range (defined for every
// value, unlike a cast), and kept far enough inside it that a tap's offset and its fold cannot overflow.
// With a saturated index, index + 2 overflowed, and the compiler, which may move an addition out of the
// clamp to the volume, read out of range. Indices that far out fold to a face either way.
__device__ __forceinline__ int floor_index(float g) { return __float2int_rd(g); }
__device__ __forceinline__ int floor_index(double g) { return __double2int_rd(g); }
__device__ __forceinline__ int safe_index(int i) { return min(max(i, -0x7fffff00), 0x7fffff00); }

// 1D Catmull-Rom through 4 samples in the reference's coefficient form
// (interpolation_cubicHermiteSpline.cuh:20-56), evaluated at buffer coordinate w + 1.
template <typename T>
__device__ __forceinline__ T hermite4(T b0, T b1, T b2, T b3, T w) {
  const T local = w + T(1);
  const int kf = floor_index(local);
  T out;
  if (kf == 1) {
    const T pf = b1, dpf = (b2 - b0) / 2, pc = b2, dpc = (b3 - b1) / 2;
    const T a = 2 * pf - 2 * pc + dpf + dpc;
    const T b = -3 * pf + 3 * pc - 2 * dpf - dpc;
    const T t = local - T(1);
    out = t * (t * (t * a + b) + dpf) + pf;
  } else {
    // w + 1 rounded up to 2.0 (w within half an ulp of 1): the reference then shifts its
    // window by one and reads a zero past the buffer end; at t = 0 this returns b2.
    const T pf = b2, dpf = (b3 - b1) / 2, pc = b3, dpc = (T(0) - b2) / 2;
    const T a = 2 * pf - 2 * pc + dpf + dpc;
    const T b = -3 * pf + 3 * pc - 2 * dpf - dpc;
    const T t = local - T(2);
    out = t * (t * (t * a + b) + dpf) + pf;
  }
  return out;
}

// Strided accessor of one component of a [NZ,NY,NX,stride] field.
template <typename T>
struct FieldRefT {
  const T* __restrict__ p;
  int nz, ny, nx, stride;
  __device__ __forceinline__ T at(int z, int y, int x) const {
    return __ldg(p + ((size_t)((size_t)z * ny + y) * nx + x) * stride);
  }
};
using FieldRef = FieldRefT<float>;

// Grid coordinate -> (floor index, fraction), the reference's floorf(c/h) and c/h - floor.
template <typename T>
__device__ __forceinline__ void split_saturated(T c, T h, int& k, T& w) {
  const T g = h == T(1) ? c : c / h;
  k = floor_index(g);
  w = g - (T)k;
}
template <typename T>
__device__ __forceinline__ void split_coord(T c, T h, int& i, T& w) {
  int k;
  split_saturated(c, h, k, w);
  i = safe_index(k);
}

// Tricubic sample (interpolation_cubicHermiteSpline.cuh:482-525, and the vector/matrix/CNN
// variants :645-791 that differ only in addressing).
template <typename T>
__device__ __forceinline__ T sample_cubic(const FieldRefT<T>& f, T cz, T cy, T cx, T hz, T hy, T hx, int bdry) {
  int ix, iy, iz;
  T wx, wy, wz;
  split_coord(cx, hx, ix, wx);
  split_coord(cy, hy, iy, wy);
  split_coord(cz, hz, iz, wz);
  int xs[4];
#pragma unroll
  for (int d = 0; d < 4; ++d) xs[d] = fold(ix + d - 1, f.nx, bdry);
  T bz[4];
#pragma unroll
  for (int dz = 0; dz < 4; ++dz) {
    const int zz = fold(iz + dz - 1, f.nz, bdry);
    T by[4];
#pragma unroll
    for (int dy = 0; dy < 4; ++dy) {
      const int yy = fold(iy + dy - 1, f.ny, bdry);
      by[dy] = hermite4(f.at(zz, yy, xs[0]), f.at(zz, yy, xs[1]), f.at(zz, yy, xs[2]), f.at(zz, yy, xs[3]), wx);
    }
    bz[dz] = hermite4(by[0], by[1], by[2], by[3], wy);
  }
  return hermite4(bz[0], bz[1], bz[2], bz[3], wz);
}

// hermite4 inside its window (w + 1 below 2) with t = (w + 1) - 1 given. The roundings are those of
// hermite4 with its products fused into its sums: halves and doubles are exact, so (b2 - b0) / 2,
// 2 pf - 2 pc and their sums are kept as differences and scaled where they are used; -3 pf + 3 pc is one
// product and one fused multiply-add. (Exact down to the smallest normal floats: below them a half
// taken early or late may differ in the last bit, as in the vanishing tails of long mask chains.)
template <typename T> __device__ __forceinline__ T hermite_one(T b0, T b1, T b2, T b3, T t) {
  const T e0 = b2 - b0, e1 = b3 - b1;
  const T a2 = fma(T(4), b1 - b2, e0) + e1;
  const T b = fma(T(-0.5), e1, fma(T(3), b2, T(-3) * b1) - e0);
  return fma(t, fma(t, fma(T(0.5) * t, a2, b), T(0.5) * e0), b1);
}


// ...and on two rows of samples at once: the packed FP32 instructions for float, one after the other
// for double. Every operation rounds as its scalar counterpart.
template <typename T> struct Two { T a, b; };
__device__ __forceinline__ Two<float> two_add(Two<float> x, Two<float> y) {
  const float2 r = __fadd2_rn(make_float2(x.a, x.b), make_float2(y.a, y.b));
  return {r.x, r.y};
}
__device__ __forceinline__ Two<float> two_mul(float s, Two<float> x) {
  const float2 r = __fmul2_rn(make_float2(s, s), make_float2(x.a, x.b));
  return {r.x, r.y};
}
__device__ __forceinline__ Two<float> two_fma(float s, Two<float> x, Two<float> y) {
  const float2 r = __ffma2_rn(make_float2(s, s), make_float2(x.a, x.b), make_float2(y.a, y.b));
  return {r.x, r.y};
}
__device__ __forceinline__ Two<double> two_add(Two<double> x, Two<double> y) { return {x.a + y.a, x.b + y.b}; }
__device__ __forceinline__ Two<double> two_mul(double s, Two<double> x) { return {s * x.a, s * x.b}; }
__device__ __forceinline__ Two<double> two_fma(double s, Two<double> x, Two<double> y) {
  return {fma(s, x.a, y.a), fma(s, x.b, y.b)};
}
template <typename T> __device__ __forceinline__ Two<T> two_sub(Two<T> x, Two<T> y) { return two_add(x, Two<T>{-y.a, -y.b}); }
template <typename T>
__device__ __forceinline__ Two<T> hermite_two(Two<T> b0, Two<T> b1, Two<T> b2, Two<T> b3, T t) {
  const Two<T> e0 = two_sub(b2, b0), e1 = two_sub(b3, b1);
  const Two<T> a2 = two_add(two_fma(T(4), two_sub(b1, b2), e0), e1);
  const Two<T> b = two_fma(T(-0.5), e1, two_sub(two_fma(T(3), b2, two_mul(T(-3), b1)), e0));
  return two_fma(t, two_fma(t, two_fma(T(0.5) * t, a2, b), two_mul(T(0.5), e0)), b1);
}

// Where one tricubic sample lies, found once for all fields sampled there: its window's first tap
// and the position in the window per axis. `plain` says that every axis takes hermite4's first branch,
// 1 <= w + 1 < 2. The others are left to sample_cubic: w + 1 rounded up to 2 (the shifted window), and
// coordinates beyond the 32-bit range, whose saturated index leaves w at any distance, or NaN.
template <typename T>
struct CubicTaps {
  int x, y, z;
  T tx, ty, tz;
  bool plain;
};
template <typename T>
__device__ __forceinline__ CubicTaps<T> cubic_taps(T cz, T cy, T cx, T hz, T hy, T hx) {
  CubicTaps<T> k;
  T wx, wy, wz;
  split_saturated(cx, hx, k.x, wx);
  split_saturated(cy, hy, k.y, wy);
  split_saturated(cz, hz, k.z, wz);
  const T lx = wx + T(1), ly = wy + T(1), lz = wz + T(1);
  k.tx = lx - T(1);
  k.ty = ly - T(1);
  k.tz = lz - T(1);
  // (w is below 0 only where the index saturated; two comparisons leave those out with all whose taps'
  // indices could overflow)
  k.plain = lx < T(2) && ly < T(2) && lz < T(2) && min(min(k.x, k.y), k.z) > -0x7fffff00 &&
            max(max(k.x, k.y), k.z) < 0x7fffff00;
  if (k.plain) --k.x, --k.y, --k.z;
  return k;
}
// The sample of one field of fewer than 2^31 elements (x step sx). The four planes one after the
// other (not unrolled): with all 64 loads in flight at once the sample takes 174 registers, and too
// few warps are left to hide them (80^3: 40 us against 23).
template <typename T>
__device__ __forceinline__ T sample_cubic_taps(const T* __restrict__ f, const CubicTaps<T>& k, int nz, int ny, int nx, int sx,
                                               int bdry) {
  int xo[4], yo[4];
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    xo[d] = fold(k.x + d, nx, bdry) * sx;
    yo[d] = fold(k.y + d, ny, bdry) * nx * sx;
  }
  T z0 = T(0), z1 = T(0), z2 = T(0), z3 = T(0);
#pragma unroll 1
  for (int dz = 0; dz < 4; ++dz) {
    const T* p = f + fold(k.z + dz, nz, bdry) * (ny * nx * sx);
    T by[4];
#pragma unroll
    for (int dy = 0; dy < 4; dy += 2) {
      const T *r = p + yo[dy], *q = p + yo[dy + 1];
      const Two<T> v = hermite_two(Two<T>{__ldg(r + xo[0]), __ldg(q + xo[0])}, Two<T>{__ldg(r + xo[1]), __ldg(q + xo[1])},
                                   Two<T>{__ldg(r + xo[2]), __ldg(q + xo[2])}, Two<T>{__ldg(r + xo[3]), __ldg(q + xo[3])}, k.tx);
      by[dy] = v.a;
      by[dy + 1] = v.b;
    }
    z0 = z1;
    z1 = z2;
    z2 = z3;
    z3 = hermite_one(by[0], by[1], by[2], by[3], k.ty);
  }
  return hermite_one(z0, z1, z2, z3, k.tz);
}

// Trilinear sample, interpolation_linear.cuh:250-295 (the 8 terms in the reference's order).
template <typename T>
__device__ __forceinline__ T sample_linear(const FieldRefT<T>& f, T cz, T cy, T cx, T hz, T hy, T hx, int bdry) {
  int ix, iy, iz;
  T wx, wy, wz;
  split_coord(cx, hx, ix, wx);
  split_coord(cy, hy, iy, wy);
  split_coord(cz, hz, iz, wz);
  const int x0 = fold(ix, f.nx, bdry), x1 = fold(ix + 1, f.nx, bdry);
  const int y0 = fold(iy, f.ny, bdry), y1 = fold(iy + 1, f.ny, bdry);
  const int z0 = fold(iz, f.nz, bdry), z1 = fold(iz + 1, f.nz, bdry);
  T out = (1 - wz) * (1 - wy) * (1 - wx) * f.at(z0, y0, x0);
  out += wz * (1 - wy) * (1 - wx) * f.at(z1, y0, x0);
  out += (1 - wz) * (1 - wy) * wx * f.at(z0, y0, x1);
  out += wz * (1 - wy) * wx * f.at(z1, y0, x1);
  out += (1 - wz) * wy * (1 - wx) * f.at(z0, y1, x0);
  out += wz * wy * (1 - wx) * f.at(z1, y1, x0);
  out += (1 - wz) * wy * wx * f.at(z0, y1, x1);
  out += wz * wy * wx * f.at(z1, y1, x1);
  return out;
}

// Nearest-node sample, interpolation_nearest.cuh:250-294 (ties go to the ceiling node).
template <typename T>
__device__ __forceinline__ int nearest_axis(T c, T h, int n, int bdry) {
  const T g = c / h;
  const int k = floor_index(g), f = safe_index(k);
  const T df = g - (T)k;
  const T dc = (T)(f + 1) - g;
  return fold(df < dc ? f : f + 1, n, bdry);
}
template <typename T>
__device__ __forceinline__ T sample_nearest(const FieldRefT<T>& f, T cz, T cy, T cx, T hz, T hy, T hx, int bdry) {
  return f.at(nearest_axis(cz, hz, f.nz, bdry), nearest_axis(cy, hy, f.ny, bdry), nearest_axis(cx, hx, f.nx, bdry));
}

template <typename T>
__device__ __forceinline__ T sample(const FieldRefT<T>& f, T cz, T cy, T cx, T hz, T hy, T hx, int interp, int bdry) {
  if (interp == SVS_INTERPOLATE_CUBIC_HERMITESPLINE) return sample_cubic(f, cz, cy, cx, hz, hy, hx, bdry);
  if (interp == SVS_INTERPOLATE_LINEAR) return sample_linear(f, cz, cy, cx, hz, hy, hx, bdry);
  return sample_nearest(f, cz, cy, cx, hz, hy, hx, bdry);
}

// Forward difference along one axis (differentialOps.cu:540-655): MIRROR is zero on both
// faces, NEAREST and REFLECT take one-sided half differences there. The reference evaluates
// 0.5*(a-b)/h in double (0.5 is a double literal) and rounds to float; 0.5f*(a-b) is exact, so
// the float quotient below is the same correctly rounded value (barring double-rounding ties).
template <typename T>
__device__ __forceinline__ T fwd_axis(T prev, T cur, T next, int i, int n, int bdry, T h) {
  T d;
  if (bdry == SVS_BOUNDARY_MIRROR) {
    if (i > 0 && i < n - 1) d = next - prev;
    else return T(0);
  } else {
    d = (i > 0) ? ((i < n - 1) ? next - prev : cur - prev) : next - cur;
  }
  return (T(0.5) * d) / h;
}

// Adjoint difference along one axis (differentialOps.cu:658-1039), rounded to T per axis.
template <typename T>
__device__ __forceinline__ T adj_axis(T prev, T cur, T next, int i, int n, int bdry) {
  if (bdry == SVS_BOUNDARY_MIRROR) {
    if (i > 1) return (i < n - 2) ? T(0.5) * (prev - next) : T(0.5) * prev;
    return T(-0.5) * next;
  }
  if (i > 0) return (i < n - 1) ? T(0.5) * (prev - next) : T(0.5) * (prev + cur);
  return T(0.5) * (-cur - next);
}

}  // namespace svs
