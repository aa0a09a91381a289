// lanes.cuh — lane-wise operations on 16-byte vectors of cells, shared by the step kernels.
#pragma once
#include "kernels.cuh"
#include "stencil2d.cuh"

namespace nw {

// A stencil weight as the lane-wise operations take it: doubled for the packed float32 instructions.
template <typename T> struct LaneWeight { using t = T; };
template <> struct LaneWeight<float> { using t = float2; };
__host__ __device__ inline float2 lane_weight(float w) { return make_float2(w, w); }
__host__ __device__ inline double lane_weight(double w) { return w; }

// Lane-wise arithmetic on a vector, each lane rounded like the scalar operation; float32 lanes go in pairs
// through the packed instructions (half the issue slots).
template <int N>
__device__ __forceinline__ void v_add(const float (&a)[N], const float (&b)[N], float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 r = __fadd2_rn(make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
    o[i] = r.x; o[i + 1] = r.y;
  }
}
template <int N>
__device__ __forceinline__ void v_mul(float2 w, const float (&a)[N], float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 r = __fmul2_rn(w, make_float2(a[i], a[i + 1]));
    o[i] = r.x; o[i + 1] = r.y;
  }
}
template <int N>
__device__ __forceinline__ void v_mul(const float (&w)[N], const float (&a)[N], float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 r = __fmul2_rn(make_float2(w[i], w[i + 1]), make_float2(a[i], a[i + 1]));
    o[i] = r.x; o[i + 1] = r.y;
  }
}
template <int N>
__device__ __forceinline__ void v_fma(float2 w, const float (&a)[N], const float (&b)[N], float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 r = __ffma2_rn(w, make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
    o[i] = r.x; o[i + 1] = r.y;
  }
}
template <int N>
__device__ __forceinline__ void v_fma(const float (&w)[N], const float (&a)[N], const float (&b)[N], float (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float2 r = __ffma2_rn(make_float2(w[i], w[i + 1]), make_float2(a[i], a[i + 1]), make_float2(b[i], b[i + 1]));
    o[i] = r.x; o[i + 1] = r.y;
  }
}
template <int N>
__device__ __forceinline__ void v_add(const double (&a)[N], const double (&b)[N], double (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = add_rn(a[i], b[i]);
}
template <int N>
__device__ __forceinline__ void v_mul(double w, const double (&a)[N], double (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = mul_rn(w, a[i]);
}
template <int N>
__device__ __forceinline__ void v_mul(const double (&w)[N], const double (&a)[N], double (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = mul_rn(w[i], a[i]);
}
template <int N>
__device__ __forceinline__ void v_fma(double w, const double (&a)[N], const double (&b)[N], double (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = fma_rn(w, a[i], b[i]);
}
template <int N>
__device__ __forceinline__ void v_fma(const double (&w)[N], const double (&a)[N], const double (&b)[N], double (&o)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) o[i] = fma_rn(w[i], a[i], b[i]);
}

// The R columns next to a vector on each side, as lap_at's Row3 expects them.
template <typename T, int R, int VZ>
__device__ __forceinline__ void load_sides(const T* p, Row3<T, VZ>& rw) {
  if constexpr (sizeof(T) == 4 && R == 2) {
    const float2 l = *reinterpret_cast<const float2*>(p - 2), r = *reinterpret_cast<const float2*>(p + VZ);
    rw.l[VZ - 2] = l.x; rw.l[VZ - 1] = l.y;
    rw.r[0] = r.x; rw.r[1] = r.y;
  } else {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      rw.l[VZ - 1 - i] = p[-1 - i];
      rw.r[i] = p[VZ + i];
    }
  }
}

}  // namespace nw
