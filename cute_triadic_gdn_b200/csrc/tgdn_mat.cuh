// What the matrix-gradient kernel and the fused gradient kernel share: sums over the slices and the gradients of the gates.  Both
// kernels form the same values in the same order, so that the stages called one by one give the bits of the whole backward; hence
// the explicit fma and mul of sums that the compiler could otherwise contract in one kernel and not in the other.
#pragma once

#include "tgdn_common.cuh"

namespace tgdn {

__device__ __forceinline__ float mexp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// Sums of sixteen values over the lanes of a warp by halving exchanges: lanes 2i and 2i + 1 end with the sum of value
// (bit 4, 3, 2, 1 of the lane).
__device__ __forceinline__ float warp_sums16(float (&v)[16], int lane) {
#pragma unroll
  for (int n = 8, keep = 16; n >= 1; n >>= 1, keep >>= 1) {
    const bool up = (lane & keep) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], mine = up ? v[i + n] : v[i];
      v[i] = mine + __shfl_xor_sync(0xffffffffu, send, keep);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// A row of E gate values as pairs: sums over the slices run on the two-wide f32 instructions, half as many instructions for the
// same products (each lane an ordinary f32 fma).
template <int E> struct GateVec {
  static constexpr int N = (E + 1) / 2;
  float2 p[N];
  __device__ __forceinline__ void set(int e, float v) { if (e & 1) p[e / 2].y = v; else p[e / 2].x = v; }
  __device__ __forceinline__ float get(int e) const { return (e & 1) ? p[e / 2].y : p[e / 2].x; }
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ float dot(const GateVec& o) const {
    float2 a = __fmul2_rn(p[0], o.p[0]);
#pragma unroll
    for (int i = 1; i < N; ++i) a = __ffma2_rn(p[i], o.p[i], a);
    return E == 1 ? a.x : a.x + a.y;
  }
  __device__ __forceinline__ void add_scaled(float f, const GateVec& o) {
    const float2 ff = make_float2(f, f);
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = __ffma2_rn(ff, o.p[i], p[i]);
  }
  __device__ __forceinline__ void load(const float* row) {       // a dense table row (the same row for the whole warp)
    if constexpr (E % 4 == 0) {
#pragma unroll
      for (int i = 0; i < N; i += 2) {
        const float4 x = *reinterpret_cast<const float4*>(row + 2 * i);
        p[i] = make_float2(x.x, x.y);
        p[i + 1] = make_float2(x.z, x.w);
      }
    } else if constexpr (E % 2 == 0) {
#pragma unroll
      for (int i = 0; i < N; ++i) p[i] = *reinterpret_cast<const float2*>(row + 2 * i);
    } else {
      p[0] = make_float2(row[0], 0.f);
    }
  }
};

// The gradients of one (row, slice): from da, dc (state part), dr, the mask-gradient sums r1, c1 (of dmp) and r2, c2 (of dm), the
// row's log2-domain cumulative gate and that of the chunk's last row.  dgc is the gradient of the cumulative log gate, drr = dr * r.
struct GateGrads { float dk2, dq2, dgc, drr; };
__device__ __forceinline__ GateGrads gate_gradients(float gc, float gl, float k2, float q2, float scale, float da, float dc, float dr,
                                                    float r1, float c1, float r2, float c2) {
  const float eg = mexp2(gc), egr = mexp2(gl - gc);
  GateGrads g;
  g.dk2 = __fmaf_rn(da, eg, __fmul_rn(dr, egr)) + c1 + r2 + c2;
  g.dq2 = __fmaf_rn(__fmul_rn(dc, scale), eg, r1);
  g.drr = __fmul_rn(dr, __fmul_rn(k2, egr));
  float x = __fmaf_rn(da, __fmul_rn(k2, eg), -g.drr);
  x = __fmaf_rn(dc, __fmul_rn(__fmul_rn(scale, q2), eg), x);
  x = __fmaf_rn(q2, r1, x);
  g.dgc = __fmaf_rn(k2, r2 - c1 - c2, x);
  return g;
}

// dg = reverse inclusive cumulative sum of dgc over the 64 rows of a chunk, by one warp: lane l holds rows 63 - l (v1) and 31 - l (v0);
// `last` is what the chunk's last row takes on top, sum_t dr * r + dd * exp(gL) with sum_t dr * r = the warp's sum of `drr`.
__device__ __forceinline__ void reverse_scan(float& v1, float& v0, float drr, float dd, float egl, int lane) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) drr += __shfl_xor_sync(0xffffffffu, drr, o);
  if (lane == 0) v1 += __fmaf_rn(dd, egl, drr);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float a1 = __shfl_up_sync(0xffffffffu, v1, o), a0 = __shfl_up_sync(0xffffffffu, v0, o);
    if (lane >= o) { v1 += a1; v0 += a0; }
  }
  v0 += __shfl_sync(0xffffffffu, v1, 31);
}

}  // namespace tgdn
