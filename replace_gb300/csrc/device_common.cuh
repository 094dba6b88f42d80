// Device helpers shared by the placement kernels.
#pragma once

#include <cuda_runtime.h>

#include "gpl_internal.h"

namespace gpl {

// Division of 0 <= n < 2^31 by a fixed d >= 1 by a multiplication: with
// 2^(l-1) < d <= 2^l, q = n ceil(2^(31+l) / d) / 2^(31+l) is exact (Granlund
// and Montgomery, PLDI'94).  Integer division is some 25 instructions here,
// and the scatter and gcell kernels need four per gcell.
struct FastDiv {
  unsigned m = 0;
  int d = 1, s = 0;
  FastDiv() = default;
  __host__ explicit FastDiv(int div) : d(div) {
    int l = 0;
    while ((1ll << l) < d) l++;
    s = l - 1;
    if (d > 1) m = (unsigned)(((1ull << (31 + l)) + (unsigned)d - 1) / (unsigned)d);
  }
  __device__ __forceinline__ int operator()(int n) const {
    return d == 1 ? n : (int)(__umulhi((unsigned)n, m) >> s);
  }
};

// Bin column/row bounds of the reference's BinGrid (src/nesterovBase.cpp:684-711):
// uniform binSize steps from the core corner, the last one clipped.
struct BinGeom {
  int core_lx, core_ly, core_ux, core_uy, size_x, size_y, cnt_x, cnt_y;
  FastDiv div_x, div_y;
  __device__ __forceinline__ int lo_x(int a) const { return core_lx + a * size_x; }
  __device__ __forceinline__ int hi_x(int a) const { return min(core_lx + (a + 1) * size_x, core_ux); }
  __device__ __forceinline__ int lo_y(int c) const { return core_ly + c * size_y; }
  __device__ __forceinline__ int hi_y(int c) const { return min(core_ly + (c + 1) * size_y, core_uy); }
  // first and past-the-last bin of [l, u) (offsets from the core corner):
  // l / size and u / size, rounded up when it does not divide (as C divides:
  // towards zero), clamped to the grid
  static __device__ __forceinline__ void span(int l, int u, int size, int cnt, const FastDiv& div, int& i0, int& i1) {
    i0 = l > 0 ? div(l) : 0;
    if (u >= 0) {
      const int q = div(u);
      i1 = q + (u - q * size != 0 ? 1 : 0);
    } else {
      i1 = u > -size ? 1 : 0;
    }
    i1 = min(i1, cnt);
  }
  // getDensityMinMaxIdxX/Y (src/nesterovBase.cpp:822-841), clamped to the
  // grid so that a coordinate outside the core cannot index outside it.
  __device__ __forceinline__ void range(int lx, int ux, int ly, int uy, int& x0, int& x1, int& y0,
                                        int& y1) const {
    span(lx - core_lx, ux - core_lx, size_x, cnt_x, div_x, x0, x1);
    span(ly - core_ly, uy - core_ly, size_y, cnt_y, div_y, y0, y1);
  }
  // getOverlapDensityArea (src/nesterovBase.cpp:1533-1547)
  __device__ __forceinline__ float overlap(int a, int c, int lx, int ux, int ly, int uy) const {
    const int rlx = max(lo_x(a), lx), rux = min(hi_x(a), ux);
    const int rly = max(lo_y(c), ly), ruy = min(hi_y(c), uy);
    if (rlx >= rux || rly >= ruy) return 0.0f;
    return __fmul_rn((float)(rux - rlx), (float)(ruy - rly));
  }
  // the overlap's two factors; 0 where there is none
  __device__ __forceinline__ float overlap_x(int a, int lx, int ux) const {
    return (float)max(min(hi_x(a), ux) - max(lo_x(a), lx), 0);
  }
  __device__ __forceinline__ float overlap_y(int c, int ly, int uy) const {
    return (float)max(min(hi_y(c), uy) - max(lo_y(c), ly), 0);
  }
};

// A gcell's fixed geometry: half density size, scale (bits), and its kind in
// the low byte (0 standard cell, 1 macro, 2 filler; bit 2: covers many bins)
// with a big cell's index above.
struct GCellGeo {
  int2 half;
  float scale;
  int kind;
  __device__ __forceinline__ int type() const { return kind & 3; }
  __device__ __forceinline__ bool big() const { return kind & 4; }
  __device__ __forceinline__ int big_index() const { return kind >> 8; }
};
__device__ __forceinline__ GCellGeo gcell_geo(int4 g) {
  GCellGeo q;
  q.half = make_int2(g.x, g.y);
  q.scale = __int_as_float(g.z);
  q.kind = g.w;
  return q;
}

// GCell::setDensityCenterLocation: float centre truncated to int, then the
// density rectangle is centre -/+ half size (src/nesterovBase.cpp:164-179).
__device__ __forceinline__ void density_rect(float2 c, int2 h, int& lx, int& ux, int& ly, int& uy) {
  const int cx = __float2int_rz(c.x), cy = __float2int_rz(c.y);
  lx = cx - h.x; ux = cx + h.x; ly = cy - h.y; uy = cy + h.y;
}

// getDensityCoordiLayoutInsideX/Y (src/nesterovBase.cpp:1270-1297)
__device__ __forceinline__ float inside(float c, int h, int lo, int hi) {
  float adj = c;
  const float hf = (float)h;
  if (__fsub_rn(c, hf) < (float)lo) adj = (float)(lo + h);
  if (__fadd_rn(c, hf) > (float)hi) adj = (float)(hi - h);
  return adj;
}

// Element i of a small pointer array held in kernel parameters, by selects:
// indexing a parameter array with a run-time index makes the compiler copy
// the whole parameter block to local memory.
template <class T>
__device__ __forceinline__ T pick4(T const (&a)[4], int i) {
  return i == 0 ? a[0] : i == 1 ? a[1] : i == 2 ? a[2] : a[3];
}
template <class T>
__device__ __forceinline__ T pick2(T const (&a)[2], int i) {
  return i == 0 ? a[0] : a[1];
}

// float -> int64 truncation and int64 -> float rounding through 32-bit
// conversions when the value fits (the same results; the 64-bit conversions
// run on the FP64 pipe, which is narrow on this part).
__device__ __forceinline__ unsigned long long trunc_u64(float f) {   // f >= 0
  return f < 4294967296.0f ? (unsigned long long)__float2uint_rz(f) : (unsigned long long)(long long)f;
}
__device__ __forceinline__ float ll_to_float(long long v) {
  return (v >= 0 && v < 2147483648ll) ? __int2float_rn((int)v) : __ll2float_rn(v);
}

// Two floats in one 64-bit register: one packed instruction, each element
// rounded like the scalar operation.
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 p, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}

// fastExp (src/nesterovBase.cpp:1568-1582) of two values: (1 + a / 1024)^1024
// by ten squarings.  The reference evaluates the first step in double; rounded
// once to float, 1 + a / 1024 of a float argument is the same value.  Fused it
// rounds as a product and a sum would: the product with 2^-10 is exact, or too
// small to change 1.
__device__ __forceinline__ F2 fast_exp2(F2 a) {
  a = fma2(a, pack2(0.0009765625f, 0.0009765625f), pack2(1.0f, 1.0f));
#pragma unroll
  for (int i = 0; i < 10; i++) a = mul2(a, a);
  return a;
}

// Block sums of N values; thread 0 writes out_base[k * stride + index]
// (index defaults to the block index).
template <int N>
__device__ __forceinline__ void block_reduce_n(double (&v)[N], double* out_base, int stride,
                                               double* sh /* [32*N] */, int index = -1) {
  if (index < 0) index = blockIdx.x;
#pragma unroll
  for (int k = 0; k < N; k++)
    for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < N; k++) sh[k * 32 + wid] = v[k];
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < N; k++) {
      double x = lane < nw ? sh[k * 32 + lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
      if (lane == 0) out_base[k * stride + index] = x;
    }
  }
  __syncthreads();
}

}  // namespace gpl
