// Electrostatic Poisson solve on the bin grid: the semantics of FFT::doFFT
// (src/fft.cpp:112-177) -- a 2-D DCT-II of the bin density, spectral
// scaling, then an inverse DCT for the potential and mixed sine/cosine
// inverses for the field (Ooura ddct2d / ddsct2d / ddcst2d,
// src/fftsg2d.cpp:569-758) -- computed with shared-memory FFTs.
//
// Layout: every grid array is row-major by y (bin index j*nx + i, the
// reference's BinGrid order); x is the reference's first FFT index.
//
// Three passes, each reading and writing every bin once:
//   A (rows)    density from the int64 areas (+ FP64 overflow partials, and
//               zeroing of the other area buffer) -> DCT-II along x -> spec
//   B (columns) DCT-II along y, spectral solve (phi^ = rho^/(wx^2+wy^2)),
//               inverse along y: P1 = IDCT_y(phi^), P2 = IDST_y(wy*phi^)
//   C (rows)    phi = IDCT_x(P1), Ex = IDST_x(wx*P1), Ey = IDCT_x(P2)
// Real transforms are taken two at a time through one complex FFT (two rows
// or two columns packed as real and imaginary parts), using Makhoul's
// even/odd reordering for the DCT-II and its inverse for the DCT-III; an
// IDST is a DCT-III of the reversed input with alternating output signs.
//
// Two forms of the same passes: on grids of 256 to 2048 bins per axis (but
// 256 x 256) a group of 16 to 64 lanes per packed pair runs a register FFT
// (the "group form", with the density in its own kernel before pass A); other
// grids use one packed pair per 256-thread block and radix-4 Stockham passes
// in shared memory.
#include <cooperative_groups.h>
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "device_common.cuh"
#include "gpl_internal.h"

namespace gpl {

namespace {

namespace cg = cooperative_groups;

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }

// exp(sign * 2 pi i m / n) for 0 <= m < n from the half table tw[m] =
// exp(-2 pi i m / n), m < n/2 (the second half is the negated first half).
__device__ __forceinline__ float2 twiddle(const float2* tw, int m, int n, int sign) {
  const int h = n >> 1;
  float2 w = m < h ? tw[m] : make_float2(-tw[m - h].x, -tw[m - h].y);
  if (sign > 0) w.y = -w.y;
  return w;
}

// Stockham FFT over `batch` sequences of length n = 2^logn stored back to
// back in the shared buffer a; b is a same-size scratch buffer.  Returns the
// buffer that holds the result.  sign -1: forward, +1: unnormalised inverse.
// tw: the half table of this n in shared memory.  Radix-4 passes (one radix-2
// pass first when logn is odd): half as many passes, barriers and shared
// round trips as radix 2.  Pass with sub-transform size ns: element j of
// quarter r is multiplied by exp(sign 2 pi i r k / 4ns), k = j mod ns, and the
// 4-point DFT's outputs go to (j - k) * 4 + k + r ns.
__device__ float2* block_fft(float2* a, float2* b, int n, int logn, int batch, int sign,
                             const float2* __restrict__ tw) {
  int ns = 1, lns = 0;
  if (logn & 1) {
    const int half = n >> 1;
    const int total = half * batch;
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
      const int bi = idx >> (logn - 1);
      const int j = idx & (half - 1);
      const float2* in = a + bi * n;
      float2* out = b + bi * n;
      const float2 u = in[j], v = in[j + half];
      out[2 * j] = cadd(u, v);
      out[2 * j + 1] = csub(u, v);
    }
    __syncthreads();
    float2* t = a; a = b; b = t;
    ns = 2;
    lns = 1;
  }
  if (logn < 2) return a;
  const int lq = logn - 2, q = 1 << lq;
  const int total = q * batch;
  for (; ns < n; ns <<= 2, lns += 2) {
    const int tstep_log = logn - 2 - lns;       // n / (4 ns) = 2^tstep_log
    for (int idx = threadIdx.x; idx < total; idx += blockDim.x) {
      const int bi = idx >> lq;
      const int j = idx & (q - 1);
      const float2* in = a + bi * n;
      float2* out = b + bi * n;
      const int k = j & (ns - 1);
      float2 x0 = in[j], x1 = in[j + q], x2 = in[j + 2 * q], x3 = in[j + 3 * q];
      if (ns > 1) {
        const int m = k << tstep_log;
        x1 = cmul(x1, twiddle(tw, m, n, sign));
        x2 = cmul(x2, twiddle(tw, 2 * m, n, sign));
        x3 = cmul(x3, twiddle(tw, 3 * m, n, sign));
      }
      // 4-point DFT with W = exp(sign 2 pi i / 4) = sign * i
      const float2 a0 = cadd(x0, x2), a1 = csub(x0, x2);
      const float2 b0 = cadd(x1, x3), b1 = csub(x1, x3);
      const float2 wb1 = sign > 0 ? make_float2(-b1.y, b1.x) : make_float2(b1.y, -b1.x);
      const int o = ((j - k) << 2) + k;
      out[o] = cadd(a0, b0);
      out[o + ns] = cadd(a1, wb1);
      out[o + 2 * ns] = csub(a0, b0);
      out[o + 3 * ns] = csub(a1, wb1);
    }
    __syncthreads();
    float2* t = a; a = b; b = t;
  }
  return a;
}

// The twiddles of a length-n FFT, exp(-2 pi i m / n) for m < n/2, copied into
// shared memory from the kFftMax table (the same values, read once per block).
__device__ __forceinline__ void load_twiddles(float2* tws, const float2* __restrict__ tw, int n) {
  const int stride = kFftMax / n;
  for (int m = threadIdx.x; m < n / 2; m += blockDim.x) tws[m] = __ldg(&tw[m * stride]);
}

// Makhoul position of element i of a length-n sequence: v[m] = x[2m],
// v[n-1-m] = x[2m+1].
__device__ __forceinline__ int makhoul_pos(int i, int n) { return (i & 1) ? n - 1 - (i >> 1) : (i >> 1); }

// DCT-II post-processing of a packed pair: from Z = FFT(v0 + i v1) at k and
// (n-k)%n, return (C0[k], C1[k]) with C[k] = Re(exp(-i pi k / 2n) V[k]).
__device__ __forceinline__ float2 dct2_post(float2 zk, float2 znk, float2 w4) {
  float2 zc = cconj(znk);
  float2 v0 = make_float2(0.5f * (zk.x + zc.x), 0.5f * (zk.y + zc.y));
  // (Z - conj Z')/(2i) = (Im part, -Re part)/2 of (Z - conj Z')
  float2 d = csub(zk, zc);
  float2 v1 = make_float2(0.5f * d.y, -0.5f * d.x);
  return make_float2(w4.x * v0.x - w4.y * v0.y, w4.x * v1.x - w4.y * v1.y);
}

// DCT-III pre-processing coefficient c[k] for one real sequence a:
// c[0] = a[0], c[k] = 1/2 exp(+i pi k / 2n) (a[k] - i a[n-k]).
__device__ __forceinline__ float2 dct3_pre(float ak, float ank, float2 w4, int k) {
  if (k == 0) return make_float2(ak, 0.0f);
  float2 e = make_float2(0.5f * w4.x, -0.5f * w4.y);      // 1/2 conj(w4)
  return cmul(e, make_float2(ak, -ank));
}

__device__ __forceinline__ void block_reduce_add(double v, double* out, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) *out = v;
  }
  __syncthreads();
}

struct PassAArgs {
  int nx, ny, logn, pairs_per_block;
  int core_lx, core_ly, core_ux, core_uy, size_x, size_y;
  float td;
  unsigned long long* area_pair[2];  // two sets of inst [nb] then filler [nb]
  const EvalCtl* ctl;                // area_cur: the set to read (the other is zeroed)
  const int64_t* nonplace;
  const float* density_in;           // standalone mode: density given
  float* density;
  float* spec;
  double* part_overflow;
  const float2* tw;
  const float2* w4;                  // exp(-i pi k / 2nx), k < nx
};

// Block vb of pass A (smem: the block's dynamic shared memory); shared by the
// per-job launch and the batched one, as are the bodies of passes B and C.
// The pass bodies are compiled once (not inlined) and called by both
// kernels: inlined into two kernels, the same float expressions can be
// contracted into fused multiply-adds differently, and a job's result would
// then depend on which kernel ran it.
__device__ __noinline__ void poisson_a_body(const PassAArgs& A, int vb, float2* smem) {
  __shared__ double red[32];
  const int n = A.nx;
  const int rp_n = A.pairs_per_block;
  float2* buf0 = smem;
  float2* buf1 = smem + rp_n * n;
  float2* tws = smem + 2 * rp_n * n;                 // [n/2] twiddles
  load_twiddles(tws, A.tw, n);
  const int nb = A.nx * A.ny;
  float ovf_f = 0.0f;          // the thread's few bins in float; FP64 across threads
  const unsigned long long* area = nullptr;
  unsigned long long* area_clear = nullptr;
  if (A.ctl) {
    const int cur = A.ctl->area_cur;
    area = cur == 0 ? A.area_pair[0] : A.area_pair[1];
    area_clear = cur == 0 ? A.area_pair[1] : A.area_pair[0];
  }
  if (A.density_in) {
    for (int idx = threadIdx.x; idx < rp_n * n; idx += blockDim.x) {
      const int rp = idx / n, i = idx - rp * n;
      const int r = vb * rp_n + rp;
      float d0 = 0.0f, d1 = 0.0f;
      if (r < A.ny / 2) {
        d0 = A.density_in[(2 * r) * n + i];
        d1 = A.density_in[(2 * r + 1) * n + i];
      }
      buf0[rp * n + makhoul_pos(i, n)] = make_float2(d0, d1);
    }
  } else {
    // restrict-qualified views: the areas read and the set cleared (and the
    // density written) are distinct arrays, so the loads of later elements
    // can be issued before the stores of earlier ones
    const unsigned long long* __restrict__ ar = area;
    unsigned long long* __restrict__ ac = area_clear;
    const int64_t* __restrict__ np = A.nonplace;
    float* __restrict__ dens = A.density;
#pragma unroll 4
    for (int idx = threadIdx.x; idx < rp_n * n; idx += blockDim.x) {
      const int rp = idx / n, i = idx - rp * n;
      const int r = vb * rp_n + rp;
      float dd[2] = {0.0f, 0.0f};
      if (r < A.ny / 2) {
        const int blx = A.core_lx + i * A.size_x;
        const int bux = min(blx + A.size_x, A.core_ux);
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int j = 2 * r + h;
          const int b = j * n + i;
          const int bly = A.core_ly + j * A.size_y;
          const int buy = min(bly + A.size_y, A.core_uy);
          const long long bin_area = (long long)(bux - blx) * (long long)(buy - bly);
          const float cap = __fmul_rn(ll_to_float(bin_area), A.td);
          const float fi = ll_to_float((long long)ar[b]);
          const float ff = ll_to_float((long long)ar[nb + b]);
          const float fn = ll_to_float(np[b]);
          // BinGrid::updateBinsGCellDensityArea (src/nesterovBase.cpp:804-818)
          dd[h] = __fdiv_rn(__fadd_rn(__fadd_rn(fi, ff), fn), cap);
          ovf_f += fmaxf(0.0f, __fsub_rn(__fadd_rn(fi, fn), cap));
          ac[b] = 0ull;
          ac[nb + b] = 0ull;
          dens[b] = dd[h];
        }
      }
      buf0[rp * n + makhoul_pos(i, n)] = make_float2(dd[0], dd[1]);
    }
  }
  __syncthreads();
  float2* res = block_fft(buf0, buf1, n, A.logn, rp_n, -1, tws);
  for (int idx = threadIdx.x; idx < rp_n * n; idx += blockDim.x) {
    const int rp = idx / n, k = idx - rp * n;
    const int r = vb * rp_n + rp;
    if (r >= A.ny / 2) continue;
    const float2* z = res + rp * n;
    float2 c = dct2_post(z[k], z[(n - k) & (n - 1)], __ldg(&A.w4[k]));
    A.spec[(2 * r) * n + k] = c.x;
    A.spec[(2 * r + 1) * n + k] = c.y;
  }
  if (A.part_overflow) block_reduce_add((double)ovf_f, &A.part_overflow[vb], red);
}

__global__ void __launch_bounds__(256) k_poisson_a(const __grid_constant__ PassAArgs A) {
  extern __shared__ float2 smem[];
  poisson_a_body(A, (int)blockIdx.x, smem);
}

struct PassBArgs {
  int nx, ny, logn, col_pairs;       // column pairs per block
  const float* spec;
  float* p1;
  float* p2;
  const float* wx;
  const float* wy;
  const float2* tw;
  const float2* w4;                  // exp(-i pi k / 2ny), k < ny
  float scale;                       // 4 / (nx ny)
  // group and cluster form (solve_pair): 4 nx / (ny pi^2) and (wy[1] / wx[1])^2,
  // each as the float nearest and the float nearest to the rest
  float num[2], aspect[2];
};

__device__ __noinline__ void poisson_b_body(const PassBArgs& B, int vb, float2* smem) {
  const int n = B.ny;
  const int cp = B.col_pairs;
  float2* s0 = smem;                 // [cp][n] work
  float2* s1 = smem + cp * n;        // [cp][n] scratch
  float2* s2 = smem + 2 * cp * n;    // [cp][n] spectrum: (phi^ col u0, phi^ col u1)
  float2* tws = smem + 3 * cp * n;   // [n/2] twiddles
  load_twiddles(tws, B.tw, n);
  const int u_base = vb * 2 * cp;
  // load: column pair q holds columns u_base + 2q, +1
#pragma unroll 4
  for (int idx = threadIdx.x; idx < 2 * cp * n; idx += blockDim.x) {
    const int v = idx / (2 * cp);           // row (y) index: consecutive threads read one row
    const int c = idx - v * 2 * cp;         // column within block
    const int q = c >> 1;
    const float val = B.spec[v * B.nx + u_base + c];
    float* slot = reinterpret_cast<float*>(&s0[q * n + makhoul_pos(v, n)]);
    slot[c & 1] = val;
  }
  __syncthreads();
  float2* res = block_fft(s0, s1, n, B.logn, cp, -1, tws);
  float2* other = (res == s0) ? s1 : s0;
  // DCT-II along y, then the spectral solve (src/fft.cpp:117-166)
  for (int idx = threadIdx.x; idx < cp * n; idx += blockDim.x) {
    const int q = idx / n, v = idx - q * n;
    const float2* z = res + q * n;
    float2 a = dct2_post(z[v], z[(n - v) & (n - 1)], __ldg(&B.w4[v]));
    float out[2];
    for (int h = 0; h < 2; h++) {
      const int u = u_base + 2 * q + h;
      float d = h ? a.y : a.x;
      if (u == 0) d *= 0.5f;
      if (v == 0) d *= 0.5f;
      d *= B.scale;
      float ph = 0.0f;
      if (u != 0 || v != 0) {
        const float wxu = __ldg(&B.wx[u]), wyv = __ldg(&B.wy[v]);
        ph = __fdiv_rn(d, __fadd_rn(__fmul_rn(wxu, wxu), __fmul_rn(wyv, wyv)));
      }
      out[h] = ph;
    }
    s2[q * n + v] = make_float2(out[0], out[1]);
  }
  __syncthreads();
  // P1 = IDCT_y(phi^) for both columns (one complex IFFT)
  for (int idx = threadIdx.x; idx < cp * n; idx += blockDim.x) {
    const int q = idx / n, k = idx - q * n;
    const float2* sp = s2 + q * n;
    const float2 w4 = __ldg(&B.w4[k]);
    float2 ak = sp[k], ank = k ? sp[n - k] : make_float2(0.f, 0.f);
    float2 c0 = dct3_pre(ak.x, ank.x, w4, k);
    float2 c1 = dct3_pre(ak.y, ank.y, w4, k);
    other[q * n + k] = make_float2(c0.x - c1.y, c0.y + c1.x);   // c0 + i c1
  }
  __syncthreads();
  float2* scratch = (other == s0) ? s1 : s0;
  res = block_fft(other, scratch, n, B.logn, cp, +1, tws);
  for (int idx = threadIdx.x; idx < 2 * cp * n; idx += blockDim.x) {
    const int v = idx / (2 * cp);
    const int c = idx - v * 2 * cp;
    const int q = c >> 1;
    const float2 w = res[q * n + makhoul_pos(v, n)];
    B.p1[v * B.nx + u_base + c] = (c & 1) ? w.y : w.x;
  }
  __syncthreads();
  // P2 = IDST_y(wy * phi^): DCT-III of b[k] = wy[n-k] phi^[n-k] (b[0] = 0)
  other = (res == s0) ? s1 : s0;
  for (int idx = threadIdx.x; idx < cp * n; idx += blockDim.x) {
    const int q = idx / n, k = idx - q * n;
    const float2* sp = s2 + q * n;
    const float2 w4 = __ldg(&B.w4[k]);
    float2 bk = make_float2(0.f, 0.f), bnk = make_float2(0.f, 0.f);
    if (k) {
      const float w = __ldg(&B.wy[n - k]);
      bk = make_float2(__fmul_rn(sp[n - k].x, w), __fmul_rn(sp[n - k].y, w));
      const float w2 = __ldg(&B.wy[k]);
      bnk = make_float2(__fmul_rn(sp[k].x, w2), __fmul_rn(sp[k].y, w2));
    }
    float2 c0 = dct3_pre(bk.x, bnk.x, w4, k);
    float2 c1 = dct3_pre(bk.y, bnk.y, w4, k);
    other[q * n + k] = make_float2(c0.x - c1.y, c0.y + c1.x);
  }
  __syncthreads();
  scratch = (other == s0) ? s1 : s0;
  res = block_fft(other, scratch, n, B.logn, cp, +1, tws);
  for (int idx = threadIdx.x; idx < 2 * cp * n; idx += blockDim.x) {
    const int v = idx / (2 * cp);
    const int c = idx - v * 2 * cp;
    const int q = c >> 1;
    const float2 w = res[q * n + makhoul_pos(v, n)];
    const float s = (v & 1) ? -1.0f : 1.0f;
    B.p2[v * B.nx + u_base + c] = s * ((c & 1) ? w.y : w.x);
  }
}

__global__ void __launch_bounds__(256) k_poisson_b(const __grid_constant__ PassBArgs B) {
  extern __shared__ float2 smem[];
  poisson_b_body(B, (int)blockIdx.x, smem);
}

struct PassCArgs {
  int nx, ny, logn, pairs_per_block;
  const float* p1;
  const float* p2;
  float2* field;          // (Ex, Ey) interleaved, may be null
  float* fx;              // or separate planes (standalone API)
  float* fy;
  float* phi;             // may be null
  const float* wx;
  const float2* tw;
  const float2* w4;       // exp(-i pi k / 2nx)
};

// One DCT-III (or IDST with sign flip) of a packed row pair held in smem
// rows a0/a1 (real inputs); writes packed c coefficients into dst.
__device__ __forceinline__ void build_dct3_pair(const float* a0, const float* a1, const float* wmul,
                                                bool reverse, float2* dst, int n, int k, float2 w4) {
  float x0k, x0nk, x1k, x1nk;
  if (!reverse) {
    x0k = a0[k]; x1k = a1[k];
    x0nk = k ? a0[n - k] : 0.f; x1nk = k ? a1[n - k] : 0.f;
  } else {
    // b[k] = w[n-k] a[n-k] for k >= 1, b[0] = 0
    if (k) {
      const float wa = wmul ? __ldg(&wmul[n - k]) : 1.0f;
      const float wb = wmul ? __ldg(&wmul[k]) : 1.0f;
      x0k = __fmul_rn(a0[n - k], wa); x1k = __fmul_rn(a1[n - k], wa);
      x0nk = __fmul_rn(a0[k], wb); x1nk = __fmul_rn(a1[k], wb);
    } else {
      x0k = x1k = x0nk = x1nk = 0.f;
    }
  }
  float2 c0 = dct3_pre(x0k, x0nk, w4, k);
  float2 c1 = dct3_pre(x1k, x1nk, w4, k);
  dst[k] = make_float2(c0.x - c1.y, c0.y + c1.x);
}

__device__ __noinline__ void poisson_c_body(const PassCArgs& C, int vb, float2* smem) {
  const int n = C.nx;
  const int rp_n = C.pairs_per_block;
  float* rows = reinterpret_cast<float*>(smem);       // [rp][4][n]: p1 row0, p1 row1, p2 row0, p2 row1
  float2* s0 = smem + rp_n * 2 * n;                    // [rp][n]
  float2* s1 = s0 + rp_n * n;                          // [rp][n]
  float2* tws = s1 + rp_n * n;                         // [n/2] twiddles
  load_twiddles(tws, C.tw, n);
#pragma unroll 4
  for (int idx = threadIdx.x; idx < rp_n * 2 * n; idx += blockDim.x) {
    const int rp = idx / (2 * n), t = idx - rp * 2 * n;
    const int h = t / n, i = t - h * n;
    const int r = vb * rp_n + rp;
    float a = 0.f, b = 0.f;
    if (r < C.ny / 2) {
      a = C.p1[(2 * r + h) * n + i];
      b = C.p2[(2 * r + h) * n + i];
    }
    rows[(rp * 4 + h) * n + i] = a;
    rows[(rp * 4 + 2 + h) * n + i] = b;
  }
  __syncthreads();
  // three transforms: 0 = phi (IDCT P1), 1 = Ex (IDST wx*P1), 2 = Ey (IDCT P2)
  for (int tr = (C.phi ? 0 : 1); tr < 3; tr++) {
    for (int idx = threadIdx.x; idx < rp_n * n; idx += blockDim.x) {
      const int rp = idx / n, k = idx - rp * n;
      const float* a0 = rows + (rp * 4 + (tr == 2 ? 2 : 0)) * n;
      const float* a1 = a0 + n;
      build_dct3_pair(a0, a1, tr == 1 ? C.wx : nullptr, tr == 1, s0 + rp * n, n, k, __ldg(&C.w4[k]));
    }
    __syncthreads();
    float2* res = block_fft(s0, s1, n, C.logn, rp_n, +1, tws);
    for (int idx = threadIdx.x; idx < rp_n * n; idx += blockDim.x) {
      const int rp = idx / n, m = idx - rp * n;
      const int r = vb * rp_n + rp;
      if (r >= C.ny / 2) continue;
      const float2 w = res[rp * n + makhoul_pos(m, n)];
      float v0 = w.x, v1 = w.y;
      if (tr == 1 && (m & 1)) { v0 = -v0; v1 = -v1; }
      const int b0 = (2 * r) * n + m, b1 = (2 * r + 1) * n + m;
      if (tr == 0) {
        C.phi[b0] = v0; C.phi[b1] = v1;
      } else if (C.field) {
        // Ex waits in the P1 rows (no longer read) and goes out with Ey as
        // one float2 per bin
        float* ex = rows + (rp * 4) * n;
        if (tr == 1) {
          ex[m] = v0; ex[n + m] = v1;
        } else {
          C.field[b0] = make_float2(ex[m], v0);
          C.field[b1] = make_float2(ex[n + m], v1);
        }
      } else {
        float* dst = tr == 1 ? C.fx : C.fy;
        dst[b0] = v0; dst[b1] = v1;
      }
    }
    __syncthreads();
    if (res != s0) { float2* t = s0; s0 = s1; s1 = t; }
  }
}

__global__ void __launch_bounds__(256) k_poisson_c(const __grid_constant__ PassCArgs C) {
  extern __shared__ float2 smem[];
  poisson_c_body(C, (int)blockIdx.x, smem);
}

// ---------------------------------------------------------------------------
// Group form, for grids whose counts are both 256, 512, 1024 or 2048 (256 x
// 256 excepted).  A group of G lanes (16, 32 or 64) runs one N-point FFT of a
// packed pair (two rows or two columns as real and imaginary parts) with
// E = N / G elements per lane in registers, four-step: DFTs along n2 inside
// each lane, the twiddle W^(n1 k2), one transpose through padded shared
// memory, then G-point DFTs along n1 (for N = 512 and 2048, where G = 2 E,
// each of those is split over a lane pair: two E-point DFTs and one radix-2
// step by shuffle).  The block form's radix-4 passes in shared memory take
// five or six passes with block barriers for the same transform.
// What bounds these passes is latency and issue, not bytes, so: independent
// transforms of a pair run on separate groups (the column pass's two inverse
// transforms, the field pass's three); elements k and n - k, which every pre-
// and post-processing step combines, are handled by one lane, in place, so
// that no second copy of the rows or the spectrum is kept (at 2048 points
// that is what lets two field blocks share an SM); and the density comes from
// its own grid-wide kernel first (fusing it into the row pass was measured
// slower: its long blocks overlap worse with the WA kernel).
// Solve of a 2048 x 2048 grid with the potential: 314 us in the block form,
// 92 us here; 512 x 256: 26.6 -> 20.5; 1024 x 1024: 34.8 -> 32.8.

template <int N>
struct GroupFft {
  static_assert(N >= 64 && N <= 2048 && (N & (N - 1)) == 0, "group form sizes");
  static constexpr int kG = N <= 128 ? 8 : N == 256 ? 16 : N == 2048 ? 64 : 32;   // lanes per transform
  static constexpr int kE = N / kG;                                // elements per lane
  static constexpr int kStride = kE + 1;                           // padded transpose row
  static constexpr int kBuf = 2 * kG * kStride;                    // floats per group buffer
  static_assert(kBuf >= 2 * N, "the transpose holds the sequence");
};

// exp(-2 pi i n1 k2 / N) at [k2 * G + n1], k2 < E, where an index in the upper
// half of its range stands for itself minus the range (group_fft): one
// coalesced row per k2.
__device__ __align__(16) float2 g_tw64[64];
__device__ __align__(16) float2 g_tw128[128];
__device__ __align__(16) float2 g_tw256[256];
__device__ __align__(16) float2 g_tw512[512];
__device__ __align__(16) float2 g_tw1024[1024];
__device__ __align__(16) float2 g_tw2048[2048];

template <int N>
__device__ __forceinline__ const float2* tw_table() {
  if constexpr (N == 2048) return g_tw2048;
  else if constexpr (N == 1024) return g_tw1024;
  else if constexpr (N == 512) return g_tw512;
  else if constexpr (N == 256) return g_tw256;
  else if constexpr (N == 128) return g_tw128;
  else return g_tw64;
}

template <int kBits>
__host__ __device__ constexpr int brev(int r) {
  int o = 0;
  for (int b = 0; b < kBits; b++) o |= ((r >> b) & 1) << (kBits - 1 - b);
  return o;
}

// cos and sin of 2 pi m / 64, m = 0..16 (the other octants by symmetry).
__host__ __device__ constexpr float cos64_quad(int m) {
  return m == 0 ? 1.0f
       : m == 1 ? 0.995184726672196929f
       : m == 2 ? 0.980785280403230431f
       : m == 3 ? 0.956940335732208824f
       : m == 4 ? 0.923879532511286738f
       : m == 5 ? 0.881921264348355050f
       : m == 6 ? 0.831469612302545236f
       : m == 7 ? 0.773010453362736993f
       : m == 8 ? 0.707106781186547573f
       : m == 9 ? 0.634393284163645488f
       : m == 10 ? 0.555570233019602289f
       : m == 11 ? 0.471396736825997809f
       : m == 12 ? 0.382683432365089837f
       : m == 13 ? 0.290284677254462331f
       : m == 14 ? 0.195090322016128331f
       : m == 15 ? 0.098017140329560770f
       : 0.0f;
}
__host__ __device__ constexpr float cos64(int m) {   // 0 <= m < 32
  return m <= 16 ? cos64_quad(m) : -cos64_quad(32 - m);
}
__host__ __device__ constexpr float sin64(int m) {   // 0 <= m < 32
  return m <= 16 ? cos64_quad(16 - m) : cos64_quad(m - 16);
}

// The inverse transforms' cos(pi / 16) and cos(pi / 8): the floats above the
// nearest ones, which lie almost as far on the other side (3.0e-8 and 3.1e-8
// instead of 3.0e-8 and 2.8e-8).  Nearest in both directions, every rotation by
// them shortens, and the error of a solve's transforms adds up in its low modes;
// so one direction shortens and the other lengthens (2048 x 2048: Ex 1.78e-7 ->
// 1.67e-7, phi 1.69e-7 -> 1.56e-7).
__host__ __device__ constexpr float up64(float c) {
  const float a = c < 0.0f ? -c : c;
  const float u = a == cos64_quad(2) ? 0.98078534f : a == cos64_quad(4) ? 0.92387956f : a;
  return c < 0.0f ? -u : u;
}

// (re, im) times exp(kSign 2 pi i m / 64), m < 32 a compile-time constant.
template <int kSign>
__device__ __forceinline__ void rot64(float& re, float& im, int m) {
  if (m == 0) return;
  const float r = re, i = im;
  if (m == 16) {                    // exp(kSign i pi / 2) = kSign i
    re = kSign > 0 ? -i : i;
    im = kSign > 0 ? r : -r;
    return;
  }
  const float c = kSign > 0 ? up64(cos64(m)) : cos64(m), sn = kSign > 0 ? up64(sin64(m)) : -sin64(m);
  re = r * c - i * sn;
  im = r * sn + i * c;
}

// (re, im) times exp(kSign 2 pi i m / 64), m < 64 a compile-time constant.
template <int kSign>
__device__ __forceinline__ void rot64_full(float& re, float& im, int m) {
  if (m >= 32) { re = -re; im = -im; m -= 32; }
  rot64<kSign>(re, im, m);
}

// In-register M-point DFT (M = 8, 16 or 32), decimation in frequency: natural
// input order, register r ends with output brev(r).  Two radix-2 stages at a
// time, so that a value meets one twiddle where two stages would give it two
// (an odd last stage has none): fewer roundings and fewer instructions than
// stage by stage (field error against 64 bits 2.17e-7 instead of 2.40e-7 at
// 2048 x 2048, before the steps of group_fft and up64).  Twiddles
// exp(kSign 2 pi i j / len) = exp(kSign 2 pi i (j 64/len) / 64) are compile-time
// constants after unrolling.
template <int M, int kSign>
__device__ __forceinline__ void dft_reg(float (&re)[M], float (&im)[M]) {
#pragma unroll
  for (int len = M; len >= 4; len >>= 2) {
    const int q = len >> 2;
#pragma unroll
    for (int start = 0; start < M; start += len) {
#pragma unroll
      for (int j = 0; j < q; j++) {
        const int a = start + j, b = a + q, c = b + q, d = c + q;
        const float sr = re[a] + re[c], si = im[a] + im[c], tr = re[a] - re[c], ti = im[a] - im[c];
        const float ur = re[b] + re[d], ui = im[b] + im[d], vr = re[b] - re[d], vi = im[b] - im[d];
        // kSign i (b - d)
        const float wr = kSign > 0 ? -vi : vi, wi = kSign > 0 ? vr : -vr;
        re[a] = sr + ur; im[a] = si + ui;
        re[b] = sr - ur; im[b] = si - ui;
        re[c] = tr + wr; im[c] = ti + wi;
        re[d] = tr - wr; im[d] = ti - wi;
        rot64_full<kSign>(re[b], im[b], 2 * j * (64 / len));
        rot64_full<kSign>(re[c], im[c], j * (64 / len));
        rot64_full<kSign>(re[d], im[d], 3 * j * (64 / len));
      }
    }
    if (len == 8) {                   // the last stage, of pairs
#pragma unroll
      for (int a = 0; a < M; a += 2) {
        const float ar = re[a], ai = im[a];
        re[a] = ar + re[a + 1]; im[a] = ai + im[a + 1];
        re[a + 1] = ar - re[a + 1]; im[a + 1] = ai - im[a + 1];
      }
    }
  }
}

// Asynchronous global -> shared copies (cp.async, sm_80+): a block issues
// all of its inputs and tables at once and waits once, so each pass pays one
// memory latency instead of one per dependent load batch.
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Barrier of the calling group: its lanes of the warp, or for 64 lanes two
// warps by the named barrier 1 + the group's number in the block.
template <int G>
__device__ __forceinline__ void group_sync() {
  if constexpr (G == 32) __syncwarp();
  else if constexpr (G < 32) __syncwarp(((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1)));
  else asm volatile("bar.sync %0, 64;\n" ::"r"(1 + (int)(threadIdx.x >> 6)) : "memory");
}

// N-point FFT of buf (natural order in and out, [GroupFft<N>::kBuf] floats,
// float2 view) by the calling group; kSign -1 forward, +1 unnormalised
// inverse.  tws: the tw_table<N>() table in shared memory.
//
// The four steps take n = n1 + G n2 and k = k2 + E k1 with n1 and k2 of either
// sign, -G/2 <= n1 < G/2 and -E/2 <= k2 < E/2: the same sums with the first
// loads and the last stores shifted.  The field lies in the modes next to 0
// and N, so its twiddles W^(n1 k2) then turn by little, and floats close to 1
// and 0 are nearer to them than floats on the rest of the circle; with
// unsigned indices the modes below N turn through all of it.  Error against 64
// bits (largest of phi, Ex, Ey, mean of eight densities, 1e-7) of the block
// form, with unsigned indices, and now (with solve_pair's squares and up64):
//   512 x 256 2.25 2.25 1.95, 512 x 1024 2.28 2.47 2.09, 1024 x 512 2.16 2.41
//   1.80, 2048 x 1024 2.29 2.59 1.91, 2048 x 2048 2.04 2.30 1.84.
template <int N, int kSign>
__device__ __forceinline__ void group_fft(float2* buf, const float2* tws) {
  using F = GroupFft<N>;
  constexpr int E = F::kE, S = F::kStride, G = F::kG;
  constexpr int kBits = E == 32 ? 5 : E == 16 ? 4 : 3;
  const int l = threadIdx.x & (G - 1);
  float re[E], im[E];
  // stage 1: lane l holds x[n1 + G n2], n2 < E, with n1 = l in the lower half
  // and l - G in the upper; DFT along n2
  const int n1 = l < G / 2 ? l : l - G;
#pragma unroll
  for (int j = 0; j < E; j++) {
    const float2 v = buf[j ? n1 + G * j : n1 & (N - 1)];
    re[j] = v.x; im[j] = v.y;
  }
  dft_reg<E, kSign>(re, im);
  // twiddle W_N^(n1 k2), register r holding k2 = brev(r)
#pragma unroll
  for (int r = 1; r < E; r++) {
    float2 w = tws[brev<kBits>(r) * G + l];
    if (kSign > 0) w.y = -w.y;
    const float xr = re[r], xi = im[r];
    re[r] = xr * w.x - xi * w.y;
    im[r] = xr * w.y + xi * w.x;
  }
  group_sync<G>();
  float* tr = reinterpret_cast<float*>(buf);
  float* ti = tr + G * S;
#pragma unroll
  for (int r = 0; r < E; r++) {
    tr[l * S + brev<kBits>(r)] = re[r];
    ti[l * S + brev<kBits>(r)] = im[r];
  }
  group_sync<G>();
  if constexpr (G == E) {
    // stage 2: lane l takes the column of k2 = l or l - E, a G-point DFT,
    // X[k2 + E k1]
#pragma unroll
    for (int i = 0; i < G; i++) {
      re[i] = tr[i * S + l];
      im[i] = ti[i * S + l];
    }
    group_sync<G>();
    dft_reg<E, kSign>(re, im);
#pragma unroll
    for (int r = 0; r < E; r++) buf[r ? n1 + E * brev<kBits>(r) : n1 & (N - 1)] = make_float2(re[r], im[r]);
  } else if constexpr (E == 2 * G) {
    // stage 2: lane l takes the columns of k2 = l and l - G, a G-point DFT each
    constexpr int kBitsG = kBits - 1;
    float r2[2][G], i2[2][G];
#pragma unroll
    for (int h = 0; h < 2; h++)
#pragma unroll
      for (int i = 0; i < G; i++) {
        r2[h][i] = tr[i * S + l + G * h];
        i2[h][i] = ti[i * S + l + G * h];
      }
    group_sync<G>();
#pragma unroll
    for (int h = 0; h < 2; h++) {
      dft_reg<G, kSign>(r2[h], i2[h]);
#pragma unroll
      for (int r = 0; r < G; r++) {
        const int k = l - G * h;
        buf[r ? k + E * brev<kBitsG>(r) : k & (N - 1)] = make_float2(r2[h][r], i2[h][r]);
      }
    }
  } else {
    // stage 2 for G = 2 E: lane pair (2 c, 2 c + 1) takes the even and odd
    // lanes' elements of column c (k2 = c or c - E), one E-point DFT each, then
    // X[k] = E[k] + W^k O[k] (even lane) and X[k + E] = E[k] - W^k O[k] (odd
    // lane), W = W_G
    static_assert(G == 2 * E, "one or two lanes or columns");
    const int c = l >> 1, odd = l & 1, k2 = c < E / 2 ? c : c - E;
#pragma unroll
    for (int i = 0; i < E; i++) {
      re[i] = tr[(2 * i + odd) * S + c];
      im[i] = ti[(2 * i + odd) * S + c];
    }
    group_sync<G>();
    dft_reg<E, kSign>(re, im);
#pragma unroll
    for (int r = 0; r < E; r++) {
      const int k = brev<kBits>(r);
      const float pr = __shfl_xor_sync(0xffffffffu, re[r], 1);
      const float pi = __shfl_xor_sync(0xffffffffu, im[r], 1);
      // W^k O: O is the partner's value on the even lane, the own on the odd
      float orr = odd ? re[r] : pr, oi = odd ? im[r] : pi;
      rot64<kSign>(orr, oi, k * (64 / G));
      const float er = odd ? pr : re[r], ei = odd ? pi : im[r];
      const float xr = odd ? er - orr : er + orr, xi = odd ? ei - oi : ei + oi;
      const int at = k2 + E * (k + E * odd);
      buf[k ? at : at & (N - 1)] = make_float2(xr, xi);
    }
  }
  group_sync<G>();
}

// c0 + i c1 of a packed pair's DCT-III coefficients (dct3_pre of each): the
// pair's values at k and at n - k.
__device__ __forceinline__ float2 pre_pair(float2 ak, float2 ank, float2 w4, int k) {
  const float2 c0 = dct3_pre(ak.x, ank.x, w4, k);
  const float2 c1 = dct3_pre(ak.y, ank.y, w4, k);
  return make_float2(c0.x - c1.y, c0.y + c1.x);
}

// Density of every bin from the int64 areas, FP64 overflow partials (one per
// block) and the other area set cleared: pass A's first half.
__global__ void __launch_bounds__(256) k_poisson_dens(PassAArgs A) {
  __shared__ double red[32];
  const int nb = A.nx * A.ny;
  const int cur = A.ctl->area_cur;
  const unsigned long long* __restrict__ ar = cur == 0 ? A.area_pair[0] : A.area_pair[1];
  unsigned long long* __restrict__ ac = cur == 0 ? A.area_pair[1] : A.area_pair[0];
  const int64_t* __restrict__ np = A.nonplace;
  float* __restrict__ dens = A.density;
  float ovf = 0.0f;
#pragma unroll 4
  for (int b = blockIdx.x * 256 + threadIdx.x; b < nb; b += gridDim.x * 256) {
    const int j = b >> A.logn, i = b & (A.nx - 1);     // bin grids are powers of 2
    const int blx = A.core_lx + i * A.size_x, bux = min(blx + A.size_x, A.core_ux);
    const int bly = A.core_ly + j * A.size_y, buy = min(bly + A.size_y, A.core_uy);
    const long long bin_area = (long long)(bux - blx) * (long long)(buy - bly);
    const float cap = __fmul_rn(ll_to_float(bin_area), A.td);
    const float fi = ll_to_float((long long)ar[b]);
    const float ff = ll_to_float((long long)ar[nb + b]);
    const float fn = ll_to_float(np[b]);
    // BinGrid::updateBinsGCellDensityArea (src/nesterovBase.cpp:804-818)
    dens[b] = __fdiv_rn(__fadd_rn(__fadd_rn(fi, ff), fn), cap);
    ovf += fmaxf(0.0f, __fsub_rn(__fadd_rn(fi, fn), cap));
    ac[b] = 0ull;
    ac[nb + b] = 0ull;
  }
  if (A.part_overflow) block_reduce_add((double)ovf, &A.part_overflow[blockIdx.x], red);
}

// Copies n floats (n a multiple of 4, both pointers 16-byte aligned) with the
// block's 16-byte cp.async.
__device__ __forceinline__ void block_copy_async(float* dst, const float* src, int n) {
  for (int t = 4 * threadIdx.x; t < n; t += 4 * blockDim.x) cp_async16(dst + t, src + t);
}

// Pass A, group form: DCT-II along x of row pairs (density rows 2r, 2r + 1),
// one pair a group, two groups of 16 lanes or one of 32 or 64 a block.
// Shared memory: FFT buffers, the twiddle table.
template <int N>
struct RowsShape {
  static constexpr int kT = GroupFft<N>::kG < 32 ? 32 : GroupFft<N>::kG;
  static constexpr int kP = kT / GroupFft<N>::kG;       // row pairs per block
  static constexpr size_t kBytes = (size_t)kP * GroupFft<N>::kBuf * 4 + N * 8;
};

template <int N>
__global__ void __launch_bounds__(RowsShape<N>::kT) k_poisson_rows_g(PassAArgs A) {
  extern __shared__ float2 smem[];
  using F = GroupFft<N>;
  constexpr int G = F::kG, P = RowsShape<N>::kP;
  const int l = threadIdx.x & (G - 1), p = threadIdx.x / G;
  float2* buf = smem + (size_t)p * (F::kBuf / 2);
  float2* tws = smem + (size_t)P * (F::kBuf / 2);
  const int r = blockIdx.x * P + p;
  const float* d0 = (A.density_in ? A.density_in : A.density) + (size_t)(2 * r) * N;
  const float* d1 = d0 + N;
  // Makhoul order: v[m] = x[2m], v[n-1-m] = x[2m+1]
#pragma unroll 8
  for (int j = 0; j < N / G; j++) {
    const int i = l + G * j;
    float* dst = reinterpret_cast<float*>(&buf[makhoul_pos(i, N)]);
    cp_async4(dst, d0 + i);
    cp_async4(dst + 1, d1 + i);
  }
  block_copy_async(reinterpret_cast<float*>(tws), reinterpret_cast<const float*>(tw_table<N>()), 2 * N);
  cp_async_wait_all();
  __syncthreads();
  group_fft<N, -1>(buf, tws);
  float* s0 = A.spec + (size_t)(2 * r) * N;
  float* s1 = s0 + N;
#pragma unroll 8
  for (int j = 0; j < N / G; j++) {
    const int k = l + G * j;
    const float2 c = dct2_post(buf[k], buf[(N - k) & (N - 1)], __ldg(&A.w4[k]));
    s0[k] = c.x;
    s1[k] = c.y;
  }
}

// Pass B, group form: kP column pairs per block (2 kP adjacent columns; row
// segments of 32 bytes at kP = 4, 16 at 2) and two groups per pair: group
// (q, 0) takes the forward transform of pair q, both form the spectrum and
// the inputs of the two inverse transforms (elements k and n - k by one lane,
// in place), which run side by side on groups (q, 0) and (q, 1).
template <int N, int kP>
constexpr size_t cols_bytes() { return (size_t)2 * kP * GroupFft<N>::kBuf * 4 + N * 8; }

// phi^ of a packed column pair (u, u + 1) at row v from Z at v and n - v
// (src/fft.cpp:117-166): 4 / (nx ny) rho^ / (wx^2 + wy^2) with pi / nx taken
// out of the frequencies, so that the low modes, which carry the field, divide
// by u^2 + (wy[1] / wx[1])^2 v^2 of exact squares instead of squares of rounded
// multiples of pi.
__device__ __forceinline__ float2 solve_pair(const PassBArgs& B, float2 z, float2 zn, float2 w4, int u, int v) {
  const float2 a = dct2_post(z, zn, w4);
  const float vv = (float)(v * v);
  float out[2];
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float d = h ? a.y : a.x;
    if (u + h == 0) d *= 0.5f;
    if (v == 0) d *= 0.5f;
    d = __fmaf_rn(d, B.num[0], __fmul_rn(d, B.num[1]));
    const float den = __fmaf_rn(vv, B.aspect[0], __fmaf_rn(vv, B.aspect[1], (float)((u + h) * (u + h))));
    out[h] = (u + h != 0 || v != 0) ? __fdiv_rn(d, den) : 0.0f;
  }
  return make_float2(out[0], out[1]);
}

template <int N, int kP>
__global__ void __launch_bounds__(2 * kP * GroupFft<N>::kG) k_poisson_cols_g(PassBArgs B) {
  extern __shared__ float2 smem[];
  using F = GroupFft<N>;
  constexpr int G = F::kG, kT = 2 * kP * G, kH = kP / 2;
  constexpr int kBufF2 = F::kBuf / 2;
  // groups: role-major, so that a warp's groups have one role
  const int g = threadIdx.x / G, l = threadIdx.x & (G - 1);
  const int role = g / kP, q = g % kP;
  float2* buf0 = smem + (size_t)q * kBufF2;                       // forward, then P1
  float2* buf1 = smem + (size_t)(kP + q) * kBufF2;                // P2
  float2* tws = smem + (size_t)2 * kP * kBufF2;                   // [n] twiddles
  const int u_base = blockIdx.x * 2 * kP, u = u_base + 2 * q;
  const int nx = B.nx;
  // inputs: 8-byte copies of column pairs into the pairs' first buffers
  // (Makhoul order), and the twiddles
  for (int idx = threadIdx.x; idx < N * kP; idx += kT) {
    const int v = idx / kP, c = idx % kP;       // row v, pair c
    cp_async8(smem + (size_t)c * kBufF2 + makhoul_pos(v, N), B.spec + (size_t)v * nx + u_base + 2 * c);
  }
  block_copy_async(reinterpret_cast<float*>(tws), reinterpret_cast<const float*>(tw_table<N>()), 2 * N);
  cp_async_wait_all();
  __syncthreads();
  if (role == 0) group_fft<N, -1>(buf0, tws);
  __syncthreads();
  // spectrum, then P1 = IDCT_y(phi^) and P2 = IDST_y(wy phi^), a DCT-III of
  // b[k] = wy[n-k] phi^[n-k] (b[0] = 0): rows k and n - k of the pair
#pragma unroll 2
  for (int k = role * G + l; k < N / 2; k += 2 * G) {
    const int m = k ? N - k : N / 2;            // (0 and n / 2 stand alone)
    const float2 zk = buf0[k], zm = buf0[m];
    const float2 w4k = __ldg(&B.w4[k]), w4m = __ldg(&B.w4[m]);
    const float wk = __ldg(&B.wy[k]), wm = __ldg(&B.wy[m]);
    const float2 pk = solve_pair(B, zk, k ? zm : zk, w4k, u, k);
    const float2 pm = solve_pair(B, zm, k ? zk : zm, w4m, u, m);
    const float2 sk = make_float2(__fmul_rn(pk.x, wk), __fmul_rn(pk.y, wk));
    const float2 sm = make_float2(__fmul_rn(pm.x, wm), __fmul_rn(pm.y, wm));
    buf0[k] = pre_pair(pk, pm, w4k, k);
    buf0[m] = pre_pair(pm, k ? pk : pm, w4m, m);
    buf1[k] = k ? pre_pair(sm, sk, w4k, k) : make_float2(0.0f, 0.0f);
    buf1[m] = pre_pair(k ? sk : sm, sm, w4m, m);
  }
  __syncthreads();
  group_fft<N, 1>(role ? buf1 : buf0, tws);
  __syncthreads();
  // stores: P1 from the first buffers, P2 (signs alternating in v) from the
  // second ones; a thread writes four columns (two pairs) as a float4
  for (int idx = threadIdx.x; idx < N * kH * 2; idx += kT) {
    const int h = idx % kH, out = (idx / kH) & 1, v = idx / (2 * kH);
    const int m = makhoul_pos(v, N);
    const float2* b0 = smem + (size_t)(out * kP + 2 * h) * kBufF2;    // pair 2h
    const float2 x0 = b0[m], x1 = b0[kBufF2 + m];
    const float sg = (out && (v & 1)) ? -1.0f : 1.0f;
    float* dst = out ? B.p2 : B.p1;
    *reinterpret_cast<float4*>(dst + (size_t)v * nx + u_base + 4 * h) =
        make_float4(sg * x0.x, sg * x0.y, sg * x1.x, sg * x1.y);
  }
}

// Pass C, group form: kP row pairs per block and one group per transform of a
// pair (Ex = IDST_x(wx * P1), Ey = IDCT_x(P2) and, where it is wanted, phi =
// IDCT_x(P1)); the block writes the field (Ex, Ey per bin) once all
// transforms are done.
template <int N>
struct FieldShape {
  static constexpr int kP = N == 2048 ? 1 : N == 256 ? 4 : 2;
  static constexpr int threads(int roles) { return roles * kP * GroupFft<N>::kG; }
  static constexpr size_t bytes(int roles) { return (size_t)roles * kP * GroupFft<N>::kBuf * 4 + N * 8; }
};

template <int N>
__global__ void __launch_bounds__(FieldShape<N>::threads(3)) k_poisson_field_g(PassCArgs C) {
  extern __shared__ float2 smem[];
  using F = GroupFft<N>;
  constexpr int G = F::kG, kP = FieldShape<N>::kP;
  constexpr int kBufF2 = F::kBuf / 2;
  const int g = threadIdx.x / G, l = threadIdx.x & (G - 1);
  const int role = g / kP, p = g % kP;          // role 0 Ex, 1 Ey, 2 phi
  float2* buf = smem + (size_t)g * kBufF2;
  float2* tws = smem + (size_t)(blockDim.x / G) * kBufF2;
  const int r0 = blockIdx.x * kP;
  block_copy_async(reinterpret_cast<float*>(tws), reinterpret_cast<const float*>(tw_table<N>()), 2 * N);
  {
    const float* __restrict__ a0 = (role == 1 ? C.p2 : C.p1) + (size_t)(2 * (r0 + p)) * N;
    const float* __restrict__ a1 = a0 + N;
    constexpr int U = 4;                        // element pairs in flight per lane
    for (int k0 = l; k0 < N / 2; k0 += U * G) {
      float2 xk[U], xm[U], w4k[U], w4m[U];
      float wk[U], wm[U];
#pragma unroll
      for (int j = 0; j < U; j++) {
        const int k = k0 + j * G, m = k ? N - k : N / 2;
        xk[j] = make_float2(__ldg(a0 + k), __ldg(a1 + k));
        xm[j] = make_float2(__ldg(a0 + m), __ldg(a1 + m));
        w4k[j] = __ldg(&C.w4[k]);
        w4m[j] = __ldg(&C.w4[m]);
        if (role == 0) { wk[j] = __ldg(&C.wx[k]); wm[j] = __ldg(&C.wx[m]); }
      }
#pragma unroll
      for (int j = 0; j < U; j++) {
        const int k = k0 + j * G, m = k ? N - k : N / 2;
        if (role != 0) {
          buf[k] = pre_pair(xk[j], xm[j], w4k[j], k);
          buf[m] = pre_pair(xm[j], k ? xk[j] : xm[j], w4m[j], m);
        } else {
          // b[k] = wx[n-k] a[n-k] for k >= 1, b[0] = 0
          const float2 sk = make_float2(__fmul_rn(xk[j].x, wk[j]), __fmul_rn(xk[j].y, wk[j]));
          const float2 sm = make_float2(__fmul_rn(xm[j].x, wm[j]), __fmul_rn(xm[j].y, wm[j]));
          buf[k] = k ? pre_pair(sm, sk, w4k[j], k) : make_float2(0.0f, 0.0f);
          buf[m] = pre_pair(k ? sk : sm, sm, w4m[j], m);
        }
      }
    }
  }
  cp_async_wait_all();
  __syncthreads();
  group_fft<N, 1>(buf, tws);
  __syncthreads();
  // outputs, bin m of rows 2r and 2r + 1 of every pair (IDST signs alternate)
  for (int idx = threadIdx.x; idx < kP * N; idx += blockDim.x) {
    const int pp = idx / N, m = idx - pp * N;
    const size_t b0 = (size_t)(2 * (r0 + pp)) * N;
    const int mp = makhoul_pos(m, N);
    const float2* bp = smem + (size_t)pp * kBufF2;
    float2 ex = bp[mp];
    const float2 ey = bp[kP * kBufF2 + mp];
    if (m & 1) { ex.x = -ex.x; ex.y = -ex.y; }
    if (C.field) {
      C.field[b0 + m] = make_float2(ex.x, ey.x);
      C.field[b0 + N + m] = make_float2(ex.y, ey.y);
    } else {
      C.fx[b0 + m] = ex.x; C.fx[b0 + N + m] = ex.y;
      C.fy[b0 + m] = ey.x; C.fy[b0 + N + m] = ey.y;
    }
    if (C.phi) {
      const float2 ph = bp[2 * kP * kBufF2 + mp];
      C.phi[b0 + m] = ph.x; C.phi[b0 + N + m] = ph.y;
    }
  }
}

// ---------------------------------------------------------------------------
// Cluster form, for 64 x 64, 128 x 128 and 256 x 256 grids given as densities
// (gpl_poisson_solve): the whole solve in one launch of one cluster of 16
// CTAs.  On these grids each of the three passes is bound by its launch and
// one round trip to memory (7 us a pass whatever the size, for 0.04 us of
// bytes), so the passes become phases of one kernel and the transposes
// between them go through distributed shared memory: CTA c transforms rows
// [c N/16, (c + 1) N/16), writes each spectrum element into the shared memory
// of its column's owner, that CTA solves its columns and writes P1 and P2
// back to the rows' owners.  Group FFTs as above (8 or 16 lanes a pair);
// elements k and n - k by one thread, in place.
// Solve with the potential: 64 x 64 19.5 -> 6.2 us, 128 x 128 20.5 -> 10.3,
// 256 x 256 22.6 -> 18.4.  Jobs keep the block form on these grids.  Another
// rounding of the field changes a job's placement (a loop amplifies it: single
// cells of 10k-cell designs move by up to 1e-3 of the core in 64 iterations),
// so a job's form changes only where its loop gains much: the group form is
// taken on 512 x 256 (89 -> 46 us an iteration at 10k cells) and up, this one,
// for 6 % of a 10k-cell loop, is not.
constexpr int kClCtas = 16;

template <int N>
struct ClusterShape {
  static constexpr int kT = N >= 128 ? 512 : 256;          // threads per CTA
  static constexpr int kP = N / (2 * kClCtas);             // row pairs, and column pairs, per CTA
  static constexpr int kBufF2 = GroupFft<N>::kBuf / 2;
  // three row buffers (Ex, P1, P2) and two column buffers a pair, twiddles
  static constexpr size_t kBytes = ((size_t)5 * kP * kBufF2 + N) * sizeof(float2);
};

// f(task) for task < n by the block's groups of G lanes
template <int G, int kT, class F>
__device__ __forceinline__ void group_tasks(int n, F f) {
  for (int t = threadIdx.x / G; t < n; t += kT / G) f(t);
}

template <int N>
__global__ void __cluster_dims__(kClCtas, 1, 1) __launch_bounds__(ClusterShape<N>::kT)
    k_poisson_cluster(const __grid_constant__ PassAArgs A, const __grid_constant__ PassBArgs B,
                      const __grid_constant__ PassCArgs C) {
  extern __shared__ float2 smem[];
  using F = GroupFft<N>;
  constexpr int G = F::kG, kP = ClusterShape<N>::kP, kBufF2 = ClusterShape<N>::kBufF2;
  constexpr int kT = ClusterShape<N>::kT;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), tid = threadIdx.x;
  float2* rowx = smem;                                     // [kP] density pairs, then Ex
  float2* row1 = rowx + kP * kBufF2;                       // [kP] P1 of row pairs
  float2* row2 = row1 + kP * kBufF2;                       // [kP] P2
  float2* col0 = row2 + kP * kBufF2;                       // [kP] spectrum of column pairs, then P1
  float2* col1 = col0 + kP * kBufF2;                       // [kP] P2
  float2* tws = col1 + kP * kBufF2;
  for (int t = tid; t < N; t += kT) tws[t] = __ldg(tw_table<N>() + t);
  // rows in Makhoul order
  const int j0 = rank * 2 * kP;
  for (int idx = tid; idx < 2 * kP * N; idx += kT) {
    const int h = idx / N, i = idx & (N - 1);
    float* slot = reinterpret_cast<float*>(&rowx[(h >> 1) * kBufF2 + makhoul_pos(i, N)]);
    slot[h & 1] = __ldg(&A.density_in[(j0 + h) * N + i]);
  }
  // every CTA of the cluster has started (its shared memory may be written)
  cl.sync();
  group_tasks<G, kT>(kP, [&](int p) { group_fft<N, -1>(rowx + p * kBufF2, tws); });
  __syncthreads();
  // DCT-II along x, each column pair to its owner (Makhoul order along y)
  for (int idx = tid; idx < kP * N; idx += kT) {
    const int p = idx / N, k = idx & (N - 1);
    const float2* z = rowx + p * kBufF2;
    const float2 c = dct2_post(z[k], z[(N - k) & (N - 1)], __ldg(&A.w4[k]));
    float2* col = cl.map_shared_rank(col0, k / (2 * kP)) + ((k >> 1) & (kP - 1)) * kBufF2;
    // a lane pair holds columns k, k + 1 of rows v, v + 1: one row each
    const int odd = k & 1, v = j0 + 2 * p + odd;
    const float got = __shfl_xor_sync(0xffffffffu, odd ? c.x : c.y, 1);
    col[makhoul_pos(v, N)] = odd ? make_float2(got, c.y) : make_float2(c.x, got);
  }
  cl.sync();
  // columns: DCT-II along y, the spectral solve, P1 = IDCT_y(phi^) and P2 =
  // IDST_y(wy phi^), as in the group form's pass B
  group_tasks<G, kT>(kP, [&](int q) { group_fft<N, -1>(col0 + q * kBufF2, tws); });
  __syncthreads();
  const int u0 = rank * 2 * kP;
  for (int idx = tid; idx < kP * (N / 2); idx += kT) {
    const int q = idx / (N / 2), k = idx & (N / 2 - 1), m = k ? N - k : N / 2, u = u0 + 2 * q;
    float2* buf0 = col0 + q * kBufF2;
    float2* buf1 = col1 + q * kBufF2;
    const float2 zk = buf0[k], zm = buf0[m];
    const float2 w4k = __ldg(&B.w4[k]), w4m = __ldg(&B.w4[m]);
    const float wk = __ldg(&B.wy[k]), wm = __ldg(&B.wy[m]);
    const float2 pk = solve_pair(B, zk, k ? zm : zk, w4k, u, k);
    const float2 pm = solve_pair(B, zm, k ? zk : zm, w4m, u, m);
    const float2 sk = make_float2(__fmul_rn(pk.x, wk), __fmul_rn(pk.y, wk));
    const float2 sm = make_float2(__fmul_rn(pm.x, wm), __fmul_rn(pm.y, wm));
    buf0[k] = pre_pair(pk, pm, w4k, k);
    buf0[m] = pre_pair(pm, k ? pk : pm, w4m, m);
    buf1[k] = k ? pre_pair(sm, sk, w4k, k) : make_float2(0.0f, 0.0f);
    buf1[m] = pre_pair(k ? sk : sm, sm, w4m, m);
  }
  __syncthreads();
  group_tasks<G, kT>(2 * kP, [&](int t) { group_fft<N, 1>(col0 + t * kBufF2, tws); });   // col1 follows col0
  __syncthreads();
  for (int idx = tid; idx < kP * N; idx += kT) {
    const int q = idx & (kP - 1), v = idx / kP, m = makhoul_pos(v, N), u = u0 + 2 * q;
    const float2 a = col0[q * kBufF2 + m];
    float2 b = col1[q * kBufF2 + m];
    if (v & 1) { b.x = -b.x; b.y = -b.y; }
    // lanes kP apart hold rows v, v + 1 of columns u, u + 1: one column each
    const int odd = v & 1, owner = v / (2 * kP), at = ((v >> 1) & (kP - 1)) * kBufF2 + u + odd;
    const float ga = __shfl_xor_sync(0xffffffffu, odd ? a.x : a.y, kP);
    const float gb = __shfl_xor_sync(0xffffffffu, odd ? b.x : b.y, kP);
    cl.map_shared_rank(row1, owner)[at] = odd ? make_float2(ga, a.y) : make_float2(a.x, ga);
    cl.map_shared_rank(row2, owner)[at] = odd ? make_float2(gb, b.y) : make_float2(b.x, gb);
  }
  cl.sync();
  // rows: Ex = IDST_x(wx P1), Ey = IDCT_x(P2), phi = IDCT_x(P1)
  for (int idx = tid; idx < kP * (N / 2); idx += kT) {
    const int p = idx / (N / 2), k = idx & (N / 2 - 1), m = k ? N - k : N / 2;
    const float2 w4k = __ldg(&C.w4[k]), w4m = __ldg(&C.w4[m]);
    const float wk = __ldg(&C.wx[k]), wm = __ldg(&C.wx[m]);
    const float2 pk = row1[p * kBufF2 + k], pm = row1[p * kBufF2 + m];
    const float2 yk = row2[p * kBufF2 + k], ym = row2[p * kBufF2 + m];
    const float2 sk = make_float2(__fmul_rn(pk.x, wk), __fmul_rn(pk.y, wk));
    const float2 sm = make_float2(__fmul_rn(pm.x, wm), __fmul_rn(pm.y, wm));
    rowx[p * kBufF2 + k] = k ? pre_pair(sm, sk, w4k, k) : make_float2(0.0f, 0.0f);
    rowx[p * kBufF2 + m] = pre_pair(k ? sk : sm, sm, w4m, m);
    row2[p * kBufF2 + k] = pre_pair(yk, ym, w4k, k);
    row2[p * kBufF2 + m] = pre_pair(ym, k ? yk : ym, w4m, m);
    if (C.phi) {
      row1[p * kBufF2 + k] = pre_pair(pk, pm, w4k, k);
      row1[p * kBufF2 + m] = pre_pair(pm, k ? pk : pm, w4m, m);
    }
  }
  __syncthreads();
  // tasks: Ex and Ey of every pair, then phi
  group_tasks<G, kT>(C.phi ? 3 * kP : 2 * kP, [&](int t) {
    float2* buf = t < kP ? rowx + t * kBufF2 : t < 2 * kP ? row2 + (t - kP) * kBufF2 : row1 + (t - 2 * kP) * kBufF2;
    group_fft<N, 1>(buf, tws);
  });
  __syncthreads();
  for (int idx = tid; idx < kP * N; idx += kT) {
    const int p = idx / N, i = idx & (N - 1), m = makhoul_pos(i, N);
    const int b = (j0 + 2 * p) * N + i;
    float2 ex = rowx[p * kBufF2 + m];
    const float2 ey = row2[p * kBufF2 + m];
    if (i & 1) { ex.x = -ex.x; ex.y = -ex.y; }
    if (C.field) {
      C.field[b] = make_float2(ex.x, ey.x);
      C.field[b + N] = make_float2(ex.y, ey.y);
    } else {
      C.fx[b] = ex.x; C.fx[b + N] = ex.y;
      C.fy[b] = ey.x; C.fy[b + N] = ey.y;
    }
    if (C.phi) {
      const float2 ph = row1[p * kBufF2 + m];
      C.phi[b] = ph.x; C.phi[b + N] = ph.y;
    }
  }
}

template <int N>
bool cluster_prepare() {
  const int bytes = (int)ClusterShape<N>::kBytes;
  const void* f = (const void*)k_poisson_cluster<N>;
  bool ok = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess &&
            cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(kClCtas);
  c.blockDim = dim3(ClusterShape<N>::kT);
  c.dynamicSmemBytes = bytes;
  int num = 0;
  ok = ok && cudaOccupancyMaxActiveClusters(&num, k_poisson_cluster<N>, &c) == cudaSuccess && num > 0;
  if (!ok) cudaGetLastError();
  return ok;
}

// Whether the cluster form takes this grid, where it can be placed at all.
bool cluster_grid(int nx, int ny) { return nx == ny && (nx == 64 || nx == 128 || nx == 256); }

// Whether the group form takes this grid.
bool group_form(int nx, int ny) {
  auto in = [](int n) { return n == 256 || n == 512 || n == 1024 || n == 2048; };
  return in(nx) && in(ny) && !(nx == 256 && ny == 256);
}

template <int N>
void launch_rows_g(const PassAArgs& A, int ny, cudaStream_t s) {
  using R = RowsShape<N>;
  k_poisson_rows_g<N><<<ny / 2 / R::kP, R::kT, R::kBytes, s>>>(A);
}
template <int N>
void launch_cols_g(const PassBArgs& B, int nx, cudaStream_t s) {
  // 32-byte row segments where that leaves 128 blocks (most of the SMs)
  if (nx >= 1024) k_poisson_cols_g<N, 4><<<nx / 8, 8 * GroupFft<N>::kG, cols_bytes<N, 4>(), s>>>(B);
  else k_poisson_cols_g<N, 2><<<nx / 4, 4 * GroupFft<N>::kG, cols_bytes<N, 2>(), s>>>(B);
}
template <int N>
void launch_field_g(const PassCArgs& C, int ny, cudaStream_t s) {
  using S = FieldShape<N>;
  const int roles = C.phi ? 3 : 2;
  k_poisson_field_g<N><<<ny / 2 / S::kP, S::threads(roles), S::bytes(roles), s>>>(C);
}

template <int N>
cudaError_t group_prepare() {
  const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
  cudaError_t e = cudaFuncSetAttribute(k_poisson_rows_g<N>, a, (int)RowsShape<N>::kBytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_poisson_cols_g<N, 4>, a, (int)cols_bytes<N, 4>());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_poisson_cols_g<N, 2>, a, (int)cols_bytes<N, 2>());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_poisson_field_g<N>, a, (int)FieldShape<N>::bytes(3));
  return e;
}

int ilog2(int v) { int l = 0; while ((1 << l) < v) l++; return l; }

}  // namespace

// Row (column) pairs per block: as few as keep 256 threads busy, so that the
// grid has up to kMinPoissonBlocks blocks (several per SM) to hide the
// latency of the loads; small grids are spread over SMs instead of being
// serialised in a few blocks.
constexpr int kMinPoissonBlocks = 512;
int pairs_a(int nx, int ny) { return max(1, min(min(ny / 2, 2048 / nx), (ny / 2) / kMinPoissonBlocks)); }
int pairs_b(int nx, int ny) {
  return max(1, min(min(nx / 2, min(4, 4096 / ny)), (nx / 2) / kMinPoissonBlocks));
}
int pairs_c(int nx, int ny) { return pairs_a(nx, ny); }

size_t smem_a(int nx, int ny) { return ((size_t)2 * pairs_a(nx, ny) * nx + nx / 2) * sizeof(float2); }
size_t smem_b(int nx, int ny) { return ((size_t)3 * pairs_b(nx, ny) * ny + ny / 2) * sizeof(float2); }
size_t smem_c(int nx, int ny) { return ((size_t)4 * pairs_c(nx, ny) * nx + nx / 2) * sizeof(float2); }

// Blocks of the density pass (one FP64 overflow partial each): the group
// form's grid-wide density kernel takes four bins per thread, more on grids
// of over a million bins (a partial per block has to fit part_stride).
int poisson_blocks_a(int nx, int ny) {
  if (group_form(nx, ny)) return min(nx * ny / 1024, 1024);
  int r = pairs_a(nx, ny);
  return (ny / 2 + r - 1) / r;
}

namespace {
// What a context holds for the Poisson kernels besides their shared-memory
// limits and twiddle tables.
struct PoissonContext {
  bool cluster = false;   // 16 CTAs (above the portable size) can be placed; otherwise the block form stays
};

int poisson_context(PoissonContext* out) {
  static PerContext<PoissonContext> contexts;
  return contexts.get(out, [](PoissonContext& pc) -> int {
    const int big = 200 * 1024;
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_a, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_b, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_c, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    GPL_CUDA(group_prepare<256>());
    GPL_CUDA(group_prepare<512>());
    GPL_CUDA(group_prepare<1024>());
    GPL_CUDA(group_prepare<2048>());
    pc.cluster = cluster_prepare<64>() && cluster_prepare<128>() && cluster_prepare<256>();
    for (int n : {64, 128, 256, 512, 1024, 2048}) {
      // the group form's twiddles (indices of either sign, see group_fft)
      const int g = n <= 128 ? GroupFft<64>::kG : n == 256 ? GroupFft<256>::kG : n == 2048 ? GroupFft<2048>::kG : GroupFft<512>::kG;
      static_assert(GroupFft<512>::kG == GroupFft<1024>::kG && GroupFft<64>::kG == GroupFft<128>::kG, "one width");
      std::vector<float2> t(n);
      const int e = n / g;
      for (int k2 = 0; k2 < e; k2++)
        for (int n1 = 0; n1 < g; n1++) {
          const int m = (n1 < g / 2 ? n1 : n1 - g) * (k2 < e / 2 ? k2 : k2 - e);
          const double a = -2.0 * M_PI * (double)m / (double)n;
          t[k2 * g + n1] = make_float2((float)cos(a), (float)sin(a));
        }
      const size_t bytes = n * sizeof(float2);
      if (n == 64) GPL_CUDA(cudaMemcpyToSymbol(g_tw64, t.data(), bytes));
      else if (n == 128) GPL_CUDA(cudaMemcpyToSymbol(g_tw128, t.data(), bytes));
      else if (n == 256) GPL_CUDA(cudaMemcpyToSymbol(g_tw256, t.data(), bytes));
      else if (n == 512) GPL_CUDA(cudaMemcpyToSymbol(g_tw512, t.data(), bytes));
      else if (n == 1024) GPL_CUDA(cudaMemcpyToSymbol(g_tw1024, t.data(), bytes));
      else GPL_CUDA(cudaMemcpyToSymbol(g_tw2048, t.data(), bytes));
    }
    // (a copy from pageable memory may return before it has arrived, and a
    // caller's non-blocking stream does not wait for it)
    GPL_CUDA(cudaStreamSynchronize(nullptr));
    return GPL_OK;
  });
}
}  // namespace

int poisson_prepare_device() {
  PoissonContext pc;
  return poisson_context(&pc);
}

namespace {
// Passes B and C of the block form, with the grids and dynamic shared memory
// of passes A, B and C.
void block_form_bc(const PoissonGrid& g, float* spec, float* p1, float* p2, float2* field, float* fx,
                   float* fy, float* phi, PassBArgs& B, PassCArgs& C, int grid[3], size_t smem[3]) {
  const int nx = g.nx, ny = g.ny;
  B.nx = nx; B.ny = ny; B.logn = ilog2(ny); B.col_pairs = pairs_b(nx, ny);
  B.spec = spec; B.p1 = p1; B.p2 = p2; B.wx = g.wx; B.wy = g.wy; B.tw = g.tw; B.w4 = g.w4y;
  B.scale = 4.0f / (float)nx / (float)ny;
  C.nx = nx; C.ny = ny; C.logn = ilog2(nx); C.pairs_per_block = pairs_c(nx, ny);
  C.p1 = p1; C.p2 = p2; C.field = field; C.fx = fx; C.fy = fy; C.phi = phi;
  C.wx = g.wx; C.tw = g.tw; C.w4 = g.w4x;
  grid[0] = poisson_blocks_a(nx, ny);
  grid[1] = nx / (2 * B.col_pairs);
  grid[2] = (ny / 2 + C.pairs_per_block - 1) / C.pairs_per_block;
  smem[0] = smem_a(nx, ny);
  smem[1] = smem_b(nx, ny);
  smem[2] = smem_c(nx, ny);
}

// solve_pair's constants.
void solve_constants(const PoissonGrid& g, PassBArgs& B) {
  const double r = (double)g.nx / g.ny * ((double)g.size_y / g.size_x);
  const double num = 4.0 * g.nx / (g.ny * M_PI * M_PI), aspect = r * r;
  B.scale = 0.0f;
  B.num[0] = (float)num;
  B.num[1] = (float)(num - B.num[0]);
  B.aspect[0] = (float)aspect;
  B.aspect[1] = (float)(aspect - B.aspect[0]);
}

PassAArgs pass_a_args(const PoissonGrid& g, unsigned long long* const* area_pair, const EvalCtl* ctl,
                      const int64_t* nonplace, float td, const float* density_in, float* density,
                      double* part_overflow, float* spec) {
  PassAArgs A;
  A.nx = g.nx; A.ny = g.ny; A.logn = ilog2(g.nx); A.pairs_per_block = pairs_a(g.nx, g.ny);
  A.core_lx = g.core_lx; A.core_ly = g.core_ly; A.core_ux = g.core_ux; A.core_uy = g.core_uy;
  A.size_x = g.size_x; A.size_y = g.size_y; A.td = td;
  A.area_pair[0] = area_pair ? area_pair[0] : nullptr;
  A.area_pair[1] = area_pair ? area_pair[1] : nullptr;
  A.ctl = ctl; A.nonplace = nonplace;
  A.density_in = density_in; A.density = density; A.spec = spec;
  A.part_overflow = part_overflow; A.tw = g.tw; A.w4 = g.w4x;
  return A;
}

PoissonGrid job_grid(const DeviceModel& d) {
  PoissonGrid g;
  g.nx = d.cnt_x; g.ny = d.cnt_y; g.size_x = d.size_x; g.size_y = d.size_y;
  g.core_lx = d.core_lx; g.core_ly = d.core_ly; g.core_ux = d.core_ux; g.core_uy = d.core_uy;
  g.wx = d.wx; g.wy = d.wy; g.w4x = d.w4x; g.w4y = d.w4y; g.tw = d.twiddle;
  return g;
}

// Batched form of the block passes: work items (instance, block); each
// block runs the per-job kernel's body on its instance's arguments.
__global__ void __launch_bounds__(256) k_poisson_a_batch(const PassAArgs* args, const int4* items, const int* count) {
  extern __shared__ float2 smem[];
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    poisson_a_body(args[it.x], it.y, smem);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_poisson_b_batch(const PassBArgs* args, const int4* items, const int* count) {
  extern __shared__ float2 smem[];
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    poisson_b_body(args[it.x], it.y, smem);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_poisson_c_batch(const PassCArgs* args, const int4* items, const int* count) {
  extern __shared__ float2 smem[];
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    poisson_c_body(args[it.x], it.y, smem);
    __syncthreads();
  }
}
}  // namespace

size_t poisson_batch_args_bytes(int pass) {
  // the element size of the device arrays the batched kernels index
  return pass == 0 ? sizeof(PassAArgs) : pass == 1 ? sizeof(PassBArgs) : sizeof(PassCArgs);
}

bool write_poisson_batch_args(const DeviceModel& d, void* dst_a, void* dst_b, void* dst_c, int grid[3],
                              size_t smem[3]) {
  if (d.poisson_path != 1 || group_form(d.cnt_x, d.cnt_y)) return false;
  const PoissonGrid g = job_grid(d);
  const PassAArgs A = pass_a_args(g, d.area, d.ctl, d.nonplace, d.target_density, nullptr, d.density,
                                  d.part + (size_t)kPartOverflow * d.part_stride, d.spec);
  PassBArgs B;
  PassCArgs C;
  block_form_bc(g, d.spec, d.p1, d.p2, d.field, nullptr, nullptr, nullptr, B, C, grid, smem);
  memcpy(dst_a, &A, sizeof(A));
  memcpy(dst_b, &B, sizeof(B));
  memcpy(dst_c, &C, sizeof(C));
  return true;
}

int poisson_batch_prepare_device() {
  static PerContext<char> contexts;
  char done;
  return contexts.get(&done, [](char&) -> int {
    const int big = 200 * 1024;
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_a_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_b_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    GPL_CUDA(cudaFuncSetAttribute(k_poisson_c_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
    return GPL_OK;
  });
}

int launch_poisson_batch(int pass, const void* args, const int4* items, const int* count, int grid, size_t smem,
                         cudaStream_t s) {
  if (pass == 0) k_poisson_a_batch<<<grid, 256, smem, s>>>(static_cast<const PassAArgs*>(args), items, count);
  else if (pass == 1) k_poisson_b_batch<<<grid, 256, smem, s>>>(static_cast<const PassBArgs*>(args), items, count);
  else k_poisson_c_batch<<<grid, 256, smem, s>>>(static_cast<const PassCArgs*>(args), items, count);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

// The three passes on arbitrary device arrays.  Area mode (area != null):
// the density comes from the int64 areas; otherwise from density_in.
int poisson_passes(const PoissonGrid& g, unsigned long long* const* area_pair,
                   const EvalCtl* ctl, const int64_t* nonplace, float td,
                   const float* density_in, float* density, double* part_overflow,
                   float* spec, float* p1, float* p2, float2* field, float* fx, float* fy,
                   float* phi, cudaStream_t s, Timer* t) {
  PoissonContext pc;
  int rc = poisson_context(&pc);
  if (rc) return rc;
  const int nx = g.nx, ny = g.ny;
  const PassAArgs A = pass_a_args(g, area_pair, ctl, nonplace, td, density_in, density, part_overflow, spec);
  if (group_form(nx, ny)) {
    const bool areas = area_pair && ctl;
    PassBArgs B;
    B.nx = nx; B.ny = ny; B.logn = ilog2(ny); B.col_pairs = 0;
    B.spec = spec; B.p1 = p1; B.p2 = p2; B.wx = g.wx; B.wy = g.wy; B.tw = g.tw; B.w4 = g.w4y;
    solve_constants(g, B);
    PassCArgs C;
    C.nx = nx; C.ny = ny; C.logn = ilog2(nx); C.pairs_per_block = 0;
    C.p1 = p1; C.p2 = p2; C.field = field; C.fx = fx; C.fy = fy; C.phi = phi;
    C.wx = g.wx; C.tw = g.tw; C.w4 = g.w4x;
    if (t) t->begin(kKPoissonA);
    if (areas) k_poisson_dens<<<poisson_blocks_a(nx, ny), 256, 0, s>>>(A);
    if (nx == 256) launch_rows_g<256>(A, ny, s);
    else if (nx == 512) launch_rows_g<512>(A, ny, s);
    else if (nx == 1024) launch_rows_g<1024>(A, ny, s);
    else launch_rows_g<2048>(A, ny, s);
    if (t) t->end(kKPoissonA);
    if (t) t->begin(kKPoissonB);
    if (ny == 256) launch_cols_g<256>(B, nx, s);
    else if (ny == 512) launch_cols_g<512>(B, nx, s);
    else if (ny == 1024) launch_cols_g<1024>(B, nx, s);
    else launch_cols_g<2048>(B, nx, s);
    if (t) t->end(kKPoissonB);
    if (t) t->begin(kKPoissonC);
    if (nx == 256) launch_field_g<256>(C, ny, s);
    else if (nx == 512) launch_field_g<512>(C, ny, s);
    else if (nx == 1024) launch_field_g<1024>(C, ny, s);
    else launch_field_g<2048>(C, ny, s);
    if (t) t->end(kKPoissonC);
    if (t) t->count(areas ? 4 : 3);
    GPL_CUDA(cudaGetLastError());
    return GPL_OK;
  }
  if (density_in && pc.cluster && cluster_grid(nx, ny)) {
    PassBArgs B;
    PassCArgs C;
    int grid[3];
    size_t smem[3];
    block_form_bc(g, spec, p1, p2, field, fx, fy, phi, B, C, grid, smem);
    solve_constants(g, B);
    if (t) t->begin(kKPoissonB);
    if (nx == 64) k_poisson_cluster<64><<<kClCtas, ClusterShape<64>::kT, ClusterShape<64>::kBytes, s>>>(A, B, C);
    else if (nx == 128) k_poisson_cluster<128><<<kClCtas, ClusterShape<128>::kT, ClusterShape<128>::kBytes, s>>>(A, B, C);
    else k_poisson_cluster<256><<<kClCtas, ClusterShape<256>::kT, ClusterShape<256>::kBytes, s>>>(A, B, C);
    if (t) t->end(kKPoissonB);
    if (t) t->count(1);
    GPL_CUDA(cudaGetLastError());
    return GPL_OK;
  }
  PassBArgs B;
  PassCArgs C;
  int grid[3];
  size_t smem[3];
  block_form_bc(g, spec, p1, p2, field, fx, fy, phi, B, C, grid, smem);
  if (t) t->begin(kKPoissonA);
  k_poisson_a<<<grid[0], 256, smem[0], s>>>(A);
  if (t) t->end(kKPoissonA);
  if (t) t->begin(kKPoissonB);
  k_poisson_b<<<grid[1], 256, smem[1], s>>>(B);
  if (t) t->end(kKPoissonB);
  if (t) t->begin(kKPoissonC);
  k_poisson_c<<<grid[2], 256, smem[2], s>>>(C);
  if (t) t->end(kKPoissonC);
  if (t) t->count(3);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

int launch_poisson_job(DeviceModel& d, bool want_phi, cudaStream_t s, Timer& t) {
  if (d.poisson_path == 2 && d.pg) return launch_poisson_gemm(d, d.pg, want_phi, s, t);
  const PoissonGrid g = job_grid(d);
  return poisson_passes(g, d.area, d.ctl, d.nonplace, d.target_density, nullptr, d.density,
                        d.part + (size_t)kPartOverflow * d.part_stride, d.spec, d.p1, d.p2,
                        d.field, nullptr, nullptr, want_phi ? d.phi : nullptr, s, &t);
}

void make_w4(int n, std::vector<float2>& w) {
  w.resize(n);
  for (int k = 0; k < n; k++) {
    double a = -M_PI * (double)k / (2.0 * n);
    w[k] = make_float2((float)cos(a), (float)sin(a));
  }
}

// Scratch and tables of the standalone solve, cached per (device, grid).  The
// scratch carries a solve's spectrum from pass to pass, so solves that may run
// at once need their own: the first stream that solves a grid owns an entry,
// whose solves its own order keeps apart, and all other streams share a second
// one, where a solve waits on the GPU for the one before it.  (One entry whose
// solves always wait costs a caller of one stream the event calls, 1.5 us of
// the 35 of a single solve.)
namespace {
struct SolveCache {
  int device = -1, nx = 0, ny = 0, bsx = 0, bsy = 0;
  unsigned long long ctx = 0;   // context the memory belongs to
  unsigned long long owner = 0; // id of the owning stream (never reused)
  bool shared = false;          // the other streams' entry
  std::mutex mu;                // held while a solve is enqueued
  cudaEvent_t done = nullptr;   // shared: behind the last solve
  char* mem = nullptr;
  float *spec = nullptr, *p1 = nullptr, *p2 = nullptr, *wx = nullptr, *wy = nullptr;
  float2 *w4x = nullptr, *w4y = nullptr, *tw = nullptr;
};
std::mutex g_cache_mu;
std::vector<std::shared_ptr<SolveCache>> g_cache;

typedef CUresult (*CtxGetCurrentFn)(CUcontext*);
typedef CUresult (*CtxGetIdFn)(CUcontext, unsigned long long*);
}  // namespace

unsigned long long current_context_id() {
  static CtxGetCurrentFn get_cur = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_cur = reinterpret_cast<CtxGetCurrentFn>(f);
    f = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) ==
            cudaSuccess && q == cudaDriverEntryPointSuccess)
      get_id = reinterpret_cast<CtxGetIdFn>(f);
  });
  CUcontext c = nullptr;
  unsigned long long id = 0;
  if (!get_cur || !get_id || get_cur(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0;
  return id;
}

}  // namespace gpl

using namespace gpl;

extern "C" gpl_status gpl_poisson_solve(int32_t nx, int32_t ny, int32_t bsx, int32_t bsy,
                                        const float* density, float* phi, float* fx, float* fy,
                                        void* stream) {
  auto pow2 = [](int v) { return v >= 2 && v <= kFftMax && (v & (v - 1)) == 0; };
  if (!pow2(nx) || !pow2(ny) || bsx <= 0 || bsy <= 0 || !density || !fx || !fy) {
    set_error("gpl_poisson_solve: sizes must be powers of two in [2, 4096], bin sizes positive, "
              "density/field pointers non-null");
    return GPL_ERR_INVALID_ARG;
  }
  int dev = 0;
  GPL_CUDA(cudaGetDevice(&dev));
  GPL_CUDA(cudaSetDevice(dev));         // initialises the device's context if needed
  const unsigned long long ctx = current_context_id();
  cudaStream_t s = (cudaStream_t)stream;
  // a captured solve takes the entry that is there (no allocation and no wait
  // for work outside the capture): the header leaves its order to the caller
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  GPL_CUDA(cudaStreamIsCapturing(s, &capture));
  const bool capturing = capture != cudaStreamCaptureStatusNone;
  unsigned long long sid = 0;
  if (!capturing) GPL_CUDA(cudaStreamGetId(s, &sid));
  std::shared_ptr<SolveCache> c;
  {
    std::lock_guard<std::mutex> lk(g_cache_mu);
    // entries of a context that no longer exists (cudaDeviceReset) hold
    // memory that went with it: forget them without freeing
    for (auto& e : g_cache)
      if (e && e->device == dev && e->ctx != ctx) e.reset();
    g_cache.erase(std::remove(g_cache.begin(), g_cache.end(), nullptr), g_cache.end());
    std::shared_ptr<SolveCache> owned, others;         // another stream's, the shared one
    for (auto& e : g_cache) {
      if (e->device != dev || e->nx != nx || e->ny != ny || e->bsx != bsx || e->bsy != bsy) continue;
      if (e->shared) others = e;
      else if (e->owner == sid) c = e;
      else owned = e;
    }
    if (!c) c = capturing && owned ? owned : others;
    if (!c) {
      auto n = std::make_shared<SolveCache>();
      SolveCache& e = *n;
      e.device = dev; e.ctx = ctx; e.nx = nx; e.ny = ny; e.bsx = bsx; e.bsy = bsy;
      e.shared = owned != nullptr;
      e.owner = sid;
      const size_t nb = (size_t)nx * ny;
      size_t bytes = 3 * nb * 4 + (nx + ny) * 4 + (nx + ny) * 8 + (kFftMax / 2) * 8 + 8 * 256;
      GPL_CUDA(cudaMalloc(&e.mem, bytes));
      char* q = e.mem;
      auto take = [&](size_t b) { char* r = q; q += ((b + 255) / 256) * 256; return r; };
      e.spec = (float*)take(nb * 4); e.p1 = (float*)take(nb * 4); e.p2 = (float*)take(nb * 4);
      e.wx = (float*)take(nx * 4); e.wy = (float*)take(ny * 4);
      e.w4x = (float2*)take(nx * 8); e.w4y = (float2*)take(ny * 8);
      e.tw = (float2*)take((kFftMax / 2) * 8);
      std::vector<float2> tw, w4x, w4y;
      std::vector<float> wx, wy;
      make_twiddle(tw); make_w4(nx, w4x); make_w4(ny, w4y); make_freq(nx, ny, bsx, bsy, wx, wy);
      GPL_CUDA(cudaMemcpy(e.wx, wx.data(), nx * 4, cudaMemcpyHostToDevice));
      GPL_CUDA(cudaMemcpy(e.wy, wy.data(), ny * 4, cudaMemcpyHostToDevice));
      GPL_CUDA(cudaMemcpy(e.w4x, w4x.data(), nx * 8, cudaMemcpyHostToDevice));
      GPL_CUDA(cudaMemcpy(e.w4y, w4y.data(), ny * 8, cudaMemcpyHostToDevice));
      GPL_CUDA(cudaMemcpy(e.tw, tw.data(), tw.size() * 8, cudaMemcpyHostToDevice));
      if (e.shared) GPL_CUDA(cudaEventCreateWithFlags(&e.done, cudaEventDisableTiming));
      // (a copy from pageable memory may return before it has arrived, and a
      // caller's non-blocking stream does not wait for it)
      GPL_CUDA(cudaStreamSynchronize(nullptr));
      g_cache.push_back(n);
      c = n;
    }
  }
  PoissonGrid g;
  g.nx = nx; g.ny = ny; g.size_x = bsx; g.size_y = bsy;
  g.core_lx = g.core_ly = 0; g.core_ux = nx * bsx; g.core_uy = ny * bsy;
  g.wx = c->wx; g.wy = c->wy; g.w4x = c->w4x; g.w4y = c->w4y; g.tw = c->tw;
  std::lock_guard<std::mutex> lk(c->mu);
  const bool ordered = c->shared && !capturing;
  if (ordered) GPL_CUDA(cudaStreamWaitEvent(s, c->done));
  int rc = poisson_passes(g, nullptr, nullptr, nullptr, 1.0f, density, nullptr, nullptr, c->spec,
                          c->p1, c->p2, nullptr, fx, fy, phi, s, nullptr);
  if (ordered) GPL_CUDA(cudaEventRecord(c->done, s));
  return (gpl_status)rc;
}
