// Density scatter (BinGrid::updateBinsGCellDensityArea, src/nesterovBase.cpp:746-798)
// fused with the Nesterov predictor (src/nesterovPlace.cpp:338-362), the
// per-gcell gradient kernel (getDensityGradient :1458-1478 + the WA gradient
// sum :1363-1375 + NesterovPlace::updateGradients src/nesterovPlace.cpp:206-273
// + the step-length distances :555-571, 598-607), and the FP64 finalize.
//
// The scatter adds, per (gcell, covered bin), the truncated int64 value of
// the float overlap area times the density scale (times the target density
// for macros) -- the reference's exact per-contribution arithmetic.  Integer
// addition is associative, so atomics give bit-exact, order-independent bin
// areas.  Lanes of a warp that hit the same bin are combined first
// (__match_any_sync), which matters when many cells sit on the same bins
// (all cells start at the core centre).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>

#include "device_common.cuh"

namespace gpl {

namespace {

constexpr int kBlock = 256;
// The gcell kernel's residency (48 registers): at six blocks the loads moved
// ahead of the pin gathers spill (10k / 200k / 1M cells: 12.2 / 28.6 / 54.1 us
// against 11.3 / 24.6 / 55.0 at five and 10.9 / 24.6 / 58.6 at four).
constexpr int kCellBlocksPerSm = 5;

struct ScatterArgs {
  BinGeom geo;
  int n_g;
  float td;
  const int4* geo_g;            // per gcell (GCellGeo)
  float2* slp[4];
  float2* sum[4];
  float2* coordi[2];
  unsigned long long* area[2];  // two sets of inst [nb], filler [nb]
  const EvalCtl* ctl;
  EvalCtl* ctl_dev;           // copy of ctl for the evaluation's other kernels (null: ctl is it)
  int one_word;                 // a window's sums fit 32 bits (scatter_one_word)
  int fits32;                   // so does every single value
};

__device__ __forceinline__ float2 predict_one(const ScatterArgs& A, const EvalCtl& C, int g, int2 h) {
  const float2 cs = pick4(A.slp, C.i_src)[g], sg = pick4(A.sum, C.i_src)[g], cc = pick2(A.coordi, C.c_cur)[g];
  float nx = __fadd_rn(cs.x, __fmul_rn(C.step, sg.x));
  float ny = __fadd_rn(cs.y, __fmul_rn(C.step, sg.y));
  float sx = __fadd_rn(nx, __fmul_rn(C.coeff, __fsub_rn(nx, cc.x)));
  float sy = __fadd_rn(ny, __fmul_rn(C.coeff, __fsub_rn(ny, cc.y)));
  const BinGeom& G = A.geo;
  pick2(A.coordi, C.c_next)[g] = make_float2(inside(nx, h.x, G.core_lx, G.core_ux), inside(ny, h.y, G.core_ly, G.core_uy));
  float2 s = make_float2(inside(sx, h.x, G.core_lx, G.core_ux), inside(sy, h.y, G.core_ly, G.core_uy));
  pick4(A.slp, C.i_eval)[g] = s;
  return s;
}

// ------------------------------------------------------------ tile order
// The scatter visits gcells tile by tile: a tile is tile_w x tile_h bins, and
// the gcells whose centres lie in it (at the last ordering) are consecutive
// in `order`.  A block takes a chunk of at most d.chunk gcells of one tile
// (the tile side and chunk size are tuned per job, see nesterov_init) and
// accumulates their bin areas in a shared-memory window over the
// tile and a margin; the window's non-zero bins then go to the global areas
// with one 64-bit atomic each.  Bins outside the window (cells that moved
// away, large cells) go to the global areas directly.  The int64 sums do not
// depend on the order, so the ordering only changes the number of global
// atomics, never a result.

constexpr int kTileMargin = 2;

struct OrderArgs {
  BinGeom geo;
  int n_g, tile_w, tile_h, tiles_x, tiles_y;
  const float2* slp;            // the coordinates to order by, or (slp == nullptr)
  const float2* slp_all[4];     // slot ctl->i_src of these (the device loop)
  const EvalCtl* ctl;
  int chunk;                    // gcells per chunk (at most)
  int32_t* tile_count;
  int32_t* tile_start;
  int32_t* order;
  int4* chunks;
  int32_t* n_chunks;
};

__device__ __forceinline__ int tile_of(const OrderArgs& O, float2 c) {
  const BinGeom& G = O.geo;
  const int bx = min(G.div_x(max(__float2int_rz(c.x) - G.core_lx, 0)), G.cnt_x - 1);
  const int by = min(G.div_y(max(__float2int_rz(c.y) - G.core_ly, 0)), G.cnt_y - 1);
  return (by / O.tile_h) * O.tiles_x + bx / O.tile_w;
}

__device__ __forceinline__ const float2* order_coords(const OrderArgs& O) {
  return O.slp ? O.slp : pick4(O.slp_all, O.ctl->i_src);
}

// Lanes of a warp on the same tile add their count with one atomic.
__global__ void __launch_bounds__(kBlock) k_order_count(OrderArgs O) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  const float2* slp = order_coords(O);
  const int t = g < O.n_g ? tile_of(O, slp[g]) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, t);    // every lane takes part
  if (t >= 0 && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&O.tile_count[t], __popc(peers));
}

// One block: exclusive scan of the tile counts into tile_start, fill cursors
// (tile_count := tile_start), and the chunk table (tiles cut into chunks of
// at most O.chunk gcells).
constexpr int kOrderScanT = 1024;
__global__ void __launch_bounds__(kOrderScanT) k_order_scan(OrderArgs O) {
  __shared__ int32_t sc[kOrderScanT], sk[kOrderScanT];
  const int nt = O.tiles_x * O.tiles_y;
  const int per = (nt + kOrderScanT - 1) / kOrderScanT;
  const int lo = min((int)threadIdx.x * per, nt), hi = min(lo + per, nt);
  int cells = 0, chunks = 0;
  for (int t = lo; t < hi; t++) {
    const int c = O.tile_count[t];
    cells += c;
    chunks += (c + O.chunk - 1) / O.chunk;
  }
  sc[threadIdx.x] = cells;
  sk[threadIdx.x] = chunks;
  __syncthreads();
  for (int o = 1; o < kOrderScanT; o <<= 1) {
    const int x = threadIdx.x >= o ? sc[threadIdx.x - o] : 0;
    const int y = threadIdx.x >= o ? sk[threadIdx.x - o] : 0;
    __syncthreads();
    sc[threadIdx.x] += x;
    sk[threadIdx.x] += y;
    __syncthreads();
  }
  int at = sc[threadIdx.x] - cells, ck = sk[threadIdx.x] - chunks;
  for (int t = lo; t < hi; t++) {
    const int c = O.tile_count[t];
    O.tile_start[t] = at;
    O.tile_count[t] = at;
    // equal chunks: a short last one would cost a block's window all the same
    const int n_ch = (c + O.chunk - 1) / O.chunk;
    for (int f = 0, k = 0; k < n_ch; k++) {
      const int e = (int)(((long long)c * (k + 1)) / n_ch);
      O.chunks[ck++] = make_int4(t, at + f, at + e, 0);
      f = e;
    }
    at += c;
  }
  if (threadIdx.x == kOrderScanT - 1) {
    O.tile_start[nt] = sc[kOrderScanT - 1];
    *O.n_chunks = sk[kOrderScanT - 1];
  }
}

__global__ void __launch_bounds__(kBlock) k_order_fill(OrderArgs O) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const float2* slp = order_coords(O);
  const int t = g < O.n_g ? tile_of(O, slp[g]) : -1;
  const unsigned peers = __match_any_sync(0xffffffffu, t);    // every lane takes part
  const int leader = __ffs(peers) - 1;
  int base = 0;
  if (t >= 0 && lane == leader) base = atomicAdd(&O.tile_count[t], __popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);               // every lane takes part
  if (t >= 0) O.order[base + __popc(peers & ((1u << lane) - 1u))] = g;
}

struct TileArgs {
  int tile_w, tile_h, tiles_x;
  FastDiv div_wx;               // by the window's width
  const int32_t* order;
  const int4* chunks;
  const int32_t* n_chunks;
};

// updateGCellDensityCenterLocation + updateBinsGCellDensityArea
// (src/nesterovBase.cpp:746-819, 1198-1207): one chunk of one tile per block.
// Per (gcell, bin) the area is (int64)(float overlap * scale [* td for a
// macro]), added into the inst or filler set.  The predictor runs here for
// every gcell (big ones included; their bins are left to scatter_big_body).
// The body of one block (chunk vb); `win` is the block's dynamic shared
// window.  Shared by the per-job launch and the batched one.
//
// What bounds it is instruction issue and the barriers around the window (600
// warp instructions for 32 gcells at a million cells, 40 % of the issue slots),
// so: bin ranges by multiplication (FastDiv), a gcell's overlap widths once
// per column and row, its up to 3 x 3 bins without loops or range tests when
// they lie inside the window, and one 32-bit window word per bin where the
// chunk's sums cannot pass 2^32 (two 16-bit halves in two words otherwise).
// 12.5k gcells 17.5 -> 9.8 us, 250k with 40 macros 28.9 -> 24, 1.25M 64.0 ->
// 42.8 (in the loop, events around the launch).
template <bool kOneWord>
__device__ __forceinline__ void scatter_body(const ScatterArgs& A, const TileArgs& T, int vb, unsigned* win) {
  if (vb >= *T.n_chunks) return;                   // block-uniform
  const EvalCtl C = *A.ctl;
  unsigned long long* area = pick2(A.area, C.area_cur);
  const BinGeom& G = A.geo;
  const int nb = G.cnt_x * G.cnt_y;
  const int4 ch = T.chunks[vb];
  const int tile_y = ch.x / T.tiles_x, tile_x = ch.x - tile_y * T.tiles_x;
  const int ox = tile_x * T.tile_w - kTileMargin;
  const int oy = tile_y * T.tile_h - kTileMargin;
  const int wx = T.tile_w + 2 * kTileMargin, wy = T.tile_h + 2 * kTileMargin, wn = wx * wy;
  unsigned* win_hi = win + 2 * wn;                 // (two-word form)
  constexpr int kWords = kOneWord ? 2 : 4;
  // (wn is even, the window 16-byte aligned)
  for (int i = threadIdx.x; i < kWords * wn / 4; i += blockDim.x) reinterpret_cast<uint4*>(win)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  // adds v at window index i: the sums return nothing and neither word can
  // wrap (one word: see scatter_one_word; two: a chunk has fewer than 2^16
  // gcells, one addition of a 16-bit half each per bin)
  auto add = [&](int i, unsigned v) {
    if (v == 0u) return;
    if constexpr (kOneWord) {
      atomicAdd(&win[i], v);
    } else {
      atomicAdd(&win[i], v & 0xffffu);
      atomicAdd(&win_hi[i], v >> 16);
    }
  };
  for (int idx = ch.y + threadIdx.x; idx < ch.z; idx += blockDim.x) {
    const int g = T.order[idx];
    const GCellGeo q = gcell_geo(A.geo_g[g]);
    const float2 c = C.predict ? predict_one(A, C, g, q.half) : pick4(A.slp, C.i_eval)[g];
    if (q.big()) continue;                         // scatter_big_body
    int lx, ux, ly, uy, x0, x1, y0, y1;
    density_rect(c, q.half, lx, ux, ly, uy);
    G.range(lx, ux, ly, uy, x0, x1, y0, y1);
    const int half = q.type() == 2 ? 1 : 0;
    const bool macro = q.type() == 1;              // scaled down by the target density
    const int u0 = x0 - ox, w0 = y0 - oy;
    const int nx = x1 - x0, ny = y1 - y0;
    if (A.fits32 && q.scale <= 1.0f && nx <= 3 && ny <= 3 && u0 >= 0 && u0 + nx <= wx && w0 >= 0 && w0 + ny <= wy) {
      float fx[3], fy[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        fx[k] = k < nx ? G.overlap_x(x0 + k, lx, ux) : 0.0f;
        fy[k] = k < ny ? G.overlap_y(y0 + k, ly, uy) : 0.0f;
      }
      const int i0 = half * wn + w0 * wx + u0;
#pragma unroll
      for (int r = 0; r < 3; r++)
#pragma unroll
        for (int k = 0; k < 3; k++) {
          float f = __fmul_rn(__fmul_rn(fx[k], fy[r]), q.scale);
          if (macro) f = __fmul_rn(f, A.td);
          add(i0 + r * wx + k, __float2uint_rz(f));
        }
      continue;
    }
    for (int cc = y0; cc < y1; cc++) {
      for (int a = x0; a < x1; a++) {
        float f = __fmul_rn(G.overlap(a, cc, lx, ux, ly, uy), q.scale);
        if (macro) f = __fmul_rn(f, A.td);
        const unsigned long long v = trunc_u64(f);
        if (!v) continue;
        const int u = a - ox, w = cc - oy;
        if (A.fits32 && q.scale <= 1.0f && u >= 0 && u < wx && w >= 0 && w < wy) add(half * wn + w * wx + u, (unsigned)v);
        else atomicAdd(&area[half * nb + cc * G.cnt_x + a], v);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * wn; i += blockDim.x) {
    unsigned long long v = win[i];
    if constexpr (!kOneWord) v += (unsigned long long)win_hi[i] << 16;
    if (!v) continue;
    const int half = i >= wn ? 1 : 0, r = i - half * wn;
    const int w = T.div_wx(r);
    const int a = ox + r - w * wx, cc = oy + w;       // inside the grid: only in-grid bins were added
    atomicAdd(&area[half * nb + cc * G.cnt_x + a], v);
  }
}

// One block per big cell (macros): threads stride over its bins.
__device__ __forceinline__ void scatter_big_body(const ScatterArgs& A, const int32_t* big, int vb) {
  const EvalCtl C = *A.ctl;
  unsigned long long* area = pick2(A.area, C.area_cur);
  const int g = big[vb];
  const BinGeom& G = A.geo;
  const int nb = G.cnt_x * G.cnt_y;
  const GCellGeo geo = gcell_geo(A.geo_g[g]);
  const int2 h = geo.half;
  // the chunk that holds this cell writes its predicted coordinates, maybe
  // later than this block runs; recomputed here with the same arithmetic
  float2 c;
  if (C.predict) {
    __shared__ float2 cs;
    if (threadIdx.x == 0) cs = predict_one(A, C, g, h);
    __syncthreads();
    c = cs;
  } else {
    c = pick4(A.slp, C.i_eval)[g];
  }
  int lx, ux, ly, uy, x0, x1, y0, y1;
  density_rect(c, h, lx, ux, ly, uy);
  G.range(lx, ux, ly, uy, x0, x1, y0, y1);
  if (x1 <= x0 || y1 <= y0) return;
  const int nbx = x1 - x0, total = nbx * (y1 - y0);
  const int k = geo.kind;
  const float sc = geo.scale;
  for (int t = threadIdx.x; t < total; t += blockDim.x) {
    const int a = x0 + t % nbx, cc = y0 + t / nbx;
    float f = __fmul_rn(G.overlap(a, cc, lx, ux, ly, uy), sc);
    if ((k & 3) == 1) f = __fmul_rn(f, A.td);
    const long long v = (long long)trunc_u64(f);
    if (v) atomicAdd(&area[((k & 3) == 2 ? nb : 0) + cc * G.cnt_x + a], (unsigned long long)v);
  }
}

// The first n_big blocks take a big cell each, the rest a chunk each: the sums
// are integers and a big cell's block predicts its own position, so neither
// needs the other.  As a launch of their own after the chunks, the big cells
// cost their latency: a loop of 200k cells with 40 macros 91.5 -> 84 us an
// iteration.
template <bool kOneWord>
__global__ void __launch_bounds__(kBlock, 5) k_scatter(const __grid_constant__ ScatterArgs A,
                                                       const __grid_constant__ TileArgs T, const int32_t* big, int n_big) {
  extern __shared__ __align__(16) unsigned win[];  // [words][2][wy][wx]: sums, or low 16-bit then high 16-bit sums
  if (A.ctl_dev && blockIdx.x == 0 && threadIdx.x < sizeof(EvalCtl) / 4)
    reinterpret_cast<unsigned*>(A.ctl_dev)[threadIdx.x] = reinterpret_cast<const unsigned*>(A.ctl)[threadIdx.x];
  if ((int)blockIdx.x < n_big) scatter_big_body(A, big, (int)blockIdx.x);
  else scatter_body<kOneWord>(A, T, (int)blockIdx.x - n_big, win);
}

struct CellArgs {
  BinGeom geo;
  int n_g;
  const int4* geo_g;          // per gcell (GCellGeo)
  float2* slp[4];
  float2* sum[4];
  const EvalCtl* ctl;
  const float2* field;        // (Ex, Ey) per bin
  const int32_t* g_pin_start;
  const int32_t* g_pins;      // device pin index of each gcell pin slot
  const float2* pin_grad;     // device pin order
  const float* area_g;        // dx*dy of each gcell (the pin count comes from its slots)
  float2* d_big;
  float min_precond;
  float2* wl_out;
  float2* d_out;
  double* part;               // [kPartSlots][stride]
  int stride;
  int n_ovf_blocks, n_phi_blocks;
  unsigned* counters;
  long long* hpwl_total;
  EvalResult* out;
  // the host's pinned record (null: none), written by the kernel itself: a
  // copy after it was a graph node of 2 to 5 us in every evaluation (loop of
  // 10k cells 43.1 -> 38.0 us an iteration, 200k with macros 84 -> 79.5, 1M
  // 240 -> 236)
  EvalResult* out_host;
};

// Density gradient of one big cell, reduced over a block (fixed tree order).
// Bound by the latency of its field loads: four in flight a thread (the sums
// stay in bin order); loop of 200k cells with 40 macros 77.9 -> 76.3 us an
// iteration.
__device__ __forceinline__ void dgrad_big_body(const CellArgs& A, const int32_t* big, int vb) {
  __shared__ float sx[kBlock], sy[kBlock];
  const int g = big[vb];
  const BinGeom& G = A.geo;
  const EvalCtl C = *A.ctl;
  int lx, ux, ly, uy, x0, x1, y0, y1;
  const GCellGeo geo = gcell_geo(A.geo_g[g]);
  density_rect(pick4(A.slp, C.i_eval)[g], geo.half, lx, ux, ly, uy);
  G.range(lx, ux, ly, uy, x0, x1, y0, y1);
  const int nbx = max(x1 - x0, 0), total = nbx * max(y1 - y0, 0);
  const float sc = geo.scale;
  float ex = 0.0f, ey = 0.0f;
  for (int t0 = threadIdx.x; t0 < total; t0 += 4 * kBlock) {
    float2 f[4];
    int a[4], cc[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int t = min(t0 + u * kBlock, total - 1);
      cc[u] = t / nbx;
      a[u] = x0 + t - cc[u] * nbx;
      cc[u] += y0;
      f[u] = A.field[cc[u] * G.cnt_x + a[u]];
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (t0 + u * kBlock < total) {
        const float ov = __fmul_rn(G.overlap(a[u], cc[u], lx, ux, ly, uy), sc);
        ex = __fadd_rn(ex, __fmul_rn(ov, f[u].x));
        ey = __fadd_rn(ey, __fmul_rn(ov, f[u].y));
      }
  }
  sx[threadIdx.x] = ex; sy[threadIdx.x] = ey;
  __syncthreads();
  for (int s = kBlock / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) { sx[threadIdx.x] += sx[threadIdx.x + s]; sy[threadIdx.x] += sy[threadIdx.x + s]; }
    __syncthreads();
  }
  if (threadIdx.x == 0) A.d_big[vb] = make_float2(sx[0], sy[0]);
}

__global__ void __launch_bounds__(kBlock) k_dgrad_big(CellArgs A, const int32_t* big, int n_big) {
  dgrad_big_body(A, big, (int)blockIdx.x);
}

// One gcell per thread, grid-stride over a grid sized to the SM count; the
// block partial sums are reduced by the last block to finish (threadfence +
// counter), in a fixed order, so there is no separate reduction launch and
// the result is the same run to run.
// Block vb of a launch of vgrid blocks.
__device__ __forceinline__ void cell_body(const CellArgs& A, int vb, int vgrid) {
  __shared__ __align__(8) float sh[64];
  __shared__ int sh_bad[8];
  __shared__ bool last;
  // per-thread sums in float over the thread's few gcells; FP64 from the
  // warp sums on (the FP64 pipe is narrow on this part)
  float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};      // |wl|, |d|, coord dist^2, grad dist^2
  int bad = 0;
  const BinGeom& G = A.geo;
  const EvalCtl C = *A.ctl;
  // restrict-qualified views (inputs and outputs are distinct arrays), so
  // the loads of a thread's next gcell can be issued before the stores of
  // its previous one
  const float2* __restrict__ slp = pick4(A.slp, C.i_eval);
  float2* __restrict__ sum_out = C.write_sum ? pick4(A.sum, C.i_eval) : nullptr;
  const float2* __restrict__ ref_slp = C.i_ref >= 0 ? pick4(A.slp, C.i_ref) : nullptr;
  const float2* __restrict__ ref_sum = C.i_ref >= 0 ? pick4(A.sum, C.i_ref) : nullptr;
  float2* __restrict__ wl_out = C.write_wd ? A.wl_out : nullptr;
  float2* __restrict__ d_out = C.write_wd ? A.d_out : nullptr;
  const float2* __restrict__ pin_grad = A.pin_grad;
  const int32_t* __restrict__ g_pins = A.g_pins;
  const int32_t* __restrict__ g_pin_start = A.g_pin_start;
  const float2* __restrict__ field = A.field;
  const int4* __restrict__ geo_g = A.geo_g;
  const float* __restrict__ area_g = A.area_g;
  const float lam = C.density_penalty;
  const int lane = threadIdx.x & 31;
  // warp-uniform grid-stride loop: the warps gather the pins of cells with
  // more than 32 pins (macros) together
#pragma unroll 2
  for (int base = vb * kBlock + (threadIdx.x & ~31); base < A.n_g; base += vgrid * kBlock) {
    const int g = base + lane;
    const bool valid = g < A.n_g;
    int ps = 0, pe = 0;
    float2 w = make_float2(0.0f, 0.0f);
    const int gg = valid ? g : A.n_g - 1;          // (loaded ahead of the pin gathers)
    const float2 c = slp[gg];
    const int4 gi = geo_g[gg];
    if (valid) {
      ps = g_pin_start[g];
      pe = g_pin_start[g + 1];
      if (pe - ps <= 32) {
        // WA gradient: the cell's pins in instance pin order, four slots'
        // loads in flight at a time (the sums stay in slot order)
        for (int t = ps; t < pe; t += 4) {
          int q[4];
#pragma unroll
          for (int u = 0; u < 4; u++) q[u] = t + u < pe ? g_pins[t + u] : -1;
          float2 pg[4];
#pragma unroll
          for (int u = 0; u < 4; u++) pg[u] = q[u] >= 0 ? pin_grad[q[u]] : make_float2(0.0f, 0.0f);
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (q[u] >= 0) {
              w.x = __fadd_rn(w.x, pg[u].x);
              w.y = __fadd_rn(w.y, pg[u].y);
            }
        }
      }
    }
    unsigned many = __ballot_sync(0xffffffffu, pe - ps > 32);
    while (many) {
      const int src = __ffs(many) - 1;
      many &= many - 1;
      const int s0 = __shfl_sync(0xffffffffu, ps, src), s1 = __shfl_sync(0xffffffffu, pe, src);
      float2 part = make_float2(0.0f, 0.0f);
      for (int t = s0 + lane; t < s1; t += 32) {
        const float2 pg = pin_grad[g_pins[t]];
        part.x = __fadd_rn(part.x, pg.x);
        part.y = __fadd_rn(part.y, pg.y);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        part.x = __fadd_rn(part.x, __shfl_xor_sync(0xffffffffu, part.x, o));
        part.y = __fadd_rn(part.y, __shfl_xor_sync(0xffffffffu, part.y, o));
      }
      if (lane == src) w = part;
    }
    if (!valid) continue;
    const GCellGeo geo = gcell_geo(gi);
    // density gradient: sum over covered bins of overlap * scale * field
    float2 d = make_float2(0.0f, 0.0f);
    if (geo.big()) {
      d = A.d_big[geo.big_index()];
    } else {
      int lx, ux, ly, uy, x0, x1, y0, y1;
      density_rect(c, geo.half, lx, ux, ly, uy);
      G.range(lx, ux, ly, uy, x0, x1, y0, y1);
      const float sc = geo.scale;
      const int ny = y1 - y0;
      if (ny <= 3) {
        // the usual cell: its row widths once, a column's field loads together
        float fy[3];
#pragma unroll
        for (int r = 0; r < 3; r++) fy[r] = r < ny ? G.overlap_y(y0 + r, ly, uy) : 0.0f;
        const float2* fp = field + y0 * G.cnt_x;
        for (int a = x0; a < x1; a++) {
          const float fx = G.overlap_x(a, lx, ux);
          float2 f[3];
#pragma unroll
          for (int r = 0; r < 3; r++) f[r] = r < ny ? fp[r * G.cnt_x + a] : make_float2(0.0f, 0.0f);
#pragma unroll
          for (int r = 0; r < 3; r++) {
            if (r < ny) {
              const float ov = __fmul_rn(__fmul_rn(fx, fy[r]), sc);
              d.x = __fadd_rn(d.x, __fmul_rn(ov, f[r].x));
              d.y = __fadd_rn(d.y, __fmul_rn(ov, f[r].y));
            }
          }
        }
      } else {
        for (int a = x0; a < x1; a++) {
          for (int cc = y0; cc < y1; cc++) {
            const float ov = __fmul_rn(G.overlap(a, cc, lx, ux, ly, uy), sc);
            const float2 f = field[cc * G.cnt_x + a];
            d.x = __fadd_rn(d.x, __fmul_rn(ov, f.x));
            d.y = __fadd_rn(d.y, __fmul_rn(ov, f.y));
          }
        }
      }
    }
    float2 s = make_float2(__fadd_rn(w.x, __fmul_rn(lam, d.x)), __fadd_rn(w.y, __fmul_rn(lam, d.y)));
    // getWireLengthPreconditioner / getDensityPreconditioner (src/nesterovBase.cpp:1442-1454)
    float px = __fadd_rn((float)(pe - ps), __fmul_rn(lam, area_g[g]));
    float py = px;
    if (px <= A.min_precond) px = A.min_precond;
    if (py <= A.min_precond) py = A.min_precond;
    s.x = __fdiv_rn(s.x, px);
    s.y = __fdiv_rn(s.y, py);
    if (sum_out) sum_out[g] = s;
    if (wl_out) wl_out[g] = w;
    if (d_out) d_out[g] = d;
    const float aw = fabsf(w.x) + fabsf(w.y);
    const float ad = fabsf(d.x) + fabsf(d.y);
    acc[0] += aw;
    acc[1] += ad;
    if (ref_slp) {
      const float2 r = ref_slp[g], q = ref_sum[g];
      // getDistance (src/nesterovPlace.cpp:598-607): float differences
      const float dx = c.x - r.x, dy = c.y - r.y;
      const float gx = s.x - q.x, gy = s.y - q.y;
      // rounding spelled out: the per-job and the batched kernel inline
      // this body, and must not fuse differently.  The sum of a term is fused,
      // the running sum is not: one rounding of the running sum a term.
      // Relative error of a thread's 7 terms against 64 bits: 4.9e-8 (5.1e-8
      // with nothing fused, 6.0e-8 with both)
      acc[2] = __fadd_rn(acc[2], __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
      acc[3] = __fadd_rn(acc[3], __fmaf_rn(gx, gx, __fmul_rn(gy, gy)));
    }
    if (!isfinite(aw) || !isfinite(ad)) bad = 1;
  }
  // The FP64 pipe takes 64 cycles a warp instruction on each of an SM's four
  // schedulers, so the sums across warps and blocks are laid out to need few:
  // each instruction serves all slots at once (block), or one slot a warp
  // (final).
  const int wid = threadIdx.x >> 5;
  static_assert(kBlock == 256, "eight warps");
  {
    // warp sums (float, fixed xor tree), then the block's eight warps in FP64.
    // Where a thread has several gcells the tree's last addition is left to
    // FP64 too (even and odd lanes' sums apart): it rounds the largest sum, half
    // the variance of the block's, and five blocks an SM instead of six make 17 %
    // fewer, larger warp sums there (with one gcell a thread the warps are the
    // same ones).  Rms relative error of the totals over 40 placements, in float
    // to the end and so: 0.58M gcells 5.1e-10 -> 3.6e-10, 1.17M 5.8e-10 ->
    // 4.1e-10 (six blocks, in float: 4.5e-10 and 4.2e-10).
    const bool apart = vgrid * kBlock < A.n_g;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
      for (int o = 16; o > 1; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
    const int any_bad = __any_sync(0xffffffffu, bad);
    if (!apart) {
#pragma unroll
      for (int k = 0; k < 4; k++) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], 1);
      if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 4; k++) sh[k * 8 + wid] = acc[k];
      }
    } else if (lane < 2) {
#pragma unroll
      for (int k = 0; k < 4; k++) sh[k * 16 + wid * 2 + lane] = acc[k];
    }
    if (lane == 0) sh_bad[wid] = any_bad;
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane 8 k + w: slot k of warp w (apart: of its two halves)
      double t;
      if (!apart) t = (double)sh[lane];
      else t = (double)sh[2 * lane] + (double)sh[2 * lane + 1];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      const int bads = __popc(__ballot_sync(0xffffffffu, lane < 8 && sh_bad[lane & 7]));
      static_assert(kPartD == kPartWl + 1 && kPartCoordDist == kPartWl + 2 && kPartGradDist == kPartWl + 3 &&
                        kPartNan == kPartWl + 4, "slot order");
      if ((lane & 7) == 0) A.part[(size_t)(kPartWl + (lane >> 3)) * A.stride + vb] = t;
      if (lane == 0) A.part[(size_t)kPartNan * A.stride + vb] = (double)bads;
      __threadfence();
      __syncwarp();
      if (lane == 0) last = atomicAdd(&A.counters[0], 1u) == (unsigned)vgrid - 1;
    }
    __syncthreads();
  }
  if (!last) return;
  // final reduction (the last block), a slot per warp: every partial is
  // visible after the fence; four loads in flight per lane
  __threadfence();
  static_assert(kPartSlots <= 7, "a slot per warp, HPWL on the last");
  if (wid < kPartSlots) {
    const int n = wid == kPartOverflow ? A.n_ovf_blocks : (wid == kPartPhi ? A.n_phi_blocks : vgrid);
    const double* p = A.part + (size_t)wid * A.stride;
    double t = 0.0;
    for (int i = lane; i < n; i += 128) {
      double x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) x[u] = i + 32 * u < n ? __ldcg(p + i + 32 * u) : 0.0;
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (i + 32 * u < n) t += x[u];
    }
    if (n > 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    }
    if (lane == 0) {
      auto put = [&](EvalResult* r) {
        double* dst = wid == kPartOverflow ? &r->overflow : wid == kPartWl ? &r->wl_sum : wid == kPartD ? &r->d_sum
                      : wid == kPartCoordDist ? &r->coord_dist : wid == kPartGradDist ? &r->grad_dist
                      : wid == kPartNan ? &r->nan_flag : &r->sum_phi;
        *dst = t;
      };
      put(A.out);
      if (A.out_host) put(A.out_host);
    }
  } else {
    // the WA kernel's HPWL accumulators: one per lane, summed by shuffles and
    // cleared for the next evaluation
    static_assert(kHpwlLanes == 32, "one HPWL accumulator per lane");
    long long hpwl = __ldcg(A.hpwl_total + lane * kHpwlStride);
    A.hpwl_total[lane * kHpwlStride] = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) hpwl += __shfl_xor_sync(0xffffffffu, hpwl, o);
    if (lane == 0) {
      auto put = [&](EvalResult* r) {
        r->hpwl = hpwl;
        r->n_g = A.n_g;
      };
      put(A.out);
      if (A.out_host) put(A.out_host);
      A.counters[0] = 0u;
    }
  }
}

__global__ void __launch_bounds__(kBlock, kCellBlocksPerSm) k_cell(CellArgs A) {
  cell_body(A, (int)blockIdx.x, (int)gridDim.x);
}

// sum over bins of phi * (nonPlace + inst + filler) in FP64
// (NesterovBase::updateDensityForceBin, src/nesterovBase.cpp:1494-1505)
__global__ void __launch_bounds__(kBlock) k_sum_phi(const float* phi, const unsigned long long* area,
                                                   const int64_t* nonplace, int nb, double* part) {
  __shared__ double sh[32];
  double v[1] = {0.0};
  for (int b = blockIdx.x * kBlock + threadIdx.x; b < nb; b += gridDim.x * kBlock)
    v[0] += (double)phi[b] * (double)(nonplace[b] + (long long)area[b] + (long long)area[nb + b]);
  block_reduce_n<1>(v, part, 0, sh);
}

BinGeom geom(const DeviceModel& d) {
  BinGeom G;
  G.core_lx = d.core_lx; G.core_ly = d.core_ly; G.core_ux = d.core_ux; G.core_uy = d.core_uy;
  G.size_x = d.size_x; G.size_y = d.size_y; G.cnt_x = d.cnt_x; G.cnt_y = d.cnt_y;
  G.div_x = FastDiv(d.size_x); G.div_y = FastDiv(d.size_y);
  return G;
}

}  // namespace

int cell_blocks(const DeviceModel& d) { return (d.n_g + kBlock - 1) / kBlock; }

namespace {
// The largest value a gcell of scale at most 1 adds to a bin, as the float
// product rounds (the factors are at most the bin's sides).
double scatter_max_value(const DeviceModel& d) {
  return 1.000001 * (double)d.size_x * (double)d.size_y * std::max(1.0, (double)d.target_density);
}
// One window word per bin: a chunk adds at most `piece` values to it.
bool scatter_one_word(const DeviceModel& d) { return scatter_max_value(d) * d.piece < 4294967295.0; }

ScatterArgs scatter_args(const DeviceModel& d) {
  ScatterArgs A;
  A.geo = geom(d);
  A.n_g = d.n_g;
  A.td = d.target_density;
  A.geo_g = d.g_geo;
  A.one_word = scatter_one_word(d) ? 1 : 0;
  A.fits32 = scatter_max_value(d) < 4294967295.0 ? 1 : 0;
  for (int k = 0; k < 4; k++) { A.slp[k] = d.slp[k]; A.sum[k] = d.sum[k]; }
  A.coordi[0] = d.coordi[0]; A.coordi[1] = d.coordi[1];
  A.area[0] = d.area[0]; A.area[1] = d.area[1];
  A.ctl = d.ctl;
  A.ctl_dev = nullptr;
  return A;
}

TileArgs tile_args(const DeviceModel& d) {
  TileArgs T;
  T.tile_w = d.tile_w; T.tile_h = d.tile_h; T.tiles_x = d.tiles_x;
  T.div_wx = FastDiv(d.tile_w + 2 * kTileMargin);
  T.order = d.order; T.chunks = d.chunks; T.n_chunks = d.n_chunks;
  return T;
}

CellArgs cell_args(const DeviceModel& d, const EvalArgs& a, int n_phi_blocks) {
  CellArgs A;
  A.geo = geom(d);
  A.n_g = d.n_g;
  A.geo_g = d.g_geo;
  for (int k = 0; k < 4; k++) { A.slp[k] = d.slp[k]; A.sum[k] = d.sum[k]; }
  A.ctl = d.ctl;
  A.field = d.field;
  A.g_pin_start = d.g_pin_start;
  A.g_pins = d.g_pins;
  A.pin_grad = d.pin_grad;
  A.area_g = d.g_area;
  A.d_big = d.d_big;
  A.min_precond = a.min_precond;
  A.wl_out = d.wl_out; A.d_out = d.d_out;
  A.part = d.part;
  A.stride = d.part_stride;
  A.n_ovf_blocks = poisson_blocks_a(d.cnt_x, d.cnt_y);
  A.n_phi_blocks = n_phi_blocks;
  A.counters = d.counters;
  A.hpwl_total = d.hpwl_total;
  A.out = d.result;
  A.out_host = nullptr;
  return A;
}
}  // namespace

int launch_scatter(DeviceModel& d, const EvalArgs& a, bool ctl_from_host, cudaStream_t s, Timer& t) {
  ScatterArgs A = scatter_args(d);
  if (ctl_from_host) { A.ctl = d.ctl_h; A.ctl_dev = d.ctl; }
  const TileArgs T = tile_args(d);
  (void)a;
  t.begin(kKScatter);
  const int grid = d.n_big + d.max_chunks;
  if (A.one_word) k_scatter<true><<<grid, kBlock, scatter_smem(d), s>>>(A, T, d.big_cells, d.n_big);
  else k_scatter<false><<<grid, kBlock, scatter_smem(d), s>>>(A, T, d.big_cells, d.n_big);
  t.end(kKScatter);
  t.count(1);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

void tile_grid(int cnt_x, int cnt_y, int side, int* tw, int* th, int* tx, int* ty) {
  *tw = std::min(side, cnt_x);
  *th = std::min(side, cnt_y);
  *tx = (cnt_x + *tw - 1) / *tw;
  *ty = (cnt_y + *th - 1) / *th;
}

// every tile's chunks: one per `chunk` gcells, plus one per tile for the
// partial last chunks
int scatter_max_chunks(int n_g, int tiles, int chunk) { return tiles + (n_g + chunk - 1) / chunk; }

bool set_scatter_shape(DeviceModel& d, int side, int chunk) {
  int tw, th, tx, ty;
  tile_grid(d.cnt_x, d.cnt_y, side, &tw, &th, &tx, &ty);
  // a design of fewer chunks than resident blocks (five per SM) takes smaller
  // ones: at 12.5k gcells 49 blocks instead of 17
  int piece = std::min(chunk, std::max(kScatterPieceMin, (d.n_g + 5 * d.sm_count - 1) / (5 * d.sm_count)));
  const double one = 4294967294.0 / scatter_max_value(d);    // up to here one window word will do
  if (one < piece && one >= std::max(0.75 * piece, (double)kScatterPieceMin)) piece = (int)one;
  const int mc = scatter_max_chunks(d.n_g, tx * ty, piece);
  if (tx * ty > d.tile_cap || mc > d.chunk_cap || chunk <= 0 || chunk >= 65536) return false;
  d.tile_w = tw; d.tile_h = th; d.tiles_x = tx; d.tiles_y = ty;
  d.chunk = chunk;
  d.piece = piece;
  d.max_chunks = mc;
  return true;
}

// the window: one 32-bit word, or two (16-bit split), per bin of the tile and
// its margin, for the inst and the filler set
size_t scatter_smem(const DeviceModel& d) {
  return (size_t)(scatter_one_word(d) ? 2 : 4) * (d.tile_w + 2 * kTileMargin) * (d.tile_h + 2 * kTileMargin) * 4;
}

int scatter_prepare_device() {
  static PerContext<char> contexts;
  char done;
  return contexts.get(&done, [](char&) -> int {
    const int side = kTileSides[sizeof(kTileSides) / sizeof(kTileSides[0]) - 1];
    const int smem = 4 * (side + 2 * kTileMargin) * (side + 2 * kTileMargin) * 4;
    GPL_CUDA(cudaFuncSetAttribute(k_scatter<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    GPL_CUDA(cudaFuncSetAttribute(k_scatter<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return GPL_OK;
  });
}

int launch_tile_order(DeviceModel& d, int slot, cudaStream_t s, Timer& t) {
  OrderArgs O;
  O.geo = geom(d);
  O.n_g = d.n_g;
  O.tile_w = d.tile_w; O.tile_h = d.tile_h; O.tiles_x = d.tiles_x; O.tiles_y = d.tiles_y;
  // slot < 0: the slot the control record's predictor starts from
  O.slp = slot >= 0 ? d.slp[slot] : nullptr;
  for (int k = 0; k < 4; k++) O.slp_all[k] = d.slp[k];
  O.ctl = d.ctl;
  O.chunk = d.piece;
  O.tile_count = d.tile_count; O.tile_start = d.tile_start; O.order = d.order;
  O.chunks = d.chunks; O.n_chunks = d.n_chunks;
  t.begin(kKOther);
  GPL_CUDA(cudaMemsetAsync(d.tile_count, 0, sizeof(int32_t) * d.tiles_x * d.tiles_y, s));
  k_order_count<<<cell_blocks(d), kBlock, 0, s>>>(O);
  k_order_scan<<<1, kOrderScanT, 0, s>>>(O);
  k_order_fill<<<cell_blocks(d), kBlock, 0, s>>>(O);
  t.end(kKOther);
  t.count(3);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

// The gcell kernel's grid-stride loop runs on one wave of resident blocks
// (kCellBlocksPerSm per SM at its register count), so its last-block
// reduction waits for no second wave.
int cell_grid(const DeviceModel& d) { return std::max(1, std::min(cell_blocks(d), d.sm_count * kCellBlocksPerSm)); }

int launch_cell(DeviceModel& d, const EvalArgs& a, int n_phi_blocks, bool to_host, cudaStream_t s, Timer& t) {
  CellArgs A = cell_args(d, a, n_phi_blocks);
  if (to_host) A.out_host = d.result_h;
  t.begin(kKCell);
  if (d.n_big) k_dgrad_big<<<d.n_big, kBlock, 0, s>>>(A, d.big_cells, d.n_big);
  k_cell<<<cell_grid(d), kBlock, 0, s>>>(A);
  t.end(kKCell);
  t.count(d.n_big ? 2 : 1);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

namespace {
// updateInitialPrevSLPCoordi (src/nesterovPlace.cpp:492-512):
// prev = inside(cur + coef * sum), one clamp per axis.
__global__ void __launch_bounds__(kBlock) k_initial_prev(BinGeom G, int n_g, const int4* geo,
                                                         const float2* cur, const float2* sum, float coef,
                                                         float2* out) {
  const int g = blockIdx.x * kBlock + threadIdx.x;
  if (g >= n_g) return;
  const int2 h = gcell_geo(geo[g]).half;
  const float2 c = cur[g], s = sum[g];
  const float x = __fadd_rn(c.x, __fmul_rn(coef, s.x));
  const float y = __fadd_rn(c.y, __fmul_rn(coef, s.y));
  out[g] = make_float2(inside(x, h.x, G.core_lx, G.core_ux), inside(y, h.y, G.core_ly, G.core_uy));
}
}  // namespace

int launch_initial_prev(DeviceModel& d, const float2* cur_slp, const float2* cur_sum, float coef,
                        float2* out, cudaStream_t s, Timer& t) {
  t.begin(kKOther);
  k_initial_prev<<<cell_blocks(d), kBlock, 0, s>>>(geom(d), d.n_g, d.g_geo, cur_slp, cur_sum, coef, out);
  t.end(kKOther);
  t.count(1);
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

int launch_sum_phi(DeviceModel& d, int area_set, cudaStream_t s, Timer& t, int* n_blocks) {
  const int nb = d.cnt_x * d.cnt_y;
  const int blocks = std::min((nb + kBlock - 1) / kBlock, d.part_stride);
  t.begin(kKOther);
  k_sum_phi<<<blocks, kBlock, 0, s>>>(d.phi, d.area[area_set], d.nonplace, nb,
                                     d.part + (size_t)kPartPhi * d.part_stride);
  t.end(kKOther);
  t.count(1);
  GPL_CUDA(cudaGetLastError());
  *n_blocks = blocks;
  return GPL_OK;
}

// ------------------------------------------------------------ batched form
// Many jobs' evaluations in one launch per phase: a persistent grid whose
// blocks take work items (instance, block of that instance's own launch,
// that launch's grid) from a table and run the same block body as the
// per-job kernels, on the instance's arguments (kept in device memory).  A
// job's blocks therefore compute exactly what its own launch computes.
namespace {

struct ScatterBatchArgs {
  ScatterArgs A;
  TileArgs T;
  const int32_t* big;
};

struct CellBatchArgs {
  CellArgs A;
  const int32_t* big;
};

__global__ void __launch_bounds__(kBlock, 5) k_scatter_batch(const ScatterBatchArgs* args, const int4* items,
                                                             const int* count) {
  extern __shared__ __align__(16) unsigned win[];
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    const ScatterBatchArgs& a = args[it.x];
    if (a.A.one_word) scatter_body<true>(a.A, a.T, it.y, win);
    else scatter_body<false>(a.A, a.T, it.y, win);
    __syncthreads();                  // the window is the next item's
  }
}

__global__ void __launch_bounds__(kBlock) k_scatter_big_batch(const ScatterBatchArgs* args, const int4* items,
                                                              const int* count) {
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    scatter_big_body(args[it.x].A, args[it.x].big, it.y);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kBlock) k_dgrad_big_batch(const CellBatchArgs* args, const int4* items,
                                                            const int* count) {
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    dgrad_big_body(args[it.x].A, args[it.x].big, it.y);
    __syncthreads();
  }
}

// (fewer resident blocks than the per-job kernel: the work-item loop and the
// arguments read from memory need the registers)
__global__ void __launch_bounds__(kBlock, 4) k_cell_batch(const CellBatchArgs* args,
                                                                         const int4* items, const int* count) {
  const int n = *count;
  for (int w = blockIdx.x; w < n; w += gridDim.x) {
    const int4 it = items[w];
    cell_body(args[it.x].A, it.y, it.z);
    __syncthreads();
  }
}

}  // namespace

size_t scatter_batch_args_bytes() { return sizeof(ScatterBatchArgs); }
size_t cell_batch_args_bytes() { return sizeof(CellBatchArgs); }

void write_scatter_batch_args(const DeviceModel& d, void* dst) {
  ScatterBatchArgs x;
  x.A = scatter_args(d);
  x.T = tile_args(d);
  x.big = d.big_cells;
  memcpy(dst, &x, sizeof(x));
}

void write_cell_batch_args(const DeviceModel& d, const EvalArgs& a, void* dst) {
  CellBatchArgs x;
  x.A = cell_args(d, a, 0);
  x.big = d.big_cells;
  memcpy(dst, &x, sizeof(x));
}

int scatter_batch_prepare_device() {
  static PerContext<char> contexts;
  char done;
  return contexts.get(&done, [](char&) -> int {
    const int side = kTileSides[sizeof(kTileSides) / sizeof(kTileSides[0]) - 1];
    const int smem = 4 * (side + 2 * kTileMargin) * (side + 2 * kTileMargin) * 4;
    GPL_CUDA(cudaFuncSetAttribute(k_scatter_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return GPL_OK;
  });
}

int launch_density_batch(int phase, const void* args, const int4* items, const int* count, int grid,
                         size_t smem, cudaStream_t s) {
  switch (phase) {
    case kBScatter:
      k_scatter_batch<<<grid, kBlock, smem, s>>>(static_cast<const ScatterBatchArgs*>(args), items, count);
      break;
    case kBScatterBig:
      k_scatter_big_batch<<<grid, kBlock, 0, s>>>(static_cast<const ScatterBatchArgs*>(args), items, count);
      break;
    case kBDgradBig:
      k_dgrad_big_batch<<<grid, kBlock, 0, s>>>(static_cast<const CellBatchArgs*>(args), items, count);
      break;
    case kBCell:
      k_cell_batch<<<grid, kBlock, 0, s>>>(static_cast<const CellBatchArgs*>(args), items, count);
      break;
    default:
      set_error("launch_density_batch: unknown phase");
      return GPL_ERR_INVALID_ARG;
  }
  GPL_CUDA(cudaGetLastError());
  return GPL_OK;
}

}  // namespace gpl
