// Tiles of output pixels with their source windows in shared memory, channel by channel, for the gradient kernels in fp32 arithmetic
// (dk_local_f32.cu, dk_local_pieces.cu).
#pragma once

#include "dk_common.cuh"

namespace dk {
namespace {

struct TilePlan {
  int TH, TW;                 // output pixels of a tile
  int across, down;           // tiles per row of tiles, per sample
  int tiles;                  // over the batch
  int XH, XW;                 // source rows and columns of a tile
  int xpitch, ypitch;         // words per channel in shared memory
  unsigned magic_x, magic_y;  // ceil(2^32 / XW), ceil(2^32 / TW)
  int per_block, blocks;      // tiles per block, blocks (bank)
  size_t smem;
};

TilePlan tile_plan(const Geom& g, int pixels) {
  TilePlan t;
  const int widest = pixels < 32 ? pixels : 32;
  t.across = (g.Wo + widest - 1) / widest;
  t.TW = (g.Wo + t.across - 1) / t.across;
  t.TH = pixels / t.TW;
  if (t.TH > g.Ho) t.TH = g.Ho;
  t.down = (g.Ho + t.TH - 1) / t.TH;
  t.TH = (g.Ho + t.down - 1) / t.down;
  t.tiles = g.N * t.down * t.across;
  t.XH = (t.TH - 1) * g.sH + 3;
  t.XW = (t.TW - 1) * g.sW + 3;
  t.xpitch = (t.XH * t.XW) | 1;
  t.ypitch = (t.TH * t.TW) | 1;
  t.magic_x = (unsigned)((0x100000000ull + t.XW - 1) / t.XW);
  t.magic_y = t.TW == 1 ? 0 : (unsigned)((0x100000000ull + t.TW - 1) / t.TW);
  t.per_block = 1;
  t.blocks = t.tiles;
  t.smem = 0;
  return t;
}

__device__ __forceinline__ int over(int e, int d, unsigned magic) { return d == 1 ? e : (int)__umulhi((unsigned)e, magic); }
__device__ __forceinline__ float hat1(float t) { return __saturatef(1.f - fabsf(t)); }  // max(0, 1 - |t|)

struct TilePos {
  int n, oh0, ow0;
};
__device__ __forceinline__ TilePos tile_pos(int tile, const TilePlan& t) {
  TilePos p;
  const int row = tile / t.across;
  p.ow0 = (tile - row * t.across) * t.TW;
  p.n = row / t.down;
  p.oh0 = (row - p.n * t.down) * t.TH;
  return p;
}

// 4 bytes from global to shared memory, asynchronously; zero where !ok (the address is not read then)
__device__ __forceinline__ void copy4(unsigned dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0));
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// One tile (rows x cols from row r0, column q0 of H x W planes) of 32 planes, the first n_c of which exist, into shared
// memory; zero outside the planes.  All of a warp's copies are in flight at once, and a lane keeps its place in the tile and
// walks down the channels: two additions per copy (with the whole address computed for each, the copies were half of all
// instructions).  fp16 planes are widened on the way, through registers.
template <int WARPS, typename T>
__device__ __forceinline__ void stage_planes(float* s, const T* __restrict__ g0, int rows, int cols, unsigned magic, int pitch, int r0,
                                             int q0, int H, int W, int n_c, int warp, int lane) {
  const size_t plane = (size_t)H * W;
  const unsigned s0 = (unsigned)__cvta_generic_to_shared(s) + 4u * (unsigned)(warp * pitch);
  const unsigned d_step = 4u * (unsigned)(WARPS * pitch);
#pragma unroll sizeof(T) == 2 ? 2 : 1
  for (int e = lane; e < rows * cols; e += 32) {
    const int r = over(e, cols, magic), ih = r0 + r, iw = q0 + (e - r * cols);
    const bool in = ih >= 0 && ih < H && iw >= 0 && iw < W;
    const T* src = g0 + (size_t)warp * plane + (in ? ih * W + iw : 0);
    if constexpr (sizeof(T) == 4) {
      unsigned dst = s0 + 4u * e;
#pragma unroll
      for (int ch = 0; ch < 32; ch += WARPS) {
        if (ch + warp < 32) copy4(dst, src, in && ch + warp < n_c);
        dst += d_step;
        src += WARPS * plane;
      }
    } else {
      constexpr int kEach = (32 + WARPS - 1) / WARPS;
      float v[kEach];
#pragma unroll
      for (int i = 0; i < kEach; ++i) v[i] = in && i * WARPS + warp < n_c ? ld<float>(src + (size_t)(i * WARPS) * plane) : 0.f;
#pragma unroll
      for (int i = 0; i < kEach; ++i)
        if (i * WARPS + warp < 32) s[(i * WARPS + warp) * pitch + e] = v[i];
    }
  }
}
template <int S, int WARPS, typename T>
__device__ __forceinline__ void stage_tile(float* xs, float* ys, const T* __restrict__ x, const T* __restrict__ dy, const Geom& g,
                                           const TilePlan& t, const TilePos& tp, int c0, int warp, int lane) {
  const int n_c = min(32, g.C - c0);
  stage_planes<WARPS>(xs, x + ((size_t)tp.n * g.C + c0) * g.HW, t.XH, t.XW, t.magic_x, t.xpitch, tp.oh0 * S - 1, tp.ow0 * S - 1, g.H, g.W,
                      n_c, warp, lane);
  stage_planes<WARPS>(ys, dy + ((size_t)tp.n * g.C + c0) * g.P, t.TH, t.TW, t.magic_y, t.ypitch, tp.oh0, tp.ow0, g.Ho, g.Wo, n_c, warp, lane);
}

// ------------------------------------------------------------------ bank
// Dense in the cells, a product dy x that is not finite reaches all cells of its channel (times a hat of zero) where only those of its
// sample should have it.  A block whose sums are not finite starts again with this: one product to the four cells it belongs to.
// acc: the lane's sums, [cell 4 x 4][32].
__device__ __forceinline__ void add_to_cells(float* acc, float dk, float u, float v, const Geom& g) {
  if (!(u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW)) return;
  const int a0 = (int)floorf(u), b0 = (int)floorf(v);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int a = a0 + (q >> 1), b = b0 + (q & 1);
    if (a >= 0 && a < g.scH && b >= 0 && b < g.scW) acc[(a * 4 + b) * 32] += hat1(u - (float)a) * hat1(v - (float)b) * dk;
  }
}

// All tiles of a block, a pixel per warp; bilinear samples of x at `off`, or x itself (off null).  red: [warp][cell][lane].
template <typename T>
__device__ __noinline__ void bank_by_cells(float* red, const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ off,
                                           const T* __restrict__ rot, const Geom& g, const TilePlan& t, int c0, int warp, int warps, int lane) {
  float* acc = red + warp * 512 + lane;
  for (int i = 0; i < 16; ++i) acc[i * 32] = 0.f;
  const unsigned live = __ballot_sync(0xffffffffu, c0 + lane < g.C);
  if (c0 + lane >= g.C) return;
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  const int first = blockIdx.x * t.per_block, last = min(first + t.per_block, t.tiles);
  // a NaN stays: once every sum of the warp is one there is nothing left to find out
  auto settled = [&]() {
    bool all = true;
    for (int i = 0; i < 16; ++i)
      if ((i >> 2) < g.scH && (i & 3) < g.scW) all &= acc[i * 32] != acc[i * 32];
    return __all_sync(live, all);
  };
  for (int tile = first; tile < last && !settled(); ++tile) {
    const TilePos tp = tile_pos(tile, t);
    const T* xc = x + ((size_t)tp.n * g.C + c0 + lane) * g.HW;
    for (int p = warp; p < t.TH * t.TW; p += warps) {
      const int oh = tp.oh0 + p / t.TW, ow = tp.ow0 + p % t.TW;
      if (oh >= g.Ho || ow >= g.Wo) continue;
      const int pix = oh * g.Wo + ow;
      const float yv = ld<float>(dy + ((size_t)tp.n * g.C + c0 + lane) * g.P + pix);
      for (int tap = 0; tap < 9; ++tap) {
        const int fh = tap / 3, fw = tap - fh * 3, ih = oh * g.sH - g.pH + fh * g.dH, iw = ow * g.sW - g.pW + fw * g.dW;
        const size_t o = ((size_t)tp.n * 18 + 2 * tap) * g.P + pix;
        float xv = 0.f;
        if (off != nullptr) {
          Bilinear<float> bi;
          if (!image_setup<float>((float)ih + ld<float>(off + o), (float)iw + ld<float>(off + o + g.P), g, bi)) continue;
          float sc[4];
          bilinear_value_coefs(bi, sc);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (bi.m[q]) xv = fmaf(sc[q], ld<float>(xc + bi.idx[q]), xv);
        } else {
          if (ih < 0 || ih >= g.H || iw < 0 || iw >= g.W) continue;
          xv = ld<float>(xc + ih * g.W + iw);
        }
        add_to_cells(acc, yv * xv, ((float)fh + ld<float>(rot + o)) + uh0, ((float)fw + ld<float>(rot + o + g.P)) + uw0, g);
      }
    }
  }
}

}  // namespace
}  // namespace dk
