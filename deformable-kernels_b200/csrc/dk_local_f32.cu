// Offset and bank gradients of the local deformable kernel in fp32 arithmetic (fp32 tensors, and fp16 where the tensor-core kernels do
// not apply), and the bank gradient of DK + DCN where those do not apply (3 x 3 taps, scopes up to 4 x 4).
//
// Both consume the products dK = dy * x, and both are dense in the 16 bank cells here: with the hat products the sampled
// cells need no data-dependent addresses, so every bank value and every hat product is one broadcast read for a whole warp.
//   bank      lanes = channels: dW[c, cell] += dK * hat_u * hat_v, 16 accumulators per lane kept in registers over all of the
//             block's pixels; x and dy of a pixel tile come through shared memory (fetched with neighbours on neighbouring
//             lanes, read back one channel per lane), the hats of a (pixel, tap) are two 16-byte broadcasts
//   offsets   lanes = pixels: G[tap, cell] += dK * W[c, cell], a warp per kernel row (48 accumulators), channel after channel;
//             then the floor-based derivative weights contract G
// 21 (bank) and 17 (offsets) multiply-adds per pixel, tap and channel, packed in pairs, beside the loads.  The bank kernel keeps the FMA
// pipe at 55 % and the issue slots at 56 % with the 16 warps that its registers allow: bound by the latency of the loads between the
// products.  The bank kernel before gathered four cells per tap with an address per lane, read x and dy one channel per lane
// from global memory (a line per lane) and added into shared memory: N = 64, C = 144, 56 x 56 2088 -> 384 us (stride 2 562 ->
// 119, N = 32, C = 384, 14 x 14 115 -> 39).
#include <cuda_runtime.h>

#include "dk_f32_tiles.cuh"

namespace dk {

namespace {

__device__ __forceinline__ bool all_finite(const unsigned long long (&acc)[2][4]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float2 v = unpair(acc[i >> 2][i & 3]);
    ok &= fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY;
  }
  return ok;
}

constexpr int kBankWarps = 8;

template <typename T, int S>
__global__ void __launch_bounds__(32 * kBankWarps, 2) f32_bank_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                      const T* __restrict__ rot, float* __restrict__ partial,
                                                                      const __grid_constant__ Geom g, const __grid_constant__ TilePlan t) {
  extern __shared__ __align__(16) float smem_f[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = blockIdx.y * 32, px = t.TH * t.TW;
  float4* hats = reinterpret_cast<float4*>(smem_f);  // [pixel][tap][hat_u | hat_v]
  float* xs = smem_f + (size_t)px * 72;
  float* ys = xs + 32 * t.xpitch;
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  unsigned long long acc[2][4];  // cell rows (2i, 2i + 1) of column k
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i >> 2][i & 3] = 0;
  const int first = blockIdx.x * t.per_block, last = min(first + t.per_block, t.tiles);
  for (int tile = first; tile < last; ++tile) {
    const TilePos tp = tile_pos(tile, t);
    __syncthreads();
    stage_tile<S, kBankWarps>(xs, ys, x, dy, g, t, tp, c0, warp, lane);
    for (int i = threadIdx.x; i < px * 9; i += 32 * kBankWarps) {
      const int tap = i / px, p = i - tap * px, r = over(p, t.TW, t.magic_y);
      const int oh = tp.oh0 + r, ow = tp.ow0 + (p - r * t.TW), fh = tap / 3, fw = tap - fh * 3;
      float u = -8.f, v = -8.f;  // samples nothing
      if (oh < g.Ho && ow < g.Wo) {
        const T* rp = rot + ((size_t)tp.n * 18 + 2 * tap) * g.P + oh * g.Wo + ow;
        u = ((float)fh + ld<float>(rp)) + uh0;
        v = ((float)fw + ld<float>(rp + g.P)) + uw0;
      }
      float4 hu, hv;
      hu.x = hat1(u), hu.y = g.scH > 1 ? hat1(u - 1.f) : 0.f, hu.z = g.scH > 2 ? hat1(u - 2.f) : 0.f, hu.w = g.scH > 3 ? hat1(u - 3.f) : 0.f;
      hv.x = hat1(v), hv.y = g.scW > 1 ? hat1(v - 1.f) : 0.f, hv.z = g.scW > 2 ? hat1(v - 2.f) : 0.f, hv.w = g.scW > 3 ? hat1(v - 3.f) : 0.f;
      hats[(p * 9 + tap) * 2] = hu;
      hats[(p * 9 + tap) * 2 + 1] = hv;
    }
    copies_done();
    __syncthreads();
    for (int p = warp; p < px; p += kBankWarps) {
      const int r = over(p, t.TW, t.magic_y);
      const float* xp = xs + lane * t.xpitch + r * S * t.XW + (p - r * t.TW) * S;
      const float yv = ys[lane * t.ypitch + p];
      const float4* hp = hats + p * 18;
#pragma unroll
      for (int i = 0; i < 9; ++i) {
        const float dk = yv * xp[(i / 3) * t.XW + i % 3];
        const ulonglong2 hu = *reinterpret_cast<const ulonglong2*>(hp + 2 * i);
        const float4 hv = hp[2 * i + 1];
        const float b[4] = {dk * hv.x, dk * hv.y, dk * hv.z, dk * hv.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const unsigned long long bb = pair(b[k], b[k]);
          fma2(acc[0][k], hu.x, bb);
          fma2(acc[1][k], hu.y, bb);
        }
      }
    }
  }
  float* red = smem_f;  // [warp][cell][lane]
  if (__syncthreads_or(!all_finite(acc))) {
    bank_by_cells<T>(red, dy, x, nullptr, rot, g, t, c0, warp, kBankWarps, lane);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = unpair(acc[i >> 2][i & 3]);
      const int cell = (i >> 2) * 8 + (i & 3);
      red[(warp * 16 + cell) * 32 + lane] = v.x;
      red[(warp * 16 + cell + 4) * 32 + lane] = v.y;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * 16; i += 32 * kBankWarps) {
    const int cell = i >> 5, a = cell >> 2, b = cell & 3, c = c0 + (i & 31);
    if (c < g.C && a < g.scH && b < g.scW) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < kBankWarps; ++w) s += red[w * 512 + i];
      partial[((size_t)blockIdx.x * g.C + c) * g.cells + a * g.scW + b] = s;
    }
  }
}

// ------------------------------------------------------------------ offsets
// 12 warps: kernel row x (PQ quads of 32 pixels, 4 / PQ shares of the channels).  A sum over L channels in one register is off by
// about 8.6e-8 sqrt(L / 24) (each addition by up to half a unit of the sum so far).  The eight warps of the general kernel keep L at
// C / 8 but lose another 1.1e-7 where the coordinate is rounded at its full size.  That part is kept here (`rest`), so chains of
// C / 8 + 39 channels are as near to fp64; after one, a share contracts what it has and adds up two numbers per tap.  2-norm:
// C = 960, 7 x 7 general kernel 2.3e-7, this one 2.2e-7, with chains of C / 4 3.0e-7.
constexpr int kOffWarps = 12;
constexpr int kChainSlack = 39;

template <typename T, int S, int PQ>
__global__ void __launch_bounds__(32 * kOffWarps, 2) f32_offsets_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                        const T* __restrict__ rot, const T* __restrict__ w,
                                                                        T* __restrict__ drot, const Geom g, const TilePlan t) {
  constexpr int SH = 4 / PQ;
  extern __shared__ __align__(16) float smem_f[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fh = warp % 3, k = warp / 3, quad = k % PQ, share = k / PQ;
  float* ws = smem_f;  // [channel][16 cells]
  float* xs = ws + 32 * 16;
  float* ys = xs + 32 * t.xpitch;
  const TilePos tp = tile_pos(blockIdx.x, t);
  const int px = t.TH * t.TW;
  const int p = quad * 32 + lane, pc = p < px ? p : 0, r = over(pc, t.TW, t.magic_y), col = pc - r * t.TW;
  const int xo = (r * S + fh) * t.XW + col * S;
  const int oh = tp.oh0 + r, ow = tp.ow0 + col;
  const bool live = p < px && oh < g.Ho && ow < g.Wo;
  const size_t o0 = ((size_t)tp.n * 18 + 6 * fh) * g.P + (live ? oh * g.Wo + ow : 0);
  unsigned long long G2[3][8];  // cells (2i, 2i + 1)
  float sum[3][2];
#pragma unroll
  for (int i = 0; i < 24; ++i) G2[i / 8][i % 8] = 0;
#pragma unroll
  for (int i = 0; i < 6; ++i) sum[i >> 1][i & 1] = 0.f;
  // sum += G times the floor-based derivative weights of the tap's four cells; the other cells are not read
  auto contract = [&]() {
    const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
    const int ih = oh * S - 1 + fh;
#pragma unroll
    for (int fw = 0; fw < 3; ++fw) {
      const int iw = ow * S - 1 + fw;
      const float ru = ld<float>(rot + o0 + (size_t)(2 * fw) * g.P), rv = ld<float>(rot + o0 + (size_t)(2 * fw + 1) * g.P);
      const float u = ((float)fh + ru) + uh0, v = ((float)fw + rv) + uw0;
      if (live && ih >= 0 && ih < g.H && iw >= 0 && iw < g.W && u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW) {
        const float fu = floorf(u), fv = floorf(v);
        // tap + shift is a small multiple of 1/2: u minus it is exact, and so is what the rounding of u lost
        const float lh = (u - fu) + (ru - (u - ((float)fh + uh0))), lw = (v - fv) + (rv - (v - ((float)fw + uw0)));
        const int a0 = (int)fu, b0 = (int)fv;
        float gu = 0.f, gv = 0.f;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          float su = 0.f, sv = 0.f;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const float2 two = unpair(G2[fw][2 * a + (b >> 1)]);
            const float v2 = b & 1 ? two.y : two.x;
            if (b == b0) su = fmaf(1.f - lw, v2, su), sv -= v2;
            if (b == b0 + 1) su = fmaf(lw, v2, su), sv += v2;
          }
          if (a == a0) gu -= su, gv = fmaf(1.f - lh, sv, gv);
          if (a == a0 + 1) gu += su, gv = fmaf(lh, sv, gv);
        }
        sum[fw][0] += gu, sum[fw][1] += gv;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) G2[fw][i] = 0;
    }
  };
  const int chunks = (g.C + 31) / 32, per = max((g.C / 8 + kChainSlack) * SH / 32, 1);
  for (int chunk = 0, left = per; chunk < chunks; ++chunk) {
    const int c0 = chunk * 32;
    __syncthreads();
    stage_tile<S, kOffWarps>(xs, ys, x, dy, g, t, tp, c0, warp, lane);
    for (int i = threadIdx.x; i < 32 * 16; i += 32 * kOffWarps) {
      const int c = c0 + (i >> 4), a = (i >> 2) & 3, b = i & 3;
      ws[i] = c < g.C && a < g.scH && b < g.scW ? ld<float>(w + (size_t)c * g.cells + a * g.scW + b) : 0.f;
    }
    copies_done();
    __syncthreads();
    const int n_c = min(32, g.C - c0);
    const float *yp = ys + share * t.ypitch + pc, *xp = xs + share * t.xpitch + xo;
    const ulonglong2* wp = reinterpret_cast<const ulonglong2*>(ws + share * 16);
#pragma unroll 4
    for (int ch = share; ch < n_c; ch += SH, yp += SH * t.ypitch, xp += SH * t.xpitch, wp += SH * 4) {
      const float yv = *yp;
      unsigned long long d[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const float v = yv * xp[a];
        d[a] = pair(v, v);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const ulonglong2 wv = wp[q];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          fma2(G2[a][2 * q], d[a], wv.x);
          fma2(G2[a][2 * q + 1], d[a], wv.y);
        }
      }
    }
    if (--left == 0 || chunk + 1 == chunks) contract(), left = per;
  }
  if (SH > 1) {  // the shares' sums, in order
    float* red = smem_f + (quad * 3 + fh) * ((SH - 1) * 6 * 32) + lane;  // [share - 1][tap, direction][lane]
    __syncthreads();
    if (share > 0) {
#pragma unroll
      for (int i = 0; i < 6; ++i) red[((share - 1) * 6 + i) * 32] = sum[i >> 1][i & 1];
    }
    __syncthreads();
    if (share == 0) {
#pragma unroll
      for (int s = 1; s < SH; ++s)
#pragma unroll
        for (int i = 0; i < 6; ++i) sum[i >> 1][i & 1] += red[((s - 1) * 6 + i) * 32];
    }
  }
  if (share != 0 || !live) return;
#pragma unroll
  for (int i = 0; i < 6; ++i) st<T, float>(drot + o0 + (size_t)i * g.P, sum[i >> 1][i & 1]);
}

// ------------------------------------------------------------------ bank of DK + DCN
// The same with x read by bilinear sampling: a warp per tap and a lane per pixel sample the 32 channels first (corners and
// coefficients once per pixel and tap, neighbours on neighbouring lanes) and leave the samples in shared memory, where the
// lanes take a channel each.  Before, every lane followed its own channel through global memory, or through whole planes on
// chip with read-modify-writes of the bank cells in shared memory: 16 x 192 channels of 28 x 28, 3 x 3 scope, 167 -> 112 us;
// 13 x 96 of 80 x 80 (planes too big to hold) 1324 -> 391; fp16, 13 x 88 of 80 x 80, 1177 -> 377.  Bound by the latency of
// the corner loads.
constexpr int kTapWarps = 9;
constexpr int kSamplePitch = 32 * 9 + 1;

template <typename T>
__global__ void __launch_bounds__(32 * kTapWarps, 2) deform_bank_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                        const T* __restrict__ off, const T* __restrict__ rot,
                                                                        float* __restrict__ partial, const __grid_constant__ Geom g,
                                                                        const __grid_constant__ TilePlan t) {
  extern __shared__ __align__(16) float smem_f[];
  const int lane = threadIdx.x & 31, tap = threadIdx.x >> 5;
  const int c0 = blockIdx.y * 32, n_c = min(32, g.C - c0), px = t.TH * t.TW;
  float4* hats = reinterpret_cast<float4*>(smem_f);  // [pixel][tap][hat_u | hat_v]
  float* xs = smem_f + 32 * 72;                      // [channel][pixel][tap]
  float* ys = xs + 32 * kSamplePitch;                // [channel][33]
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  const int fh = tap / 3, fw = tap - fh * 3;
  unsigned long long acc[2][4];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i >> 2][i & 3] = 0;
  const int first = blockIdx.x * t.per_block, last = min(first + t.per_block, t.tiles);
  const int r = over(lane, t.TW, t.magic_y);
  for (int tile = first; tile < last; ++tile) {
    const TilePos tp = tile_pos(tile, t);
    const int oh = tp.oh0 + r, ow = tp.ow0 + (lane - r * t.TW);
    const bool live = lane < px && oh < g.Ho && ow < g.Wo;
    const size_t o = ((size_t)tp.n * 18 + 2 * tap) * g.P + (live ? oh * g.Wo + ow : 0);
    Bilinear<float> bi;
    float sc[4] = {0.f, 0.f, 0.f, 0.f};
    bool used = false;
    float4 hu = make_float4(0.f, 0.f, 0.f, 0.f), hv = hu;
    if (live) {
      used = image_setup<float>((float)(oh * g.sH - g.pH + fh * g.dH) + ld<float>(off + o),
                                (float)(ow * g.sW - g.pW + fw * g.dW) + ld<float>(off + o + g.P), g, bi);
      if (used) {
        bilinear_value_coefs(bi, sc);
        const float u = ((float)fh + ld<float>(rot + o)) + uh0, v = ((float)fw + ld<float>(rot + o + g.P)) + uw0;
        hu.x = hat1(u), hu.y = g.scH > 1 ? hat1(u - 1.f) : 0.f, hu.z = g.scH > 2 ? hat1(u - 2.f) : 0.f, hu.w = g.scH > 3 ? hat1(u - 3.f) : 0.f;
        hv.x = hat1(v), hv.y = g.scW > 1 ? hat1(v - 1.f) : 0.f, hv.z = g.scW > 2 ? hat1(v - 2.f) : 0.f, hv.w = g.scW > 3 ? hat1(v - 3.f) : 0.f;
      }
    }
    __syncthreads();  // the tile before has been read
    hats[(lane * 9 + tap) * 2] = hu;
    hats[(lane * 9 + tap) * 2 + 1] = hv;
    {
      const T* xc = x + ((size_t)tp.n * g.C + c0) * g.HW;
      float* d = xs + lane * 9 + tap;
      int q[4] = {0, 0, 0, 0};
      if (used) q[0] = bi.idx[0], q[1] = bi.idx[1], q[2] = bi.idx[2], q[3] = bi.idx[3];
#pragma unroll 4
      for (int ch = 0; ch < n_c; ++ch, xc += g.HW, d += kSamplePitch) {
        float v = 0.f;
        if (used) v = sc[0] * ld<float>(xc + q[0]) + sc[1] * ld<float>(xc + q[1]) + sc[2] * ld<float>(xc + q[2]) + sc[3] * ld<float>(xc + q[3]);
        *d = v;
      }
    }
    {
      const T* yc = dy + ((size_t)tp.n * g.C + c0) * g.P + (live ? oh * g.Wo + ow : 0);
      for (int ch = tap; ch < n_c; ch += kTapWarps) ys[ch * 33 + lane] = live ? ld<float>(yc + (size_t)ch * g.P) : 0.f;
    }
    __syncthreads();
    if (lane < n_c) {
      for (int p = tap; p < px; p += kTapWarps) {
        const float* xp = xs + lane * kSamplePitch + p * 9;
        const float yv = ys[lane * 33 + p];
        const float4* hp = hats + p * 18;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
          const float dk = yv * xp[i];
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(hp + 2 * i);
          const float4 b = hp[2 * i + 1];
          const float bb[4] = {dk * b.x, dk * b.y, dk * b.z, dk * b.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned long long w2 = pair(bb[k], bb[k]);
            fma2(acc[0][k], a.x, w2);
            fma2(acc[1][k], a.y, w2);
          }
        }
      }
    }
  }
  float* red = smem_f;  // [warp][cell][lane]
  if (__syncthreads_or(!all_finite(acc))) {
    bank_by_cells<T>(red, dy, x, off, rot, g, t, c0, tap, kTapWarps, lane);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = unpair(acc[i >> 2][i & 3]);
      const int cell = (i >> 2) * 8 + (i & 3);
      red[(tap * 16 + cell) * 32 + lane] = v.x;
      red[(tap * 16 + cell + 4) * 32 + lane] = v.y;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * 16; i += 32 * kTapWarps) {
    const int cell = i >> 5, a = cell >> 2, b = cell & 3, c = c0 + (i & 31);
    if (c < g.C && a < g.scH && b < g.scW) {
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < kTapWarps; ++w) sum += red[w * 512 + i];
      partial[((size_t)blockIdx.x * g.C + c) * g.cells + a * g.scW + b] = sum;
    }
  }
}
constexpr size_t kDeformBankSmem = (32 * 72 + 32 * (size_t)kSamplePitch + 32 * 33) * sizeof(float);
static_assert(kDeformBankSmem >= (size_t)kTapWarps * 512 * sizeof(float), "the warps' sums reuse the tile's room");

// ------------------------------------------------------------------ host side
bool deform_bank_shape(const Geom& g) {
  return g.kH == 3 && g.kW == 3 && g.G == 1 && g.scH <= 4 && g.scW <= 4 && (long long)g.N * g.P < 0x3fffffff && (g.C + 31) / 32 <= 65535;
}
TilePlan deform_bank_plan(const Geom& g) {
  TilePlan t = tile_plan(g, 32);
  int want = 4 * device_sm_count() / ((g.C + 31) / 32);
  if (want < 1) want = 1;
  t.per_block = (t.tiles + want - 1) / want;
  t.blocks = (t.tiles + t.per_block - 1) / t.per_block;
  t.smem = kDeformBankSmem;
  return t;
}
bool f32_shape(const Geom& g) {
  return g.kH == 3 && g.kW == 3 && g.dH == 1 && g.dW == 1 && g.pH == 1 && g.pW == 1 && g.sH == g.sW && (g.sH == 1 || g.sH == 2) &&
         g.G == 1 && g.scH <= 4 && g.scW <= 4 && (long long)g.N * g.P < 0x3fffffff;
}

// Tiles of up to 128 pixels; smaller ones while that leaves SMs without a block; then as many blocks as are resident at once.
TilePlan bank_plan(const Geom& g) {
  const int groups = (g.C + 31) / 32;
  TilePlan t = tile_plan(g, 128);
  for (int px = 64; px >= 16 && (long long)t.tiles * groups < 2LL * device_sm_count(); px /= 2) t = tile_plan(g, px);
  int want = 2 * device_sm_count() / groups;
  if (want < 1) want = 1;
  t.per_block = (t.tiles + want - 1) / want;
  t.blocks = (t.tiles + t.per_block - 1) / t.per_block;
  t.smem = ((size_t)t.TH * t.TW * 72 + 32 * (size_t)(t.xpitch + t.ypitch)) * sizeof(float);
  const size_t red = (size_t)kBankWarps * 512 * sizeof(float);
  if (t.smem < red) t.smem = red;
  return t;
}

}  // namespace

size_t local_filter_f32_workspace(const Geom& g) {
  return f32_shape(g) ? (size_t)bank_plan(g).blocks * g.C * g.cells * sizeof(float) : 0;
}

template <typename T>
int local_filter_f32(const T* dy, const T* x, const T* rot, float* partial, const Geom& g, size_t ws_bytes, int* blocks,
                     cudaStream_t s) {
  if (!f32_shape(g)) return DK_ERR_UNSUPPORTED;
  const TilePlan t = bank_plan(g);
  if (t.smem > (size_t)device_smem_optin() || (g.C + 31) / 32 > 65535) return DK_ERR_UNSUPPORTED;
  if (partial == nullptr || ws_bytes < (size_t)t.blocks * g.C * g.cells * sizeof(float)) return DK_ERR_WORKSPACE;
  auto kern = g.sH == 1 ? f32_bank_kernel<T, 1> : f32_bank_kernel<T, 2>;
  const int rc = enable_smem(kern, t.smem);
  if (rc) return rc;
  kern<<<dim3(t.blocks, (g.C + 31) / 32), 32 * kBankWarps, t.smem, s>>>(dy, x, rot, partial, g, t);
  *blocks = t.blocks;
  return check_launch();
}

template int local_filter_f32<float>(const float*, const float*, const float*, float*, const Geom&, size_t, int*, cudaStream_t);
template int local_filter_f32<__half>(const __half*, const __half*, const __half*, float*, const Geom&, size_t, int*, cudaStream_t);

template <typename T>
int local_rot_f32(const T* dy, const T* x, const T* rot, const T* w, T* drot, const Geom& g, cudaStream_t s) {
  if (!f32_shape(g)) return DK_ERR_UNSUPPORTED;
  // Calls with few pixels: the general kernel (32 pixels per block, gathered cells) leaves SMs without a block there.  N = 2, C = 64,
  // 28 x 28: 13.6 -> 10.7 us; N = 32, C = 960, 7 x 7: 109 -> 82.  With the GPU full, up to 32 channels, which that kernel's warps share
  // too thinly: 64 x 24 of 112 x 112 666 -> 327 us (fp16 633 -> 443, stride 2 172 -> 156), 64 x 16 of 56 x 56 158 -> 79; 32 x 72 139 -> 137 (fp16
  // 133 -> 195), 64 x 144 389 -> 438.
  TilePlan t = tile_plan(g, 128);
  int pq = 4;
  if (t.tiles >= 2 * device_sm_count()) {
    if (g.C > 32) return DK_ERR_UNSUPPORTED;
  } else {
    // fp16: few channels too, its planes pass through registers (2 x 24 of 14 x 14 16.5 -> 12 us, 1 x 40 of 28 x 28 19.5 -> 17; 64 x 936 of
    // 7 x 7 132 -> 177)
    if (sizeof(T) == 2 && (g.C > 64 || tile_plan(g, 32).tiles >= device_sm_count())) return DK_ERR_UNSUPPORTED;
    pq = 2, t = tile_plan(g, 64);
    if (t.tiles < 2 * device_sm_count()) pq = 1, t = tile_plan(g, 32);
  }
  size_t words = 512 + 32 * (size_t)(t.xpitch + t.ypitch);
  const size_t red = (size_t)pq * 3 * (4 / pq - 1) * 6 * 32;
  if (words < red) words = red;
  t.smem = words * sizeof(float);
  if (t.smem > (size_t)device_smem_optin()) return DK_ERR_UNSUPPORTED;
  auto kern = g.sH == 1 ? (pq == 4 ? f32_offsets_kernel<T, 1, 4> : pq == 2 ? f32_offsets_kernel<T, 1, 2> : f32_offsets_kernel<T, 1, 1>)
                        : (pq == 4 ? f32_offsets_kernel<T, 2, 4> : pq == 2 ? f32_offsets_kernel<T, 2, 2> : f32_offsets_kernel<T, 2, 1>);
  const int rc = enable_smem(kern, t.smem);
  if (rc) return rc;
  kern<<<t.tiles, 32 * kOffWarps, t.smem, s>>>(dy, x, rot, w, drot, g, t);
  return check_launch();
}
template int local_rot_f32<float>(const float*, const float*, const float*, const float*, float*, const Geom&, cudaStream_t);
template int local_rot_f32<__half>(const __half*, const __half*, const __half*, const __half*, __half*, const Geom&, cudaStream_t);

size_t deform_bank_workspace(const Geom& g) {
  return deform_bank_shape(g) ? (size_t)deform_bank_plan(g).blocks * g.C * g.cells * sizeof(float) : 0;
}

template <typename T>
int deform_bank(const T* dy, const T* x, const T* off, const T* rot, float* partial, const Geom& g, size_t ws_bytes, int* blocks,
                cudaStream_t s) {
  if (!deform_bank_shape(g)) return DK_ERR_UNSUPPORTED;
  const TilePlan t = deform_bank_plan(g);
  if (partial == nullptr || ws_bytes < (size_t)t.blocks * g.C * g.cells * sizeof(float)) return DK_ERR_WORKSPACE;
  const int rc = enable_smem(deform_bank_kernel<T>, t.smem);
  if (rc) return rc;
  deform_bank_kernel<T><<<dim3(t.blocks, (g.C + 31) / 32), 32 * kTapWarps, t.smem, s>>>(dy, x, off, rot, partial, g, t);
  *blocks = t.blocks;
  return check_launch();
}
template int deform_bank<float>(const float*, const float*, const float*, const float*, float*, const Geom&, size_t, int*, cudaStream_t);
template int deform_bank<__half>(const __half*, const __half*, const __half*, const __half*, float*, const Geom&, size_t, int*, cudaStream_t);

}  // namespace dk
