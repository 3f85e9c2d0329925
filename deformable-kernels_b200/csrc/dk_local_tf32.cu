// Offset and bank gradients of the local deformable kernel in one pass, fp32 arithmetic on the tensor cores (fp32 tensors, and fp16 where
// the fp16 kernels do not apply; 3 x 3 taps, scopes up to 4 x 4).
//
// Both are contractions of dK = dy * x with 16 cells: G[pixel, tap][cell] = sum_c dK W[c, cell] (then the floor-based derivative
// weights) and dW[c][cell] = sum over pixels and taps of dK beta[(pixel, tap), cell].  An fp32 value is two tf32 pieces, 11 bits rounded and
// the rest, so a product is three mma.m16n8k8: small * large, large * small, large * large in this order; what is left out is 2^-24 of it.
// The tensor cores truncate their sums, so no accumulator runs longer than these three: a step of 8 channels (G) or 8 pixels (dW) of a tap is
// added to the sums with one rounded addition.  fp16 banks are one piece.
//
// Block: a tile of up to 96 pixels, a warp 8 of them, over all channels, 32 at a time, whose dy and x are staged while the previous ones are
// multiplied.  G stays in registers (9 taps x 16 cells x 8 pixels per warp); the warps' bank sums of 32 channels meet in
// shared memory, in their order, and are added to the block's partial sums.
//
// fp32 64 x 144 of 56 x 56: 758 us in two kernels that gather or hold the cells with one fp32 multiply-add each -> 557.  Tensor pipe 39 %,
// issue 44 %: mma.sync and the fp32 work around it (two pieces, rounded additions) do not overlap much, three products with their pieces
// take 10.2 cycles of an SM in a loop by themselves, 6.2 of them the products (here 17, with staging, the warps' sums and tiles that do not
// fill).  At 128 registers and two blocks of eight warps the compiler moves operands about (663 us), 8 warps with 254 take as long as 12 with 168.
#include "dk_f32_tiles.cuh"

namespace dk {

namespace {

constexpr int kWarps = 12, kPixels = 8 * kWarps, kRedPitch = 40;
constexpr int kBetaBytes = kWarps * 9 * 32 * 16, kRedBytes = kWarps * 16 * kRedPitch * 4, kBankBytes = 4 * 32 * 32;
// Words of a channel of x and of dy in shared memory: 12 modulo 32, so that neither way of reading them has bank conflicts.  At stride 2 two
// buffers do not fit.
template <int S> struct Room {
  static constexpr int X = S == 1 ? 140 : 428, Y = 108, kBuffers = S == 1 ? 2 : 1, kWords = 32 * (X + Y);
  static constexpr int kBytes = kBetaBytes + kRedBytes + kBuffers * (kBankBytes + kWords * 4);
};

using f2 = unsigned long long;
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned large(float v) {
  return (__float_as_uint(v) + 0x1000u) & 0xffffe000u;
}
// two values as pieces: 11 bits rounded, and the rest (of which the tensor cores see 11 bits)
struct Pieces {
  unsigned hi[2], lo[2];
};
__device__ __forceinline__ Pieces split2(f2 v) {
  const float2 w = unpair(v);
  Pieces p;
  p.hi[0] = large(w.x), p.hi[1] = large(w.y);
  const float2 l = unpair(sub2(v, pair(__uint_as_float(p.hi[0]), __uint_as_float(p.hi[1]))));
  p.lo[0] = __float_as_uint(l.x), p.lo[1] = __float_as_uint(l.y);
  return p;
}
__device__ __forceinline__ void mul8(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ void mad8(float (&d)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// sums += a * b for N of b, side by side: each is a chain of three products.  ONE: a has no small piece.
template <bool ONE, int N>
__device__ __forceinline__ void add8(f2 (&sum)[N][2], const unsigned (&hi)[4], const unsigned (&lo)[4], const Pieces (&b)[N]) {
  float d[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (ONE) mul8(d[i], hi, b[i].lo);
    else mul8(d[i], lo, b[i].hi);
  }
  if (!ONE) {
#pragma unroll
    for (int i = 0; i < N; ++i) mad8(d[i], hi, b[i].lo);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) mad8(d[i], hi, b[i].hi);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    sum[i][0] = add2(sum[i][0], pair(d[i][0], d[i][1]));
    sum[i][1] = add2(sum[i][1], pair(d[i][2], d[i][3]));
  }
}

// derivative towards the kernel-space offset (u: !dv, v: dv) from G [cell][8 pixels]
__device__ __forceinline__ float derivative(const float* G, float r_h, float r_w, int fh, int fw, bool dv, const Geom& g) {
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  const float u = ((float)fh + r_h) + uh0, v = ((float)fw + r_w) + uw0;
  if (!(u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW)) return 0.f;
  const float fu = floorf(u), fv = floorf(v);
  // tap + shift is a small multiple of 1/2: u minus it is exact, and so is what the rounding of u lost
  const float lh = (u - fu) + (r_h - (u - ((float)fh + uh0))), lw = (v - fv) + (r_w - (v - ((float)fw + uw0)));
  const int a0 = (int)fu, b0 = (int)fv;
  float c[2][2];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int a = a0 + (k >> 1), b = b0 + (k & 1);
    c[k >> 1][k & 1] = a >= 0 && a < g.scH && b >= 0 && b < g.scW ? G[(a * 4 + b) * 8] : 0.f;
  }
  return dv ? (1.f - lh) * (c[0][1] - c[0][0]) + lh * (c[1][1] - c[1][0]) : (1.f - lw) * (c[1][0] - c[0][0]) + lw * (c[1][1] - c[0][1]);
}

// G of one pixel and tap, cell by cell, where a product that is not finite would have reached the others' pieces (Inf - Inf)
template <typename T>
__device__ __noinline__ void cells_alone(float* G, const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ w, const Geom& g) {
  float sum[16];
  for (int k = 0; k < 16; ++k) sum[k] = 0.f;
  for (int c = 0; c < g.C; ++c) {
    const float dk = ld<float>(dy + (size_t)c * g.P) * ld<float>(x + (size_t)c * g.HW);
    for (int k = 0; k < 16; ++k)
      if ((k >> 2) < g.scH && (k & 3) < g.scW) sum[k] += dk * ld<float>(w + (size_t)c * g.cells + (k >> 2) * g.scW + (k & 3));
  }
  for (int k = 0; k < 16; ++k) G[k * 8] = sum[k];
}

template <typename T, int S>
__global__ void __launch_bounds__(32 * kWarps, 1) tf32_gradients_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                        const T* __restrict__ rot, const T* __restrict__ w,
                                                                        T* __restrict__ drot, float* __restrict__ partial,
                                                                        const __grid_constant__ Geom g, const __grid_constant__ TilePlan t) {
  extern __shared__ __align__(16) unsigned char smem[];
  using R = Room<S>;
  constexpr bool kOnePiece = sizeof(T) == 2, kTwo = R::kBuffers == 2;
  constexpr int NX = (R::X + 31) / 32, NY = (kPixels + 31) / 32;  // words of a lane per channel
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, q = lane & 3;
  float4* beta = reinterpret_cast<float4*>(smem) + warp * 9 * 32 + lane;            // the warp's hat products as mma operands, [tap][lane]
  float* red = reinterpret_cast<float*>(smem + kBetaBytes);                         // [warp][cell][kRedPitch]
  uint4* banks = reinterpret_cast<uint4*>(smem + kBetaBytes + kRedBytes);           // [buffer][step of 8 channels][hi | lo][lane]
  float* stage = reinterpret_cast<float*>(banks + R::kBuffers * kBankBytes / 16);   // [buffer] of x [32][X], dy [32][Y]
  const int px = t.TH * t.TW, chunks = (g.C + 31) / 32;
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  float* mine = partial + (size_t)blockIdx.x * g.C * g.cells;
  const int first = blockIdx.x * t.per_block, last = min(first + t.per_block, t.tiles);
  for (int tile = first; tile < last; ++tile) {
    const TilePos tp = tile_pos(tile, t);
    // offsets of pixel p of the tile in the staged planes, and whether it exists
    auto place = [&](int p, int& xo, int& yo, int& oh, int& ow) {
      const bool in = p < px;
      yo = in ? p : 0;
      const int r = over(yo, t.TW, t.magic_y), col = yo - r * t.TW;
      xo = r * S * t.XW + col * S;
      oh = tp.oh0 + r, ow = tp.ow0 + col;
      return in && oh < g.Ho && ow < g.Wo;
    };
    // the lane's words of the window and of the tile, the same for every channel: element of the plane, -1 outside
    int from_x[NX], from_y[NY];
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int e = lane + 32 * i, r = over(e, t.XW, t.magic_x), ih = tp.oh0 * S - 1 + r, iw = tp.ow0 * S - 1 + (e - r * t.XW);
      from_x[i] = e < t.XH * t.XW && ih >= 0 && ih < g.H && iw >= 0 && iw < g.W ? ih * g.W + iw : -1;
    }
#pragma unroll
    for (int i = 0; i < NY; ++i) {
      const int e = lane + 32 * i, r = over(e, t.TW, t.magic_y), oh = tp.oh0 + r, ow = tp.ow0 + (e - r * t.TW);
      from_y[i] = e < px && oh < g.Ho && ow < g.Wo ? oh * g.Wo + ow : -1;
    }
    auto fill = [&](int chunk) {
      const int c0 = chunk * 32, buffer = kTwo ? chunk & 1 : 0;
      float* xs = stage + buffer * R::kWords + warp * R::X + lane;
      float* ys = stage + buffer * R::kWords + 32 * R::X + warp * R::Y + lane;
      const T* xc = x + ((size_t)tp.n * g.C + c0 + warp) * g.HW;
      const T* yc = dy + ((size_t)tp.n * g.C + c0 + warp) * g.P;
#pragma unroll
      for (int k = 0; k < (32 + kWarps - 1) / kWarps; ++k, xc += kWarps * (size_t)g.HW, yc += kWarps * (size_t)g.P) {
        if (32 % kWarps && warp + kWarps * k >= 32) break;
        const bool has = c0 + warp + kWarps * k < g.C;
        if constexpr (sizeof(T) == 4) {
          const unsigned to_x = (unsigned)__cvta_generic_to_shared(xs + k * kWarps * R::X), to_y = (unsigned)__cvta_generic_to_shared(ys + k * kWarps * R::Y);
#pragma unroll
          for (int i = 0; i < NX; ++i)
            if (lane + 32 * i < R::X) copy4(to_x + 128 * i, xc + max(from_x[i], 0), has && from_x[i] >= 0);
#pragma unroll
          for (int i = 0; i < NY; ++i) copy4(to_y + 128 * i, yc + max(from_y[i], 0), has && from_y[i] >= 0);
        } else {
          float v[NX + NY];
#pragma unroll
          for (int i = 0; i < NX; ++i) v[i] = has && from_x[i] >= 0 ? ld<float>(xc + from_x[i]) : 0.f;
#pragma unroll
          for (int i = 0; i < NY; ++i) v[NX + i] = has && from_y[i] >= 0 ? ld<float>(yc + from_y[i]) : 0.f;
#pragma unroll
          for (int i = 0; i < NX; ++i)
            if (lane + 32 * i < R::X) xs[k * kWarps * R::X + 32 * i] = v[i];
#pragma unroll
          for (int i = 0; i < NY; ++i) ys[k * kWarps * R::Y + 32 * i] = v[NX + i];
        }
      }
      if (warp < 4) {  // the bank of step `warp`: {cell gq, cell gq + 8} of channel 2 q, then of 2 q + 1
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = c0 + warp * 8 + 2 * q + (i >> 1), a = (gq >> 2) + 2 * (i & 1), b = gq & 3;
          v[i] = c < g.C && a < g.scH && b < g.scW ? ld<float>(w + (size_t)c * g.cells + a * g.scW + b) : 0.f;
        }
        const Pieces p0 = split2(pair(v[0], v[1])), p1 = split2(pair(v[2], v[3]));
        uint4* to = banks + (buffer * 4 + warp) * 64 + lane;
        to[0] = make_uint4(p0.hi[0], p0.hi[1], p1.hi[0], p1.hi[1]);
        if (!kOnePiece) to[32] = make_uint4(p0.lo[0], p0.lo[1], p1.lo[0], p1.lo[1]);
      }
    };
    __syncthreads();  // the previous tile's last sums have been read
    fill(0);
    int xg, yg, xk[2], yk[2];
    bool live_k[2];
    {
      int oh, ow;
      place(warp * 8 + gq, xg, yg, oh, ow);
#pragma unroll
      for (int e = 0; e < 2; ++e) {  // k-slots q and q + 4 of the bank's operands: the warp's pixels of these numbers; cells gq and gq + 8
        live_k[e] = place(warp * 8 + q + 4 * e, xk[e], yk[e], oh, ow);
        const T* rp = rot + (size_t)tp.n * 18 * g.P + (live_k[e] ? oh * g.Wo + ow : 0);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
          const float u = live_k[e] ? ((float)(tap / 3) + ld<float>(rp + (size_t)(2 * tap) * g.P)) + uh0 : -8.f;
          const float v = ((float)(tap % 3) + ld<float>(rp + (size_t)(2 * tap + 1) * g.P)) + uw0;
          const float hv = (gq & 3) < g.scW ? hat1(v - (float)(gq & 3)) : 0.f;
          const float h0 = (gq >> 2) < g.scH ? hat1(u - (float)(gq >> 2)) : 0.f, h1 = (gq >> 2) + 2 < g.scH ? hat1(u - (float)((gq >> 2) + 2)) : 0.f;
          reinterpret_cast<float2*>(beta + tap * 32)[e] = make_float2(h0 * hv, h1 * hv);
        }
      }
    }
    f2 G[3][3][2];  // cell gq, then gq + 8, of the warp's pixels 2 q, + 1
#pragma unroll
    for (int i = 0; i < 9; ++i) G[i / 3][i % 3][0] = G[i / 3][i % 3][1] = 0;
    for (int chunk = 0; chunk < chunks; ++chunk) {
      const int c0 = chunk * 32, buffer = kTwo ? chunk & 1 : 0;
      if (!kTwo && chunk > 0) fill(chunk);  // behind the barrier that ended the previous chunk's products
      copies_done();
      __syncthreads();
      if (kTwo && chunk + 1 < chunks) fill(chunk + 1);
      const float* xs = stage + buffer * R::kWords;
      const float* ys = xs + 32 * R::X;
      // offsets: k-slots q and q + 4 are the channels 2 q and 2 q + 1 of a step of 8
      const int steps = min(4, (g.C - c0 + 7) >> 3);
#pragma unroll 1
      for (int ks = 0; ks < steps; ++ks) {
        const uint4* wp = banks + (buffer * 4 + ks) * 64 + lane;
        const uint4 h4 = wp[0], l4 = kOnePiece ? make_uint4(0, 0, 0, 0) : wp[32];
        const unsigned hi[4] = {h4.x, h4.y, h4.z, h4.w}, lo[4] = {l4.x, l4.y, l4.z, l4.w};
        const float* xp = xs + (ks * 8 + 2 * q) * R::X + xg;
        const float* yp = ys + (ks * 8 + 2 * q) * R::Y + yg;
        const f2 d = pair(yp[0], yp[R::Y]);
#pragma unroll
        for (int fh = 0; fh < 3; ++fh, xp += t.XW) {
          Pieces p[3];
#pragma unroll
          for (int fw = 0; fw < 3; ++fw) p[fw] = split2(mul2(d, pair(xp[fw], xp[R::X + fw])));
          add8<kOnePiece, 3>(G[fh], hi, lo, p);
        }
      }
      // bank
      {
        f2 acc[4][2], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[j][0] = acc[j][1] = 0;
          const float* yp = ys + (8 * j + gq) * R::Y;
          d[j] = pair(live_k[0] ? yp[yk[0]] : 0.f, live_k[1] ? yp[yk[1]] : 0.f);
        }
        const float* xa = xs + gq * R::X + xk[0];
        const float* xb = xs + gq * R::X + xk[1];
        const float4* bp = beta;
#pragma unroll 1
        for (int fh = 0; fh < 3; ++fh, xa += t.XW, xb += t.XW)
#pragma unroll
          for (int fw = 0; fw < 3; ++fw, bp += 32) {
            const float4 b = *bp;
            const Pieces p0 = split2(pair(b.x, b.y)), p1 = split2(pair(b.z, b.w));
            const unsigned hi[4] = {p0.hi[0], p0.hi[1], p1.hi[0], p1.hi[1]}, lo[4] = {p0.lo[0], p0.lo[1], p1.lo[0], p1.lo[1]};
            Pieces p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) p[j] = split2(mul2(d[j], pair(xa[8 * j * R::X + fw], xb[8 * j * R::X + fw])));
            add8<false, 4>(acc, hi, lo, p);
          }
        float* r = red + (warp * 16 + gq) * kRedPitch + 2 * q;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          *reinterpret_cast<f2*>(r + 8 * j) = acc[j][0];
          *reinterpret_cast<f2*>(r + 8 * kRedPitch + 8 * j) = acc[j][1];
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = threadIdx.x; i < 512; i += 32 * kWarps) {
        const int cell = i >> 5, a = cell >> 2, b = cell & 3, c = c0 + (i & 31);
        float s = 0.f;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) s += red[(k * 16 + cell) * kRedPitch + (i & 31)];
        float* to = mine + (size_t)c * g.cells + a * g.scW + b;  // this thread's alone: its additions arrive in order
        if (c < g.C && a < g.scH && b < g.scW) {
          if (tile == first) *to = s;
          else atomicAdd(to, s);
        }
      }
    }
    // the derivatives: G through shared memory (the warp's part of `red`), tap by tap
    __syncthreads();
    float* cells = red + warp * 16 * kRedPitch;  // [tap of three][cell][8 pixels]
    const int p = lane & 7, part = lane >> 3;
    int xo, yo, oh, ow;
    const bool live = place(warp * 8 + p, xo, yo, oh, ow);
    const size_t o0 = (size_t)tp.n * 18 * g.P + (live ? oh * g.Wo + ow : 0);
#pragma unroll
    for (int fh = 0; fh < 3; ++fh) {
      __syncwarp();
#pragma unroll
      for (int fw = 0; fw < 3; ++fw) {
        *reinterpret_cast<f2*>(cells + (fw * 16 + gq) * 8 + 2 * q) = G[fh][fw][0];
        *reinterpret_cast<f2*>(cells + (fw * 16 + gq + 8) * 8 + 2 * q) = G[fh][fw][1];
      }
      __syncwarp();
      for (int e = part; e < 6; e += 4) {
        const int fw = e >> 1, tap = fh * 3 + fw;
        const bool dv = e & 1;
        const int ih = oh * S - 1 + fh, iw = ow * S - 1 + fw;
        if (!live) continue;
        float d = 0.f;
        if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W) {
          const float r_h = ld<float>(rot + o0 + (size_t)(2 * tap) * g.P), r_w = ld<float>(rot + o0 + (size_t)(2 * tap + 1) * g.P);
          d = derivative(cells + fw * 128 + p, r_h, r_w, fh, fw, dv, g);
          if (!(fabsf(d) < INFINITY)) {
            float alone[16 * 8];
            cells_alone<T>(alone, dy + (size_t)tp.n * g.C * g.P + oh * g.Wo + ow, x + (size_t)tp.n * g.C * g.HW + ih * g.W + iw, w, g);
            d = derivative(alone, r_h, r_w, fh, fw, dv, g);
          }
        }
        st<T, float>(drot + o0 + (size_t)(2 * tap + dv) * g.P, d);
      }
    }
  }
  bool finite = true;
  __syncthreads();
  for (int i = threadIdx.x; i < g.C * g.cells; i += 32 * kWarps) finite &= fabsf(__ldcg(mine + i)) < INFINITY;
  if (__syncthreads_or(!finite)) {  // one product to the four cells it belongs to, the whole run of the block again
    float* sums = reinterpret_cast<float*>(smem);
    for (int c0 = 0; c0 < g.C; c0 += 32) {
      __syncthreads();
      bank_by_cells<T>(sums, dy, x, nullptr, rot, g, t, c0, warp, kWarps, lane);
      __syncthreads();
      for (int i = threadIdx.x; i < 512; i += 32 * kWarps) {
        const int cell = i >> 5, a = cell >> 2, b = cell & 3, c = c0 + (i & 31);
        if (c >= g.C || a >= g.scH || b >= g.scW) continue;
        float s = 0.f;
        for (int k = 0; k < kWarps; ++k) s += sums[k * 512 + i];
        mine[(size_t)c * g.cells + a * g.scW + b] = s;
      }
    }
  }
}

TilePlan search_plan(const Geom& g) {
  TilePlan t;
  const int most = g.sH == 1 ? Room<1>::X : Room<2>::X;
  long long best = -1;
  for (int wide = 1; wide <= (g.Wo < kPixels ? g.Wo : kPixels); ++wide) {
    for (int high = kPixels / wide < g.Ho ? kPixels / wide : g.Ho; high >= 1; --high) {
      const int across = (g.Wo + wide - 1) / wide, TW = (g.Wo + across - 1) / across, down = (g.Ho + high - 1) / high, TH = (g.Ho + down - 1) / down;
      const int words = ((TH - 1) * g.sH + 3) * ((TW - 1) * g.sW + 3);
      if (words > most) continue;
      // a tile costs its eight warps' steps whatever part of their pixels there is, and a fiftieth of a pixel per staged word
      const long long cost = (long long)across * down * (kPixels * 50 + words + TH * TW);
      if (best < 0 || cost < best) best = cost, t.TW = TW, t.TH = TH, t.across = across, t.down = down;
      break;
    }
  }
  t.tiles = g.N * t.down * t.across;
  t.XH = (t.TH - 1) * g.sH + 3;
  t.XW = (t.TW - 1) * g.sW + 3;
  t.xpitch = most, t.ypitch = Room<1>::Y;
  t.magic_x = (unsigned)((0x100000000ull + t.XW - 1) / t.XW);
  t.magic_y = t.TW == 1 ? 0 : (unsigned)((0x100000000ull + t.TW - 1) / t.TW);
  t.smem = g.sH == 1 ? Room<1>::kBytes : Room<2>::kBytes;
  const int want = 1 * device_sm_count();
  t.per_block = (t.tiles + want - 1) / want;
  t.blocks = (t.tiles + t.per_block - 1) / t.per_block;
  return t;
}

// A call asks for its plan several times (is it taken, scratch, launch); a search takes some microseconds, so a thread keeps its last one.
const TilePlan& gradients_plan(const Geom& g) {
  struct Last {
    int n = 0, h = 0, w = 0, s = 0;
    TilePlan t;
  };
  static thread_local Last last;
  if (last.n != g.N || last.h != g.H || last.w != g.W || last.s != g.sH) last.t = search_plan(g), last.n = g.N, last.h = g.H, last.w = g.W, last.s = g.sH;
  return last.t;
}

}  // namespace

// us, separate kernels (f32_offsets_kernel or local_rot_kernel, f32_bank_kernel) -> this one: fp32 64 x 144 of 56 x 56 758 -> 557, 8 x 64 of
// 28 x 28 (72 tiles) 24 -> 19, 4 x 64 (36 tiles) 17 -> 19, 40 x 40 of 60 x 111 455 -> 289, 128 x 960 of 7 x 7 221 -> 175; stride 2, 40 x 96 of
// 30 x 41 74 -> 51, 16 x 96 of 28 x 28 (48 tiles) 23 -> 27.  fp16 8 x 72 of 75 x 101 165 -> 118, 6 x 104 of 40 x 44 54 -> 34, 24 x 104 of
// 28 x 28 77 -> 62, 64 x 200 of 14 x 14 (1.3 tiles per SM) 90 -> 97, 128 x 200 160 -> 150; stride 2, 40 x 72 of 56 x 50 114 -> 121.
bool local_gradients_tf32_takes(const Geom& g, size_t elem) {
  if (g.kH != 3 || g.kW != 3 || g.dH != 1 || g.dW != 1 || g.pH != 1 || g.pW != 1 || g.sH != g.sW || (g.sH != 1 && g.sH != 2)) return false;
  if (g.G != 1 || g.scH > 4 || g.scW > 4 || (long long)g.N * g.P >= 0x3fffffff) return false;
  if ((long long)g.N * g.P < 1536) return false;  // few tiles whatever their shape
  const int tiles = gradients_plan(g).tiles, sms = device_sm_count();
  return tiles >= 64 && (elem == 4 || (g.sH == 1 && (tiles <= sms || 2 * tiles >= 3 * sms)));
}
size_t local_gradients_tf32_workspace(const Geom& g, size_t elem) {
  return local_gradients_tf32_takes(g, elem) ? (size_t)gradients_plan(g).blocks * g.C * g.cells * sizeof(float) : 0;
}
template <typename T>
int local_gradients_tf32(const T* dy, const T* x, const T* rot, const T* w, T* drot, T* dw, const Geom& g, void* ws, size_t ws_bytes,
                         cudaStream_t s) {
  if (!local_gradients_tf32_takes(g, sizeof(T))) return DK_ERR_UNSUPPORTED;
  const TilePlan& t = gradients_plan(g);
  if (t.smem > (size_t)device_smem_optin() || ws == nullptr || ws_bytes < (size_t)t.blocks * g.C * g.cells * sizeof(float)) return DK_ERR_UNSUPPORTED;
  auto kern = g.sH == 1 ? tf32_gradients_kernel<T, 1> : tf32_gradients_kernel<T, 2>;
  if (int rc = enable_smem(kern, t.smem)) return rc;
  float* partial = reinterpret_cast<float*>(ws);
  kern<<<t.blocks, 32 * kWarps, t.smem, s>>>(dy, x, rot, w, drot, partial, g, t);
  if (int rc = check_launch()) return rc;
  return reduce_bank<T>(partial, dw, g.C * g.cells, t.blocks, s);
}
template int local_gradients_tf32<float>(const float*, const float*, const float*, const float*, float*, float*, const Geom&, void*, size_t,
                                         cudaStream_t);
template int local_gradients_tf32<__half>(const __half*, const __half*, const __half*, const __half*, __half*, __half*, const Geom&, void*,
                                          size_t, cudaStream_t);

}  // namespace dk
