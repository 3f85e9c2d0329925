// Offset and bank gradients of the local deformable kernel in one pass, fp32 arithmetic on the tensor cores (fp32 tensors, and fp16 where
// the fp16 kernels do not apply; 3 x 3 taps, scopes up to 4 x 4).
//
// Both are contractions of dK = dy * x with 16 cells: G[pixel, tap][cell] = sum_c dK W[c, cell] (then the floor-based derivative
// weights) and dW[c][cell] = sum over pixels and taps of dK beta[(pixel, tap), cell].  An fp32 value is three bf16 pieces, 8 bits rounded each time,
// which together are all of it (down to 2^-110, below which the last ones underflow); a product is six of their products, the smallest first,
// and what is left out is 2^-23 of it at the most, 2^-26 in the mean (a rounding: 2^-24 and 2^-25.8).  The tensor cores truncate their
// sums, so no accumulator runs longer than these six: a step of 16 channels (G) or of 8 pixels at two taps (dW) is added to the sums with
// one rounded addition.  Against fp64, separate fp32 kernels -> this one, 2-norm: 16 x 16 of 61 x 63 at stride 2 offsets 7.5e-8 -> 6.9e-8,
// bank 1.9e-7 -> 1.7e-7 (most of it the rounding of the coordinates), 64 x 144 of 56 x 56 1.4e-7 -> 0.9e-7 and 5.2e-7 -> 2.0e-7.
//
// Block: a tile of up to 96 pixels, a warp 8 of them, over all channels, 32 at a time, whose dy and x are staged while the previous ones are
// multiplied.  G stays in registers (9 taps x 16 cells x 8 pixels per warp); the warps' bank sums of 32 channels meet in
// shared memory, in their order, and are added to the block's partial sums.  dK is split once: movmatrix turns the pieces from the lanes'
// order of the offsets (k = channels) to that of the bank (k = pixels).  Pairs of steps and pairs of taps fill the 16 k-slots so that every operand lies
// in registers as it was loaded or made; two pieces of one step beside each other need copies of one of them and take 629 us below.  A step left
// over takes them that way for the offsets (64 x 24 of 112 x 110: 674 us beside a step of zeros, 617 so, 637 in separate kernels).
//
// fp32 64 x 144 of 56 x 56: 753 us in two kernels that gather or hold the cells with one fp32 multiply-add each -> 558.  Tensor pipe 40 %,
// issue 37 %: products, the pieces that feed them and the additions behind them follow each other in a warp, and 3 warps per scheduler (168 registers)
// overlap part of it; tiles that do not fill and the tenth tap of the pairs are 15 % of the products.
#include <type_traits>

#include "dk_f32_tiles.cuh"

namespace dk {

namespace {

constexpr int kWarps = 12, kPixels = 8 * kWarps, kRedPitch = 40;
constexpr int kBetaBytes = kWarps * 5 * 3 * 32 * 16, kRedBytes = kWarps * 16 * kRedPitch * 4, kBankBytes = 2 * 3 * 32 * 16;
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
// Two values as three pieces of bf16, 8 bits rounded and the rest: together they are the values, all 24 bits.  Low half: the first value.
struct Pieces {
  unsigned p[3];
};
__device__ __forceinline__ unsigned two_bf16(f2 v) {
  const float2 w = unpair(v);
  unsigned r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(w.y), "f"(w.x));
  return r;
}
__device__ __forceinline__ f2 widened(unsigned p) { return pair(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)); }
__device__ __forceinline__ Pieces split3(f2 v) {
  Pieces s;
  s.p[0] = two_bf16(v);
  v = sub2(v, widened(s.p[0]));
  s.p[1] = two_bf16(v);
  s.p[2] = two_bf16(sub2(v, widened(s.p[1])));
  return s;
}
__device__ __forceinline__ unsigned turned(unsigned v) {
  unsigned r;
  asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;\n" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ void mul16(float (&d)[4], const uint4& a, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mad16(float (&d)[4], const uint4& a, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// Product E of the six of two operands in pieces.  a: [piece], b and c: the pieces of the k-slots 0-7 and 8-15.
template <int E>
__device__ __forceinline__ void product(float (&d)[4], const uint4 (&a)[3], const Pieces& b, const Pieces& c) {
  constexpr int A = E == 0 || E > 3 ? 0 : E == 1 ? 2 : 1, B = E == 0 ? 2 : E == 2 || E == 4 ? 1 : 0;
  if (E == 0) mul16(d, a[A], b.p[B], c.p[B]);
  else mad16(d, a[A], b.p[B], c.p[B]);
}
// The same in three products of two pieces each.  a: {third | first}, {second | second}, {first | first} from a[2] on down.
template <int E>
__device__ __forceinline__ void beside(float (&d)[4], const uint4 (&a)[3], const Pieces& b) {
  if (E == 0) mul16(d, a[2], b.p[0], b.p[2]);
  else mad16(d, a[2 - E], b.p[0], b.p[1]);
}
__device__ __forceinline__ void add4(f2 (&s)[2], const float (&d)[4]) {
  s[0] = add2(s[0], pair(d[0], d[1]));
  s[1] = add2(s[1], pair(d[2], d[3]));
}

// where a sample falls in the bank: upper left cell (-1 .. last) and the fractions
struct Cells {
  int a, b;
  float lh, lw;
};
__device__ __forceinline__ bool cells_at(Cells& q, float r_h, float r_w, int fh, int fw, const Geom& g) {
  const float uh0 = 0.5f * (float)(g.scH - 3), uw0 = 0.5f * (float)(g.scW - 3);
  const float u = ((float)fh + r_h) + uh0, v = ((float)fw + r_w) + uw0;
  if (!(u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW)) return false;
  const float fu = floorf(u), fv = floorf(v);
  // tap + shift is a small multiple of 1/2: u minus it is exact, and so is what the rounding of u lost
  q.lh = (u - fu) + (r_h - (u - ((float)fh + uh0))), q.lw = (v - fv) + (r_w - (v - ((float)fw + uw0)));
  q.a = (int)fu, q.b = (int)fv;
  return true;
}
__device__ __forceinline__ bool cell_in(const Cells& q, int k, const Geom& g) {  // k-th of the four
  return (unsigned)(q.a + (k >> 1)) < (unsigned)g.scH && (unsigned)(q.b + (k & 1)) < (unsigned)g.scW;
}
// derivatives towards the kernel-space offset from G of the four cells
__device__ __forceinline__ float2 derivatives(const Cells& q, const float (&c)[4]) {
  return make_float2((1.f - q.lw) * (c[2] - c[0]) + q.lw * (c[3] - c[1]), (1.f - q.lh) * (c[1] - c[0]) + q.lh * (c[3] - c[2]));
}

// The derivatives of one pixel and tap where G [cell][8 pixels] is not finite in a cell of theirs: the pieces of an infinite product are infinite and NaN.
// Its four cells again, a multiply-add each.  Where other cells are finite every dK is, and only the bank's values that are not (or round to
// infinity) count; else all channels do, until a NaN settles both derivatives.  64 x 144 of 56 x 56, offsets and bank, us, with all sixteen cells for
// either derivative -> so: every dy NaN 36144 -> 1278, one infinite bank value 29929 -> 1725 (in
// separate kernels 4326 and 767).
template <typename T>
__device__ __noinline__ float2 cells_alone(const Cells& q, const float* G, const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ w,
                                           const Geom& g) {
  constexpr float kRounds = 3.3961e38f;  // bf16 values end at 2^128 (1 - 2^-8), those from 2^128 (1 - 2^-9) on round to infinity
  float sum[4];
  bool bad[4], by_bank = false;
#pragma unroll
  for (int k = 0; k < 16; ++k) by_bank |= fabsf(G[k * 8]) < INFINITY;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool in = cell_in(q, k, g);
    sum[k] = in ? G[((q.a + (k >> 1)) * 4 + q.b + (k & 1)) * 8] : 0.f;
    bad[k] = !(fabsf(sum[k]) < INFINITY);
  }
  const T* wk = w + q.a * g.scW + q.b;
  if (by_bank) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (!bad[k]) continue;
      sum[k] = 0.f;
      for (int c0 = 0; c0 < g.C; c0 += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = ld<float>(wk + (size_t)min(c0 + i, g.C - 1) * g.cells + (k >> 1) * g.scW + (k & 1));
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (c0 + i < g.C && !(fabsf(v[i]) < kRounds)) sum[k] += ld<float>(dy + (size_t)(c0 + i) * g.P) * ld<float>(x + (size_t)(c0 + i) * g.HW) * v[i];
      }
      by_bank &= !(fabsf(sum[k]) < INFINITY);
    }
    if (by_bank) return derivatives(q, sum);
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) sum[k] = 0.f;
  for (int c0 = 0; c0 < g.C; c0 += 4) {
    float dk[4], b[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = min(c0 + i, g.C - 1);
      dk[i] = ld<float>(dy + (size_t)c * g.P) * ld<float>(x + (size_t)c * g.HW);
#pragma unroll
      for (int k = 0; k < 4; ++k) b[i][k] = cell_in(q, k, g) ? ld<float>(wk + (size_t)c * g.cells + (k >> 1) * g.scW + (k & 1)) : 0.f;
    }
    bool settled = false;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (c0 + i < g.C && cell_in(q, k, g)) sum[k] += dk[i] * b[i][k];
        settled |= sum[k] != sum[k];
      }
    if (settled) break;
  }
  return derivatives(q, sum);
}

template <typename T, int S>
__global__ void __launch_bounds__(32 * kWarps, 1) pieces_gradients_kernel(const T* __restrict__ dy, const T* __restrict__ x,
                                                                        const T* __restrict__ rot, const T* __restrict__ w,
                                                                        T* __restrict__ drot, float* __restrict__ partial,
                                                                        const __grid_constant__ Geom g, const __grid_constant__ TilePlan t) {
  extern __shared__ __align__(16) unsigned char smem[];
  using R = Room<S>;
  constexpr bool kTwo = R::kBuffers == 2;
  constexpr int NX = (R::X + 31) / 32, NY = (kPixels + 31) / 32;  // words of a lane per channel
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, q = lane & 3;
  uint4* beta = reinterpret_cast<uint4*>(smem) + warp * 15 * 32 + lane;             // the warp's hat products as mma operands, [taps 2 i, + 1][piece][lane]
  float* red = reinterpret_cast<float*>(smem + kBetaBytes);                         // [warp][cell][kRedPitch]
  uint4* banks = reinterpret_cast<uint4*>(smem + kBetaBytes + kRedBytes) + lane;    // [buffer][steps 2 i, + 1 of 8 channels][piece][lane]
  float* stage = reinterpret_cast<float*>(smem + kBetaBytes + kRedBytes + R::kBuffers * kBankBytes);  // [buffer] of x [32][X], dy [32][Y]
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
    // half `h` (eight k-slots) of an operand in pieces: rows gq and gq + 8
    auto put = [](uint4* to, int h, const Pieces& r0, const Pieces& r1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) reinterpret_cast<uint2*>(to + 32 * k)[h] = make_uint2(r0.p[k], r1.p[k]);
    };
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
      if (warp < 4) {  // the bank of step `warp`: channels 2 q, + 1 of cell gq, then of gq + 8
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int c = c0 + warp * 8 + 2 * q + (i & 1), a = (gq >> 2) + 2 * (i >> 1), b = gq & 3;
          v[i] = c < g.C && a < g.scH && b < g.scW ? ld<float>(w + (size_t)c * g.cells + a * g.scW + b) : 0.f;
        }
        put(banks + (buffer * 2 + (warp >> 1)) * 96, warp & 1, split3(pair(v[0], v[1])), split3(pair(v[2], v[3])));
      }
    };
    __syncthreads();  // the previous tile's last sums have been read
    fill(0);
    int xg, yg;
    bool live_g;
    {
      int oh, ow, xk, yk;
      live_g = place(warp * 8 + gq, xg, yg, oh, ow);
      bool live_k[2];
      const T* rp[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        live_k[e] = place(warp * 8 + 2 * q + e, xk, yk, oh, ow);
        rp[e] = rot + (size_t)tp.n * 18 * g.P + (live_k[e] ? oh * g.Wo + ow : 0);
      }
#pragma unroll
      for (int tap = 0; tap < 9; ++tap) {
        float b[2][2];  // cells gq and gq + 8, pixels 2 q and 2 q + 1
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float u = live_k[e] ? ((float)(tap / 3) + ld<float>(rp[e] + (size_t)(2 * tap) * g.P)) + uh0 : -8.f;
          const float v = ((float)(tap % 3) + ld<float>(rp[e] + (size_t)(2 * tap + 1) * g.P)) + uw0;
          const float hv = (gq & 3) < g.scW ? hat1(v - (float)(gq & 3)) : 0.f;
          b[0][e] = (gq >> 2) < g.scH ? hat1(u - (float)(gq >> 2)) * hv : 0.f;
          b[1][e] = (gq >> 2) + 2 < g.scH ? hat1(u - (float)((gq >> 2) + 2)) * hv : 0.f;
        }
        put(beta + (tap >> 1) * 96, tap & 1, split3(pair(b[0][0], b[0][1])), split3(pair(b[1][0], b[1][1])));
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
      // Two taps and two steps at a time: 16 k-slots are the channels of both steps (offsets), or the warp's pixels at both taps (bank).  The
      // products of a tap and a step are split once, in the lanes as the offsets want them, and movmatrix turns the pieces for the bank.
      // A step that is left over by itself has two pieces beside each other in the products of the offsets.
      const int steps = min(4, (g.C - c0 + 7) >> 3);
      float* r = red + (warp * 16 + gq) * kRedPitch + 2 * q;
      const uint4* wq = banks + buffer * 6 * 32;
      const float* yq = ys + 2 * q * R::Y + yg;
      const float* xq = xs + 2 * q * R::X + xg;
      auto pass = [&](auto pair_of_steps) {
        constexpr int N = decltype(pair_of_steps)::value ? 2 : 1;
        f2 acc[N][2], d[N];
        uint4 wp[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) wp[k] = wq[32 * k];
        if (N == 1) {
          const uint2 w0 = make_uint2(wp[0].x, wp[0].y), w1 = make_uint2(wp[1].x, wp[1].y);
          wp[2] = make_uint4(wp[2].x, wp[2].y, w0.x, w0.y), wp[1] = make_uint4(w1.x, w1.y, w1.x, w1.y), wp[0] = make_uint4(w0.x, w0.y, w0.x, w0.y);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
          const float* yp = yq + j * 8 * R::Y;
          d[j] = live_g ? pair(yp[0], yp[R::Y]) : 0;
          acc[j][0] = acc[j][1] = 0;
        }
#pragma unroll
        for (int t0 = 0; t0 < 9; t0 += 2) {
          uint4 bp[3];
#pragma unroll
          for (int k = 0; k < 3; ++k) bp[k] = beta[(t0 >> 1) * 96 + 32 * k];
          Pieces p[2][N], pt[2][N];  // [tap][step]
          float u[2][4], v[N][4];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int tap = t0 + i;
            if (tap > 8) break;
            const float* at = xq + (tap / 3) * t.XW + tap % 3;
#pragma unroll
            for (int j = 0; j < N; ++j) p[i][j] = split3(mul2(d[j], pair(at[j * 8 * R::X], at[j * 8 * R::X + R::X])));
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < N; ++j)
#pragma unroll
              for (int k = 0; k < 3; ++k) pt[i][j].p[k] = t0 + i < 9 ? turned(p[i][j].p[k]) : 0u;
          if (t0 == 8) bp[0].z = bp[0].w = bp[1].z = bp[1].w = bp[2].z = bp[2].w = 0u;
#define DK_PRODUCT(E)                                                                    \
  if (N == 2 && (E != 1 || sizeof(T) == 4)) { /* fp16 banks are two pieces */            \
    product<E>(u[0], wp, p[0][0], p[0][N - 1]);                                          \
    if (t0 < 8) product<E>(u[1], wp, p[1][0], p[1][N - 1]);                              \
  }                                                                                      \
  if (N == 1 && E < 3)                                                                   \
    for (int i = 0; i < (t0 < 8 ? 2 : 1); ++i) beside<E>(u[i], wp, p[i][0]);             \
  for (int j = 0; j < N; ++j) product<E>(v[j], bp, pt[0][j], pt[1][j]);
          DK_PRODUCT(0) DK_PRODUCT(1) DK_PRODUCT(2) DK_PRODUCT(3) DK_PRODUCT(4) DK_PRODUCT(5)
#undef DK_PRODUCT
          add4(G[t0 / 3][t0 % 3], u[0]);
          if (t0 < 8) add4(G[(t0 + 1) / 3 % 3][(t0 + 1) % 3], u[1]);
#pragma unroll
          for (int j = 0; j < N; ++j) add4(acc[j], v[j]);
        }
#pragma unroll
        for (int j = 0; j < N; ++j) {
          *reinterpret_cast<f2*>(r + 8 * j) = acc[j][0];
          *reinterpret_cast<f2*>(r + 8 * kRedPitch + 8 * j) = acc[j][1];
        }
      };
#pragma unroll 1
      for (int h = 1; h < steps; h += 2, r += 16, wq += 96, yq += 16 * R::Y, xq += 16 * R::X) pass(std::true_type());
      if (steps & 1) pass(std::false_type());
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
      if (part < 3 && live) {
        const int fw = part, tap = fh * 3 + fw, ih = oh * S - 1 + fh, iw = ow * S - 1 + fw;
        const size_t o = o0 + (size_t)(2 * tap) * g.P;
        float2 d = make_float2(0.f, 0.f);
        Cells at;
        if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W && cells_at(at, ld<float>(rot + o), ld<float>(rot + o + g.P), fh, fw, g)) {
          const float* G4 = cells + fw * 128 + p;
          float c[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) c[k] = cell_in(at, k, g) ? G4[((at.a + (k >> 1)) * 4 + at.b + (k & 1)) * 8] : 0.f;
          d = derivatives(at, c);
          if (!(fabsf(d.x) < INFINITY && fabsf(d.y) < INFINITY))
            d = cells_alone<T>(at, G4, dy + (size_t)tp.n * g.C * g.P + oh * g.Wo + ow, x + (size_t)tp.n * g.C * g.HW + ih * g.W + iw, w, g);
        }
        st<T, float>(drot + o, d.x);
        st<T, float>(drot + o + g.P, d.y);
      }
    }
  }
  // one product to the four cells it belongs to, the whole run of the block again, for 32 channels with a sum that is not finite
  float* sums = reinterpret_cast<float*>(smem);
  for (int c0 = 0; c0 < g.C; c0 += 32) {
    bool finite = true;
    __syncthreads();
    for (int i = threadIdx.x; i < min(32, g.C - c0) * g.cells; i += 32 * kWarps) finite &= fabsf(__ldcg(mine + c0 * g.cells + i)) < INFINITY;
    if (!__syncthreads_or(!finite)) continue;
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

TilePlan search_plan(const Geom& g, int sms) {
  TilePlan t;
  const int most = g.sH == 1 ? Room<1>::X : Room<2>::X;
  long long best = -1;
  for (int wide = 1; wide <= (g.Wo < kPixels ? g.Wo : kPixels); ++wide) {
    for (int high = kPixels / wide < g.Ho ? kPixels / wide : g.Ho; high >= 1; --high) {
      const int across = (g.Wo + wide - 1) / wide, TW = (g.Wo + across - 1) / across, down = (g.Ho + high - 1) / high, TH = (g.Ho + down - 1) / down;
      const int words = ((TH - 1) * g.sH + 3) * ((TW - 1) * g.sW + 3);
      if (words > most) continue;
      // a tile costs its twelve warps' steps whatever part of their pixels there is, and a fiftieth of a pixel per staged word
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
  t.per_block = (t.tiles + sms - 1) / sms;
  t.blocks = (t.tiles + t.per_block - 1) / t.per_block;
  return t;
}

// A call asks for its plan several times (is it taken, scratch, launch); a search takes some microseconds, so a thread keeps its last one.
const TilePlan& gradients_plan(const Geom& g) {
  struct Last {
    int n = 0, h = 0, w = 0, s = 0, sms = 0;
    TilePlan t;
  };
  static thread_local Last last;
  const int sms = device_sm_count();  // of the thread's current device
  if (last.n != g.N || last.h != g.H || last.w != g.W || last.s != g.sH || last.sms != sms)
    last.t = search_plan(g, sms), last.n = g.N, last.h = g.H, last.w = g.W, last.s = g.sH, last.sms = sms;
  return last.t;
}

}  // namespace

// A block's tiles take the time of their twelve warps whatever part of them is pixels, so planes that leave tiles half empty (4 x 4 outputs: 16
// of 96 pixels) and one tile too many for a round make this kernel the slower one.  Both sides are estimated in us, from 2000 measured calls of
// 16 to 968 channels, planes of 7 x 7 to 56 x 56, 1536 to 70 k pixels, inputs in L2 and not: this one within 4 to 8 %, the separate kernels
// (f32_offsets_kernel or local_rot_kernel, f32_bank_kernel) within 5 to 13 %; of the faster choice 0.5 % are lost in the mean, a quarter at most.  us,
// separate -> this one, taken: fp32 64 x 144 of 56 x 56 758 -> 557, 8 x 64 of 28 x 28 (72 tiles) 24 -> 19, 40 x 40 of 60 x 111 455 -> 289, 128 x 960
// of 7 x 7 217 -> 172; stride 2, 40 x 96 of 30 x 41 74 -> 51.  fp16 8 x 72 of 75 x 101 165 -> 118, 6 x 104 of 40 x 44 54 -> 34, 24 x 104 of 28 x 28
// 77 -> 62.  Not taken: fp32 4 x 64 of 28 x 28 (36 tiles) 17 -> 19; stride 2, 16 x 96 of 28 x 28 (48 tiles) 23 -> 27, 128 x 960 of 7 x 7
// 132 -> 195, 388 x 192 of 7 x 7 55 -> 127, 317 x 192 of 9 x 12 71 -> 130; fp16 64 x 200 of 14 x 14 (1.3 tiles per SM) 90 -> 97, 153 x 584 of 9 x 12
// 267 -> 350; stride 2, 40 x 72 of 56 x 50 114 -> 121.
bool local_gradients_pieces_takes(const Geom& g, size_t elem) {
  if (g.kH != 3 || g.kW != 3 || g.dH != 1 || g.dW != 1 || g.pH != 1 || g.pW != 1 || g.sH != g.sW || (g.sH != 1 && g.sH != 2)) return false;
  if (g.G != 1 || g.scH > 4 || g.scW > 4 || (long long)g.N * g.P >= 0x3fffffff) return false;
  if ((long long)g.N * g.P < 1536) return false;  // few tiles whatever their shape
  const TilePlan& t = gradients_plan(g);
  const int sms = device_sm_count();
  if (t.tiles < 64 || (elem == 2 && (g.sH == 2 || (t.tiles > sms && 2 * t.tiles < 3 * sms)))) return false;
  const double steps = (g.C + 7) / 8, thousands = (double)g.N * g.P / 1000 * 148 / sms;
  const double here = 4.6 + t.per_block * (3.6 + (elem == 2 ? 1.95 : g.sH == 1 ? 1.5 : 1.7) * steps);
  const double separate = 14 + 0.08 * g.C + thousands * (0.5 + (elem == 2 ? 0.19 : g.sH == 1 ? 0.195 : 0.22) * steps);
  return here < separate;
}
size_t local_gradients_pieces_workspace(const Geom& g, size_t elem) {
  return local_gradients_pieces_takes(g, elem) ? (size_t)gradients_plan(g).blocks * g.C * g.cells * sizeof(float) : 0;
}
template <typename T>
int local_gradients_pieces(const T* dy, const T* x, const T* rot, const T* w, T* drot, T* dw, const Geom& g, void* ws, size_t ws_bytes,
                         cudaStream_t s) {
  if (!local_gradients_pieces_takes(g, sizeof(T))) return DK_ERR_UNSUPPORTED;
  const TilePlan& t = gradients_plan(g);
  if (t.smem > (size_t)device_smem_optin() || ws == nullptr || ws_bytes < (size_t)t.blocks * g.C * g.cells * sizeof(float)) return DK_ERR_UNSUPPORTED;
  auto kern = g.sH == 1 ? pieces_gradients_kernel<T, 1> : pieces_gradients_kernel<T, 2>;
  if (int rc = enable_smem(kern, t.smem)) return rc;
  float* partial = reinterpret_cast<float*>(ws);
  kern<<<t.blocks, 32 * kWarps, t.smem, s>>>(dy, x, rot, w, drot, partial, g, t);
  if (int rc = check_launch()) return rc;
  return reduce_bank<T>(partial, dw, g.C * g.cells, t.blocks, s);
}
template int local_gradients_pieces<float>(const float*, const float*, const float*, const float*, float*, float*, const Geom&, void*, size_t,
                                         cudaStream_t);
template int local_gradients_pieces<__half>(const __half*, const __half*, const __half*, const __half*, __half*, __half*, const Geom&, void*,
                                          size_t, cudaStream_t);

}  // namespace dk
