// fp16 DK + DCN with the operands in channel order: forward, both offset gradients with the bank gradient, grad-input.
//
// Where a sample lands depends on (pixel, tap) and not on the channel, so x and dy are first brought into lines, [unit of 64
// channels][pixel][64] (lines_kernel), and what a sample needs besides (line of its upper left corner, corner coefficients, hat
// products of the bank) is worked out once in shared memory for all channels.  The kernels with whole planes on chip
// (dk_deform_mma.cu) build it again for every 16 channels.
//
// A load of 16 bytes per lane is served eight lanes at a time, 4.2 cycles of the load pipe if those read one line, 8.0 if
// they read the same 64 bytes of two.  So eight lanes read the 64 channels of one pixel: lane = 4 g + t has the channels
// 32 (g & 1) + 8 t .. + 7 of the pixels 4 (g >> 1) + i, i = 0 .. 3, of a group of 16.  The products with the hat functions come
// out of mma.sync in that layout: the rows 2 q and 2 q + 1 are the same pixel, the even rows count for the lower 32 channels and the odd
// rows for the upper ones (two mma, one with the bank of each half, and a lane keeps the result of its rows: zeroed rows instead would let a
// bank value that is not finite reach the channel 32 away), and the columns 2 t, 2 t + 1 of tile j are the channels 8 t + 2 j, + 1.  mma.sync,
// because its results are needed in registers beside the gathered values.
//
// 64 x 256 of 56 x 56, forward and backward 3384 -> 1324 us: lines 35 and 65, forward 300, sort 56, gather 290, offsets and bank
// 573.  Forward: load pipe 69 % (64 of its 109 passes per 16 pixels, tap and 64 channels are the corners, 44 % of the
// rest misses and offsets), 2.8 warps per scheduler at 168 registers; 8 loads in flight instead of 16 with 16 warps instead of
// 12 takes as long.  Offsets and bank: load pipe 46 %, tensor pipe 33 %, issue 44 %, the half-rate fp16 pipe with 14 instructions where the tensor
// pipe has 10: latency at twelve warps of an SM in three blocks, which the 64 registers of bank sums and bank operands leave.  Gather: load pipe
// 60 %, tensor 37 %, issue 52 %.
#include <cooperative_groups.h>

#include "dk_mma_common.cuh"

namespace dk {

using namespace mma;

namespace {

namespace cg = cooperative_groups;

constexpr int kLineTaps = 9;
constexpr int kStrip = 16;       // pixels are taken in strips of 16 columns: 64 of them are 16 x 4
constexpr int kSortBlocks = 8, kSortThreads = 512;
constexpr int kChunk = 96;       // samples of the gather between two barriers

// division of numbers below 2^31 by a constant: ceil(2^(31 + l) / d) with 2^l >= d
struct Div {
  unsigned m, s, d;
};
Div make_div(unsigned d) {
  unsigned l = 0;
  while ((1u << l) < d) ++l;
  if (l == 0) return {0u, 0u, 1u};
  return {(unsigned)(((1ull << (31 + l)) + d - 1) / d), l - 1, d};
}
__device__ __forceinline__ int operator/(int n, const Div& v) { return v.m ? (int)(__umulhi((unsigned)n, v.m) >> v.s) : n; }

struct LineGeom {
  Geom g;
  Div P, strip, last, Wo, W;  // pixels of a sample, of a strip, columns of the last strip, of a row of y and of x
  int units, xs;           // of 64 channels; lines of x of a sample: (H + 2) (W + 2), its border of zeros included
  size_t xu, yu;           // bytes of a unit of x and of dy
};
constexpr unsigned kLine = 128;  // bytes

// ------------------------------------------------------------------ lines
// x: a border of zeros around every sample and a row of zeros at the end, so that the four corners of any sample point are
// the line of its upper left corner and fixed distances from it; a sample that is not used takes the two rows of zeros from its
// image's lower border on.  dy: a line of zeros at the end.
struct LineJob {
  const __half* src;
  __half* dst;
  int P, vec;
};

// Block (tile of 64 pixels, unit of x or dy or the zeros, sample); a word in shared memory = two neighbouring channels of a pixel.
__global__ void __launch_bounds__(256) lines_kernel(const LineJob jx, const LineJob jy, const __grid_constant__ LineGeom lg) {
  __shared__ __align__(16) unsigned tile[64 * 32];
  const Geom& g = lg.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n = blockIdx.z;
  const uint4 z = make_uint4(0, 0, 0, 0);
  int ct = blockIdx.y;
  bool is_x = jx.src != nullptr;
  if (is_x && ct >= lg.units) is_x = false, ct -= lg.units;
  if (!is_x && (jy.src == nullptr || ct >= lg.units)) {  // the zeros
    const int rows = 2 * (g.W + 2) + 2 * g.H + (n == g.N - 1 ? g.W + 2 : 0), at0 = blockIdx.x * 256 + tid, step = gridDim.x * 256;
    if (jx.src)
      for (int i = at0; i < lg.units * rows * 8; i += step) {
        const int u = i / (rows * 8), r8 = i - u * rows * 8;
        int l = r8 >> 3;
        if (l >= 2 * (g.W + 2) + 2 * g.H) {
          l = lg.xs + l - 2 * (g.W + 2) - 2 * g.H;
        } else if (l >= g.W + 2) {
          l -= g.W + 2;
          const int r = l - (g.W + 2);
          l = r < 0 ? (g.H + 1) * (g.W + 2) + l : ((r >> 1) + 1) * (g.W + 2) + (r & 1 ? g.W + 1 : 0);
        }
        reinterpret_cast<uint4*>(reinterpret_cast<char*>(jx.dst) + u * lg.xu)[((size_t)n * lg.xs + l) * 8 + (r8 & 7)] = z;
      }
    if (n == 0 && jy.src)
      for (int i = at0; i < lg.units * 8; i += step)
        reinterpret_cast<uint4*>(reinterpret_cast<char*>(jy.dst) + (i >> 3) * lg.yu)[(size_t)g.N * g.P * 8 + (i & 7)] = z;
    return;
  }
  const LineJob j = {is_x ? jx.src : jy.src, is_x ? jx.dst : jy.dst, is_x ? jx.P : jy.P, is_x ? jx.vec : jy.vec};
  const int p0 = blockIdx.x * 64;
  if (p0 >= j.P) return;
  const __half* src = j.src + ((size_t)n * g.C + ct * 64) * j.P;
  auto at = [&](int px, int cp) { return px * 32 + (((cp >> 2) ^ (px >> 3)) << 2) + (cp & 3); };
  if (j.vec) {
    const int pg = lane & 7, cp = warp * 4 + (lane >> 3);
    uint4 a = z, c = z;
    if (p0 + pg * 8 < j.P && ct * 64 + 2 * cp < g.C) {
      const __half* s = src + (size_t)(2 * cp) * j.P + p0 + pg * 8;
      a = __ldg(reinterpret_cast<const uint4*>(s));
      c = __ldg(reinterpret_cast<const uint4*>(s + j.P));
    }
    const unsigned aw[4] = {a.x, a.y, a.z, a.w}, cw[4] = {c.x, c.y, c.z, c.w};
    unsigned* to = tile + at(pg * 8, cp);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      to[64 * k] = __byte_perm(aw[k], cw[k], 0x5410);
      to[64 * k + 32] = __byte_perm(aw[k], cw[k], 0x7632);
    }
  } else {
    unsigned short v[4][2][2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cp = warp * 4 + k, p = p0 + 32 * h + lane;
        const bool in = p < j.P && ct * 64 + 2 * cp < g.C;
        const __half* s = src + (size_t)(2 * cp) * j.P + p;
        v[k][h][0] = in ? __half_as_ushort(__ldg(s)) : 0;
        v[k][h][1] = in ? __half_as_ushort(__ldg(s + j.P)) : 0;
      }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int h = 0; h < 2; ++h) tile[at(32 * h + lane, warp * 4 + k)] = v[k][h][0] | ((unsigned)v[k][h][1] << 16);
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int px = (tid >> 3) + 32 * k, o = tid & 7, p = p0 + px;
    if (p < j.P) {
      const uint4 v = *reinterpret_cast<const uint4*>(tile + at(px, o * 4));
      size_t line = (size_t)n * g.P + p;
      if (is_x) {
        const int h = p / lg.W;
        line = (size_t)n * lg.xs + (h + 1) * (g.W + 2) + p - h * g.W + 1;
      }
      reinterpret_cast<uint4*>(reinterpret_cast<char*>(j.dst) + ct * (is_x ? lg.xu : lg.yu))[line * 8 + o] = v;
    }
  }
}

// ------------------------------------------------------------------ samples
// pixel f of the call in the order of the strips
__device__ __forceinline__ void strip_pixel(int f, const LineGeom& lg, int& n, int& oh, int& ow) {
  n = f / lg.P;
  int r = f - n * lg.g.P;
  const int s = r / lg.strip;
  r -= s * kStrip * lg.g.Ho;
  if (lg.g.Wo - s * kStrip >= kStrip) {
    oh = r / kStrip;
    ow = s * kStrip + (r & (kStrip - 1));
  } else {
    oh = r / lg.last;
    ow = s * kStrip + r - oh * (int)lg.last.d;
  }
}

struct Sample {
  bool image, bank;  // inside (-1, H) x (-1, W); inside the bank
  int h0, w0, u0, v0;
  float lh, lw, lu, lv, pw;
};
__device__ __forceinline__ void bank_point(Sample& q, int tap, float r_h, float r_w, const Geom& g) {
  const int fh = tap / 3, fw = tap - fh * 3;
  const float u = ((float)fh + r_h) + (float)(g.scH - 3) * 0.5f, v = ((float)fw + r_w) + (float)(g.scW - 3) * 0.5f;
  q.bank = u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW;  // NaN fails
  const float fu = floorf(u), fv = floorf(v);
  q.u0 = q.bank ? (int)fu : 0, q.v0 = q.bank ? (int)fv : 0;
  q.lu = u - fu, q.lv = v - fv;
}
// offsets of a (pixel, tap): image space h, w, kernel space h, w
struct Offsets {
  __half v[4];
};
// off_n, rot_n: the sample's 18 planes; rot_n may be null (zeros)
__device__ __forceinline__ Offsets offsets_at(int tap, int oh, int ow, const __half* __restrict__ off_n, const __half* __restrict__ rot_n,
                                              const Geom& g) {
  const size_t o = (size_t)(2 * tap) * g.P + oh * g.Wo + ow;
  const __half z = __float2half(0.f);
  return {{__ldg(off_n + o), __ldg(off_n + o + g.P), rot_n ? __ldg(rot_n + o) : z, rot_n ? __ldg(rot_n + o + g.P) : z}};
}
__device__ __forceinline__ Sample sample_at(int tap, int oh, int ow, const Offsets& by, const Geom& g) {
  const int fh = tap / 3, fw = tap - fh * 3;
  Sample q;
  const float ph = (float)(oh * g.sH - 1 + fh) + __half2float(by.v[0]);
  q.pw = (float)(ow * g.sW - 1 + fw) + __half2float(by.v[1]);
  q.image = ph > -1.f && q.pw > -1.f && ph < (float)g.H && q.pw < (float)g.W;
  const float fph = floorf(ph), fpw = floorf(q.pw);
  q.h0 = q.image ? (int)fph : 0, q.w0 = q.image ? (int)fpw : 0;
  q.lh = ph - fph, q.lw = q.pw - fpw;
  bank_point(q, tap, __half2float(by.v[2]), __half2float(by.v[3]), g);
  return q;
}
__device__ __forceinline__ Sample sample_at(int tap, int oh, int ow, const __half* __restrict__ off_n, const __half* __restrict__ rot_n,
                                            const Geom& g) {
  return sample_at(tap, oh, ow, offsets_at(tap, oh, ow, off_n, rot_n, g), g);
}

// rows of 16 halves whose two 16-byte halves change places in every other group of four rows: ldmatrix reads eight rows without conflict
__device__ __forceinline__ int swz(int row, int half) { return row * 2 + (half ^ ((row >> 2) & 1)); }

// row of the hat products of pixel px: the pixels 4 q + i of a group of 16 that are read together are neighbours
__device__ __forceinline__ int beta_row(int px) { return (px & ~15) + (px & 3) * 4 + ((px & 15) >> 2); }
// hat products of the bank, one row of 16 cells: 4 x 4 whatever the scope is, the bank has zeros in the cells it lacks
__device__ __forceinline__ void put_beta(uint4* rows, int row, bool used, const Sample& q) {
  const float u = used && q.bank ? (float)q.u0 + q.lu : 1e30f, v = (float)q.v0 + q.lv;
  unsigned r[8];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    const float hu = hat(u - (float)a);
    r[2 * a] = pack2(hu * hat(v), hu * hat(v - 1.f));
    r[2 * a + 1] = pack2(hu * hat(v - 2.f), hu * hat(v - 3.f));
  }
  rows[swz(row, 0)] = make_uint4(r[0], r[1], r[2], r[3]);
  rows[swz(row, 1)] = make_uint4(r[4], r[5], r[6], r[7]);
}
template <int OFF = 0>
__device__ __forceinline__ void ldsm4(unsigned (&r)[4], unsigned a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4 + %5];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a), "n"(OFF));
}
template <int OFF = 0>
__device__ __forceinline__ void ldsm4t(unsigned (&r)[4], unsigned a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4 + %5];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a), "n"(OFF));
}
__device__ __forceinline__ unsigned saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
// The products of dk_mma_common.cuh without `volatile`: here the compiler may interleave the chains.
__device__ __forceinline__ void mul16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mad16(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mul16h(unsigned (&d)[2], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f16.f16.f16.f16 {%0,%1}, {%2,%3,%4,%5}, {%6,%7}, {%8,%8};\n"
      : "=r"(d[0]), "=r"(d[1])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0u));
}
__device__ __forceinline__ unsigned fma2h(unsigned a, unsigned b, unsigned c) {
  const __half2 r = __hfma2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b), *reinterpret_cast<const __half2*>(&c));
  return *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ unsigned word(const uint4& v, int k) { return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w; }
__device__ __forceinline__ uint4 line16(const char* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ unsigned sub2h(unsigned a, unsigned b) {
  const __half2 r = __hsub2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
  return *reinterpret_cast<const unsigned*>(&r);
}
// differences of the corners: lower - upper on the left and on the right, right - left above and below
__device__ __forceinline__ unsigned across(const uint4 (&x)[4], int k, int j) {
  return k < 2 ? sub2h(word(x[k + 2], j), word(x[k], j)) : sub2h(word(x[2 * k - 3], j), word(x[2 * k - 4], j));
}
// the four corners of a sample
__device__ __forceinline__ void corners(uint4 (&x)[4], const char* upper, size_t below) {
  const char* lower = upper + below;
  x[0] = line16(upper), x[1] = line16(upper + kLine), x[2] = line16(lower), x[3] = line16(lower + kLine);
}
__device__ __forceinline__ unsigned short cell_bits(const __half* __restrict__ w, int c, int k, const Geom& g) {  // cell k of the 4 x 4 grid
  const int a = k >> 2, b = k & 3;
  return c < g.C && a < g.scH && b < g.scW ? __half_as_ushort(__ldg(w + (size_t)c * g.cells + a * g.scW + b)) : (unsigned short)0;
}
__device__ __forceinline__ unsigned cells2(const __half* __restrict__ w, int c, int k, const Geom& g) {  // cells k, k + 1 of channel c
  return cell_bits(w, c, k, g) | (unsigned)cell_bits(w, c, k + 1, g) << 16;
}
__device__ __forceinline__ unsigned chans2(const __half* __restrict__ w, int c, int k, const Geom& g) {  // channels c, c + 1 of cell k
  return cell_bits(w, c, k, g) | (unsigned)cell_bits(w, c + 1, k, g) << 16;
}

// byte offset of the line of the upper left corner
__device__ __forceinline__ unsigned corner_line(const Sample& q, int n, const LineGeom& lg) {
  const int W2 = lg.g.W + 2, at = q.image ? (q.h0 + 1) * W2 + q.w0 + 1 : (lg.g.H + 1) * W2;
  return (unsigned)(n * lg.xs + at) * kLine;
}
__device__ __forceinline__ unsigned low2(unsigned c) {
  const __half2 r = __low2half2(*reinterpret_cast<const __half2*>(&c));
  return *reinterpret_cast<const unsigned*>(&r);
}
__device__ __forceinline__ unsigned high2(unsigned c) {
  const __half2 r = __high2half2(*reinterpret_cast<const __half2*>(&c));
  return *reinterpret_cast<const unsigned*>(&r);
}

// Bank operand of K for the lane's 64 channels from c0 on: [half][tile]
__device__ __forceinline__ void bank_tiles(unsigned (&wb)[2][4][2], const __half* __restrict__ w, int c0, int lane, const Geom& g) {
  const int gq = lane >> 2, t = lane & 3;
#pragma unroll
  for (int hf = 0; hf < 2; ++hf)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = c0 + hf * 32 + 8 * (gq >> 1) + 2 * j + (gq & 1);
      wb[hf][j][0] = cells2(w, c, 2 * t, g);
      wb[hf][j][1] = cells2(w, c, 2 * t + 8, g);
    }
}
// the lane's row of the hat products of a group of 16 pixels for ldmatrix
__device__ __forceinline__ unsigned kernel_rows(const uint4* rows, int lane) {
  return saddr(rows + swz(((lane >> 3) & 1) * 4 + ((lane & 7) >> 1), lane >> 4));
}
// K of the pixels 4 q + I, + I + 1
template <int I>
__device__ __forceinline__ void kernel_values(unsigned (&kk)[4][2], unsigned rows, const unsigned (&wb)[2][4][2], bool upper) {
  unsigned a[4];
  ldsm4<I * 128>(a, rows);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    unsigned low[2], high[2];
    mul16h(low, a, wb[0][j][0], wb[0][j][1]);
    mul16h(high, a, wb[1][j][0], wb[1][j][1]);
    kk[j][0] = upper ? high[0] : low[0], kk[j][1] = upper ? high[1] : low[1];
  }
}

// ------------------------------------------------------------------ forward
// Block: 64 pixels, a unit of 64 channels after the other; a warp has 16 of the pixels.
constexpr int kFwdPixels = 64;
struct FwdSmem {
  uint4 beta[kLineTaps][kFwdPixels * 2];
  uint4 cf[kLineTaps][kFwdPixels / 2];    // per pixel two words: coefficients of the upper and the lower corners
  uint4 line[kLineTaps][kFwdPixels / 4];  // per pixel a word
  unsigned at[kFwdPixels];                // element of y of channel 0, ~0u behind the last pixel
};

__device__ __forceinline__ void forward_unit(const FwdSmem& sm, const __half* __restrict__ xt, const __half* __restrict__ w,
                                             __half* __restrict__ y, const LineGeom& lg, int m, int c0, int lane, int run) {
  const Geom& g = lg.g;
  const int gq = lane >> 2, t = lane & 3, q = lane >> 3;
  unsigned wb[2][4][2];
  bank_tiles(wb, w, c0, lane, g);
  float acc[4][8];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int k = 0; k < 8; ++k) acc[i][k] = 0.f;
  const char* base = reinterpret_cast<const char*>(xt) + (c0 >> 6) * lg.xu + (lane & 7) * 16;
  const size_t below = (g.W + 2) * kLine;
  // the next tap's corners are loaded while this one's samples are multiplied
  uint4 x[4][4];
  auto fetch = [&](const uint4& lines) {
#pragma unroll
    for (int i = 0; i < 4; ++i) corners(x[i], base + word(lines, i), below);
  };
  const uint4* lines = sm.line[0] + m / 4 + q;
  const uint4* cfs = sm.cf[0] + m / 2 + 2 * q;
  unsigned rows = kernel_rows(sm.beta[0] + m * 2, lane);
  const bool upper = lane & 4;
  fetch(*lines);
#pragma unroll 1
  for (int tap = 0; tap < kLineTaps; ++tap, cfs += kFwdPixels / 2, rows += sizeof(sm.beta[0])) {
    unsigned v[4][4];
    const uint4 c01 = cfs[0], c23 = cfs[1];
    const unsigned cf[8] = {c01.x, c01.y, c01.z, c01.w, c23.x, c23.y, c23.z, c23.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        v[i][j] = fma2h(word(x[i][3], j), high2(cf[2 * i + 1]), fma2h(word(x[i][2], j), low2(cf[2 * i + 1]),
                  fma2h(word(x[i][1], j), high2(cf[2 * i]), hmul2u(word(x[i][0], j), low2(cf[2 * i])))));
    lines += kFwdPixels / 4;
    if (tap + 1 < kLineTaps) fetch(*lines);
    unsigned kk[4][2];
    auto products = [&](int i) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fma_hh<0, 0>(acc[i][2 * j], kk[j][0], v[i][j]);
        fma_hh<1, 1>(acc[i][2 * j + 1], kk[j][0], v[i][j]);
        fma_hh<0, 0>(acc[i + 1][2 * j], kk[j][1], v[i + 1][j]);
        fma_hh<1, 1>(acc[i + 1][2 * j + 1], kk[j][1], v[i + 1][j]);
      }
    };
    kernel_values<0>(kk, rows, wb, upper);
    products(0);
    kernel_values<2>(kk, rows, wb, upper);
    products(2);
  }
  // after the transposition a lane has two channels, c and c + 32, of the four neighbouring pixels 4 t + i
  const uint4 at = *reinterpret_cast<const uint4*>(sm.at + m + 4 * t);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    unsigned v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = movmatrix_trans(pack2(acc[i][2 * j], acc[i][2 * j + 1]));
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int c = c0 + hf * 32 + 8 * (gq >> 1) + 2 * j + (gq & 1);
      const unsigned lo = __byte_perm(v[0], v[1], hf ? 0x7632 : 0x5410), hi = __byte_perm(v[2], v[3], hf ? 0x7632 : 0x5410);
      if (c < g.C) {
        __half* to = y + (size_t)c * g.P;
        if (run == 4) {
          if (at.x != ~0u) *reinterpret_cast<uint2*>(to + at.x) = make_uint2(lo, hi);
        } else if (run == 2) {
          if (at.x != ~0u) *reinterpret_cast<unsigned*>(to + at.x) = lo;
          if (at.z != ~0u) *reinterpret_cast<unsigned*>(to + at.z) = hi;
        } else {
          if (at.x != ~0u) to[at.x] = __ushort_as_half((unsigned short)lo);
          if (at.y != ~0u) to[at.y] = __ushort_as_half((unsigned short)(lo >> 16));
          if (at.z != ~0u) to[at.z] = __ushort_as_half((unsigned short)hi);
          if (at.w != ~0u) to[at.w] = __ushort_as_half((unsigned short)(hi >> 16));
        }
      }
    }
  }
}

__global__ void __launch_bounds__(128, 3) line_forward_kernel(const __half* __restrict__ xt, const __half* __restrict__ off,
                                                              const __half* __restrict__ rot, const __half* __restrict__ w,
                                                              __half* __restrict__ y, const __grid_constant__ LineGeom lg, const int run) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FwdSmem& sm = *reinterpret_cast<FwdSmem*>(smem_raw);
  const Geom& g = lg.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int total = g.N * g.P, f0 = blockIdx.x * kFwdPixels;
  {
    const int px = threadIdx.x & 63, f = f0 + px;
    int n = 0, oh = 0, ow = 0;
    if (f < total) strip_pixel(f, lg, n, oh, ow);
    if (threadIdx.x < 64) sm.at[px] = f < total ? (unsigned)n * g.C * g.P + oh * g.Wo + ow : ~0u;
    const size_t pn = (size_t)n * 18 * g.P;
    constexpr int kEach = (kLineTaps + 1) / 2;
    Offsets by[kEach];  // all loads of the thread in flight together
#pragma unroll
    for (int k = 0; k < kEach; ++k)
      by[k] = offsets_at(min((int)(threadIdx.x >> 6) + 2 * k, kLineTaps - 1), oh, ow, off + pn, rot ? rot + pn : nullptr, g);
#pragma unroll
    for (int k = 0; k < kEach; ++k) {
      const int tap = (threadIdx.x >> 6) + 2 * k;
      if (tap >= kLineTaps) break;
      Sample q = sample_at(tap, oh, ow, by[k], g);
      if (f >= total) q.image = false;
      const float hh = 1.f - q.lh, hw = 1.f - q.lw;
      reinterpret_cast<unsigned*>(sm.line[tap])[px] = corner_line(q, n, lg);
      reinterpret_cast<uint2*>(sm.cf[tap])[px] = q.image ? make_uint2(pack2(hh * hw, hh * q.lw), pack2(q.lh * hw, q.lh * q.lw)) : make_uint2(0u, 0u);
      put_beta(sm.beta[tap], beta_row(px), q.image, q);
    }
  }
  __syncthreads();
  const int m = warp * 16;
  for (int c0 = blockIdx.y * 64; c0 < g.C; c0 += gridDim.y * 64) {
    forward_unit(sm, xt, w, y, lg, m, c0, lane, run);
  }
}

// ------------------------------------------------------------------ offset and bank gradients
// d(kernel offset) = sum_c dy xs dK/d(u|v): G = (dy xs) W as an mma over the channels, then the four cells around the sample
// with the derivatives of the hats.  d(image offset) = sum_c dy K dxs/d(h|w): from the four sums S_k = sum_c (dy K) dx_k over
// the differences of neighbouring corners, an mma of the products whose other operand is one in the columns k, k + 4; a pixel's two rows are its two
// halves of the channels.  Products with the corners themselves, subtracted afterwards, overflow where only the corners are large (x of 100, dy
// of 500) and lose what they have in common: 8 x 512 of 28 x 28 with x around 10, 1.1e-3 off fp64 against 4.5e-4 (4.6e-4 and 5.1e-4 around 0).
// 543 -> 590 us for the differences, 573 with runs of tiles as equal as they can be.  dW = beta^T (dy xs) over the pixels, for which movmatrix turns the products.
// A warp has 64 channels for the whole run of its block (the bank sums stay in registers) and walks over groups of 16 pixels;
// the warps of a stream have different channels of the same pixels, and their sums over channels meet in shared memory.
struct CoordPlan {
  int units, upb, streams, sets, tiles, blocks;  // units of channels, of a block; groups of pixels of a block; channel sets
  size_t smem;
};
constexpr int kGridRow = 6, kGridNone = 36, kGridCells = 44, kGridPitch = 16;  // 6 x 6 cells with a border of zeros, and zeros behind; 16 pixels

template <bool ROT>
__global__ void __launch_bounds__(128, 3) line_coords_kernel(const __half* __restrict__ dyt, const __half* __restrict__ xt,
                                                             const __half* __restrict__ off, const __half* __restrict__ rot,
                                                             const __half* __restrict__ w, __half* __restrict__ doff,
                                                             __half* __restrict__ drot, float* __restrict__ sums,
                                                             float* __restrict__ bank, const __grid_constant__ LineGeom lg, const CoordPlan pl) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const Geom& g = lg.g;
  const int npx = 16 * pl.streams, nwarps = blockDim.x >> 5;
  constexpr int NP = ROT ? 160 : 128;  // floats that a warp leaves for 16 pixels and a tap: S [half][pixel][difference], then u and v
  uint4* beta = reinterpret_cast<uint4*>(smem_raw);                               // [tap][npx][2]
  uint4* wgs = beta + kLineTaps * npx * 2;                                        // [unit][4 steps of 16 channels][lane]
  float* grids = reinterpret_cast<float*>(wgs + (ROT ? pl.upb * 128 : 0));        // [warp][kGridCells][kGridPitch]
  float* part = grids + (ROT ? nwarps * kGridCells * kGridPitch : 0);             // [warp][tap][NP]
  float4* bp = reinterpret_cast<float4*>(part + nwarps * kLineTaps * NP);         // [tap][npx] {cell of the grid, lu, lv, -}
  uint2* cf = reinterpret_cast<uint2*>(bp + (ROT ? kLineTaps * npx : 0));         // [tap][npx] coefficients of the upper, the lower corners
  float2* frac = reinterpret_cast<float2*>(cf + kLineTaps * npx);                 // [2][tap][npx] {lh, lw}
  unsigned* line = reinterpret_cast<unsigned*>(frac + 2 * kLineTaps * npx);       // [tap][npx]
  unsigned* at = line + kLineTaps * npx;                                          // [npx] line of dy
  unsigned* to_px = at + npx;                                                     // [2][npx] element of the first offset plane, ~0u behind the last pixel
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, t = lane & 3, q4 = (lane >> 3) * 4;
  const int stream = warp / pl.upb, ub = warp - stream * pl.upb, unit = blockIdx.y * pl.upb + ub, c0 = unit * 64;
  const bool active = unit < pl.units, upper = lane & 4;
  const int total = g.N * g.P;
  float* grid = grids + warp * kGridCells * kGridPitch;
  if (ROT)
    for (int i = lane; i < kGridCells * kGridPitch; i += 32) grid[i] = 0.f;

  unsigned wk[2][4][2];
  bank_tiles(wk, w, active ? c0 : g.C, lane, g);
  const uint4* wg = wgs + ub * 128 + lane;
  if (ROT && stream == 0) {
#pragma unroll
    for (int s = 0; s < 4; ++s) {  // W^T of the half s >> 1 and its tiles 2 (s & 1), + 1
      const int c = active ? c0 + (s >> 1) * 32 + 8 * t + 4 * (s & 1) : g.C;
      wgs[ub * 128 + lane + s * 32] = make_uint4(chans2(w, c, gq, g), chans2(w, c, gq + 8, g), chans2(w, c + 2, gq, g), chans2(w, c + 2, gq + 8, g));
    }
  }
  unsigned one[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) one[k] = (gq & 3) == k ? 0x3C003C00u : 0u;
  // where the lane's cell gq of G, pixels 4 t .. + 3, goes; cell gq + 8 is two rows below
  float* grid_w = grid + (((gq >> 2) + 1) * kGridRow + (gq & 3) + 1) * kGridPitch + 4 * t;
  float acc[8][4];
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  const size_t below = (g.W + 2) * kLine;
  const char* xb = reinterpret_cast<const char*>(xt) + unit * lg.xu + (lane & 7) * 16;
  const char* yb = reinterpret_cast<const char*>(dyt) + unit * lg.yu + (lane & 7) * 16;
  const int my_px = threadIdx.x & (npx - 1), tap0 = threadIdx.x / npx, taps_step = blockDim.x / npx;  // npx is a power of two
  // the hat products turned: the two k-slots of a lane are the pixels 4 t, + 1 and 4 t + 2, + 3
  const int trow = stream * 16 + ((lane & 1) + 2 * (lane >> 4)) * 4 + ((lane & 7) >> 1);
  const int tile_end = (int)((long long)pl.tiles * (blockIdx.x + 1) / pl.blocks);
  for (int tile = (int)((long long)pl.tiles * blockIdx.x / pl.blocks); tile < tile_end; ++tile) {
    const int f0 = tile * npx, flip = tile & 1;
    {
      const int f = f0 + my_px;
      int n = 0, oh = 0, ow = 0;
      if (f < total) strip_pixel(f, lg, n, oh, ow);
      const size_t pn = (size_t)n * 18 * g.P;
      if (tap0 == 0) {
        at[my_px] = (unsigned)(f < total ? n * g.P + oh * g.Wo + ow : total) * kLine;
        to_px[flip * npx + my_px] = f < total ? (unsigned)pn + oh * g.Wo + ow : ~0u;
      }
      for (int tap = tap0; tap < kLineTaps; tap += taps_step) {
        const int e = tap * npx + my_px;
        Sample q = sample_at(tap, oh, ow, off + pn, rot ? rot + pn : nullptr, g);
        if (f >= total) q.image = false;
        const float hh = 1.f - q.lh, hw = 1.f - q.lw;
        line[e] = corner_line(q, n, lg);
        cf[e] = q.image ? make_uint2(pack2(hh * hw, hh * q.lw), pack2(q.lh * hw, q.lh * q.lw)) : make_uint2(0u, 0u);
        frac[flip * kLineTaps * npx + e] = q.image ? make_float2(q.lh, q.lw) : make_float2(0.f, 0.f);
        put_beta(beta + tap * npx * 2, beta_row(my_px), q.image, q);
        if (ROT) bp[e] = make_float4(__int_as_float((q.bank ? (q.u0 + 1) * kGridRow + q.v0 + 1 : kGridNone) * kGridPitch), q.bank ? q.lu : 0.f, q.bank ? q.lv : 0.f, 0.f);
      }
    }
    __syncthreads();
    if (active) {
      uint4 dy[4];
      {
        const uint4 a = *reinterpret_cast<const uint4*>(at + stream * 16 + q4);
#pragma unroll
        for (int i = 0; i < 4; ++i) dy[i] = line16(yb + word(a, i));
      }
      float* out = part + (size_t)warp * kLineTaps * NP;
      const unsigned* lines = line + stream * 16 + q4;
      const uint2* cfs = cf + stream * 16 + q4;
      const float4* bps = bp + stream * 16 + (lane & 15);
      unsigned rows = kernel_rows(beta + stream * 32, lane), turned = saddr(beta + swz(trow, (lane >> 3) & 1));
      uint4 xa[4], xe[4];
      {
        const uint2 l = *reinterpret_cast<const uint2*>(lines);
        corners(xa, xb + l.x, below), corners(xe, xb + l.y, below);
      }
#pragma unroll 1
      for (int tap = 0; tap < kLineTaps; ++tap, cfs += npx, bps += npx, out += NP, rows += npx * 32, turned += npx * 32) {
        unsigned dk[4][4];
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const uint4 c = *reinterpret_cast<const uint4*>(cfs + i);
          unsigned kk[4][2];
          if (i == 0) kernel_values<0>(kk, rows, wk, upper);
          else kernel_values<2>(kk, rows, wk, upper);
          unsigned yk[4][2];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            auto sampled = [&](const uint4 (&x)[4], unsigned up, unsigned low) {
              return fma2h(word(x[3], j), high2(low), fma2h(word(x[2], j), low2(low), fma2h(word(x[1], j), high2(up), hmul2u(word(x[0], j), low2(up)))));
            };
            dk[i][j] = hmul2u(word(dy[i], j), sampled(xa, c.x, c.y));
            dk[i + 1][j] = hmul2u(word(dy[i + 1], j), sampled(xe, c.z, c.w));
            yk[j][0] = hmul2u(kk[j][0], word(dy[i], j));
            yk[j][1] = hmul2u(kk[j][1], word(dy[i + 1], j));
          }
          float D[4], E[4];
#pragma unroll
          for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              const unsigned a[4] = {hmul2u(yk[j][0], across(xa, k, j)), hmul2u(yk[j][1], across(xe, k, j)),
                                     hmul2u(yk[j + 1][0], across(xa, k, j + 1)), hmul2u(yk[j + 1][1], across(xe, k, j + 1))};
              if (k == 0) mul16(j ? E : D, a, one[k], one[k]);
              else mad16(j ? E : D, a[0], a[1], a[2], a[3], one[k], one[k]);
            }
#pragma unroll
          for (int k = 0; k < 4; ++k) D[k] += E[k];
          // the next two pixels' corners, under the products that follow
          if (i == 0) {
            const uint2 l = *reinterpret_cast<const uint2*>(lines + 2);
            corners(xa, xb + l.x, below), corners(xe, xb + l.y, below);
          } else if (tap + 1 < kLineTaps) {
            lines += npx;
            const uint2 l = *reinterpret_cast<const uint2*>(lines);
            corners(xa, xb + l.x, below), corners(xe, xb + l.y, below);
          }
          // columns 2 t, 2 t + 1 are the corners 2 (t & 1), + 1; the lanes t < 2 store pixel i, the others i + 1
          *reinterpret_cast<float2*>(out + ((gq & 1) * 16 + q4 + i + (t >> 1)) * 4 + 2 * (t & 1)) = t & 2 ? make_float2(D[2], D[3]) : make_float2(D[0], D[1]);
        }
        {
          unsigned bt[4];
          ldsm4t(bt, turned);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const unsigned m0 = movmatrix_trans(dk[0][j]), m1 = movmatrix_trans(dk[1][j]), m2 = movmatrix_trans(dk[2][j]), m3 = movmatrix_trans(dk[3][j]);
            mad16(acc[j], bt[0], bt[1], bt[2], bt[3], __byte_perm(m0, m1, 0x5410), __byte_perm(m2, m3, 0x5410));
            mad16(acc[4 + j], bt[0], bt[1], bt[2], bt[3], __byte_perm(m0, m1, 0x7632), __byte_perm(m2, m3, 0x7632));
          }
        }
        if (ROT) {
          // G of a pixel: the column of its lower channels with their bank plus the column beside it with that of the upper ones
          float G[2][4];  // cells gq and gq + 8 of the pixels 4 t + i
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            const uint4 w0 = wg[hf * 64], w1 = wg[hf * 64 + 32];
            const unsigned a0[4] = {w0.x, w0.y, w0.z, w0.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              float d[4];
              mul16(d, a0, dk[i][0], dk[i][1]);
              mad16(d, w1.x, w1.y, w1.z, w1.w, dk[i][2], dk[i][3]);
              G[0][i] = hf ? G[0][i] + d[1] : d[0];
              G[1][i] = hf ? G[1][i] + d[3] : d[2];
            }
          }
          __syncwarp();  // the previous tap's sums have been read
          *reinterpret_cast<float4*>(grid_w) = make_float4(G[0][0], G[0][1], G[0][2], G[0][3]);
          *reinterpret_cast<float4*>(grid_w + 2 * kGridRow * kGridPitch) = make_float4(G[1][0], G[1][1], G[1][2], G[1][3]);
          __syncwarp();
          const int px = lane & 15;
          const bool dv = lane >= 16;
          const float4 b = *bps;
          const float* c = grid + __float_as_int(b.x) + px;
          const float g00 = c[0], g01 = c[kGridPitch], g10 = c[kGridRow * kGridPitch], g11 = c[(kGridRow + 1) * kGridPitch];
          const float l = dv ? b.y : b.z;
          out[128 + lane] = (1.f - l) * ((dv ? g01 : g10) - g00) + l * (g11 - (dv ? g10 : g01));
        }
      }
    }
    __syncthreads();
    // sums over the warps of a stream, in their order; the next tile's samples are written meanwhile
    const int live = min(pl.upb, pl.units - (int)blockIdx.y * pl.upb), px = threadIdx.x & 15;
    for (int i = threadIdx.x >> 4; i < pl.streams * kLineTaps * (ROT ? 2 : 1); i += blockDim.x >> 4) {
      const int r = ROT ? i >> 1 : i, st = pl.streams == 1 ? 0 : r / kLineTaps, tap = r - st * kLineTaps;
      const unsigned o = to_px[flip * npx + st * 16 + px];
      if (o == ~0u) continue;
      const float* from = part + ((size_t)st * pl.upb * kLineTaps + tap) * NP;
      float a = 0.f, b = 0.f;
      const bool kernel_space = ROT && (i & 1);
      if (kernel_space) {
        for (int q = 0; q < live; ++q) a += from[q * kLineTaps * NP + 128 + px], b += from[q * kLineTaps * NP + 144 + px];
      } else {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int q = 0; q < 2 * live; ++q) {
          const float4 v = *reinterpret_cast<const float4*>(from + (q >> 1) * kLineTaps * NP + ((q & 1) * 16 + px) * 4);
          s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
        }
        const float2 l = frac[flip * kLineTaps * npx + tap * npx + st * 16 + px];
        a = (1.f - l.y) * s.x + l.y * s.y;
        b = (1.f - l.x) * s.z + l.x * s.w;
      }
      if (pl.sets == 1) {
        __half* to = kernel_space ? drot : doff;
        if (to) to += o + (unsigned)(2 * tap) * g.P, to[0] = __float2half_rn(a), to[g.P] = __float2half_rn(b);
      } else {
        float* to = sums + (((size_t)blockIdx.y * kLineTaps + tap) * (ROT ? 4 : 2) + (kernel_space ? 2 : 0)) * total + f0 + st * 16 + px;
        to[0] = a, to[total] = b;
      }
    }
  }
  if (bank != nullptr) {
    __syncthreads();
    float* red = reinterpret_cast<float*>(smem_raw);  // [warp][64 channels][16 cells]
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) red[(warp * 64 + (j >> 2) * 32 + 8 * t + 2 * (j & 3) + (k & 1)) * 16 + gq + (k >> 1) * 8] = acc[j][k];
    __syncthreads();
    for (int i = threadIdx.x; i < pl.upb * 1024; i += blockDim.x) {
      const int q = i >> 10, r = i & 1023, c = (blockIdx.y * pl.upb + q) * 64 + (r >> 4), a = (r >> 2) & 3, b = r & 3;
      if (c >= g.C || a >= g.scH || b >= g.scW) continue;
      float s = 0.f;
      for (int st = 0; st < pl.streams; ++st) s += red[(st * pl.upb + q) * 1024 + r];
      bank[((size_t)blockIdx.x * g.C + c) * g.cells + a * g.scW + b] = s;
    }
  }
}

// offset gradients from the sums of the channel sets, in their order
__global__ void __launch_bounds__(256) line_coord_sums_kernel(const float* __restrict__ sums, __half* __restrict__ doff,
                                                              __half* __restrict__ drot, const __grid_constant__ LineGeom lg, int sets, int NK) {
  const Geom& g = lg.g;
  const int total = g.N * g.P, tk = blockIdx.y, tap = tk / NK, k = tk - tap * NK;
  const int f = blockIdx.x * 256 + threadIdx.x;
  __half* to = k < 2 ? doff : drot;
  if (f >= total || to == nullptr) return;
  float s = 0.f;
  for (int q = 0; q < sets; ++q) s += __ldg(sums + ((size_t)q * kLineTaps * NK + tk) * total + f);
  int n, oh, ow;
  strip_pixel(f, lg, n, oh, ow);
  to[((size_t)n * 18 + 2 * tap + (k & 1)) * g.P + oh * g.Wo + ow] = __float2half_rn(s);
}

// ------------------------------------------------------------------ grad-input
// Counting sort of the samples of an image by the cell of the input grid they fall into, by a cluster of blocks with a
// contiguous share of the samples each: a block counts its share and lays its numbers out by cell in shared memory; the blocks
// share the prefix sums (a part of the cells each, through distributed shared memory); a sample's place is then the first of its
// cell and block plus its rank by number among those: the order, and with it every sum of the gather, is the same in every run.
// record: {column of the sample point, fraction of its row, kernel-space offsets, tap << 27 | pixel}
__global__ void __launch_bounds__(kSortThreads, 3) line_sort_kernel(const __half* __restrict__ off, const __half* __restrict__ rot,
                                                                    int* __restrict__ starts, float4* __restrict__ recs,
                                                                    const __grid_constant__ LineGeom lg, const int bins, const int share) {
  extern __shared__ __align__(16) int hist[];  // [bins] counts, then first places; [bins + 1] first local places; [share] numbers
  __shared__ int slices[kSortBlocks], warp_sum[kSortThreads / 32];
  int* local = hist + bins;
  int* ids = local + bins + 1;
  const Geom& g = lg.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = blockIdx.x / kSortBlocks, rank = blockIdx.x - n * kSortBlocks;
  cg::cluster_group cluster = cg::this_cluster();
  const size_t pn = (size_t)n * 18 * g.P;
  const __half* off_n = off + pn;
  const __half* rot_n = rot ? rot + pn : nullptr;
  const int count = kLineTaps * g.P, lo_i = min(rank * share, count), hi_i = min(lo_i + share, count);
  auto cell_of = [&](int i, Sample& q, int& tap, int& p) {
    tap = i / lg.P, p = i - tap * g.P;
    const int oh = p / lg.Wo;
    q = sample_at(tap, oh, p - oh * g.Wo, off_n, rot_n, g);
    return q.image && q.bank ? (q.h0 + 1) * (g.W + 1) + q.w0 + 1 : -1;
  };
  // exclusive prefix sums over the threads
  auto scan = [&](int v, int& all) {
    int s = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, s, d);
      if (lane >= d) s += o;
    }
    __syncthreads();
    if (lane == 31) warp_sum[warp] = s;
    __syncthreads();
    int base = 0;
    all = 0;
#pragma unroll
    for (int k = 0; k < kSortThreads / 32; ++k) {
      if (k < warp) base += warp_sum[k];
      all += warp_sum[k];
    }
    return base + s - v;
  };
  for (int i = tid; i < bins; i += kSortThreads) hist[i] = 0;
  __syncthreads();
#pragma unroll 2
  for (int i = lo_i + tid; i < hi_i; i += kSortThreads) {
    Sample q;
    int tap, p;
    const int cell = cell_of(i, q, tap, p);
    if (cell >= 0) atomicAdd(&hist[cell], 1);
  }
  __syncthreads();
  {
    const int each = (bins + kSortThreads - 1) / kSortThreads, lo = min(tid * each, bins), end = min(lo + each, bins);
    int sum = 0, all;
    for (int b = lo; b < end; ++b) sum += hist[b];
    int run = scan(sum, all);
    for (int b = lo; b < end; ++b) local[b] = run, run += hist[b];
    if (tid == 0) local[bins] = all;
  }
  cluster.sync();
  {
    const int per = (bins + kSortBlocks - 1) / kSortBlocks, each = (per + kSortThreads - 1) / kSortThreads;
    const int hi = min((rank + 1) * per, bins), lo = min(rank * per + tid * each, hi), end = min(lo + each, hi);
    int sum = 0, all;
    for (int b = lo; b < end; ++b)
#pragma unroll
      for (int k = 0; k < kSortBlocks; ++k) sum += cluster.map_shared_rank(hist, k)[b];
    int run = scan(sum, all);
    if (tid < kSortBlocks) cluster.map_shared_rank(slices, tid)[rank] = all;
    cluster.sync();
    int before = 0;
    for (int k = 0; k < rank; ++k) before += slices[k];
    run += before;
    int* out = starts + (size_t)n * (bins + 1);
    for (int b = lo; b < end; ++b) {
      out[b] = run;
      int c[kSortBlocks];
#pragma unroll
      for (int k = 0; k < kSortBlocks; ++k) c[k] = cluster.map_shared_rank(hist, k)[b];
#pragma unroll
      for (int k = 0; k < kSortBlocks; ++k) {
        cluster.map_shared_rank(hist, k)[b] = run;
        run += c[k];
      }
    }
    if (rank == kSortBlocks - 1 && tid == 0) out[bins] = before + all;
  }
  // the numbers by cell: local[cell] moves to the end of its cell, which is where the next one begins
#pragma unroll 2
  for (int i = lo_i + tid; i < hi_i; i += kSortThreads) {
    Sample q;
    int tap, p;
    const int cell = cell_of(i, q, tap, p);
    if (cell >= 0) ids[atomicAdd(&local[cell], 1)] = i;
  }
  cluster.sync();
  float4* to = recs + (size_t)n * count;
#pragma unroll 2
  for (int i = lo_i + tid; i < hi_i; i += kSortThreads) {
    Sample q;
    int tap, p;
    const int cell = cell_of(i, q, tap, p);
    if (cell >= 0) {
      int place = hist[cell];
      for (int k = cell ? local[cell - 1] : 0; k < local[cell]; ++k) place += ids[k] < i;
      const size_t o = (size_t)(2 * tap) * g.P + p;
      const unsigned r = rot_n ? (unsigned)__half_as_ushort(__ldg(rot_n + o)) | ((unsigned)__half_as_ushort(__ldg(rot_n + o + g.P)) << 16) : 0u;
      to[place] = make_float4(q.pw, q.lh, __uint_as_float(r), __uint_as_float((unsigned)tap << 27 | (unsigned)p));
    }
  }
}

struct GatherPlan {
  int R, bands, windows, warps, sets, bins;
};

// Grad-input of a row of a window, every product to its own corners only: for the elements whose sums in the window are not finite.  A lane has
// the channels c, c + 1; bit t (4 + t) of `wanted`: the columns 2 t, 2 t + 1 of c (c + 1).  The warp walks over the records of the two rows of
// cells once for all its channels and columns (an element at a time, all of 64 x 256 of 56 x 56 17 ms, so 3).
__device__ __noinline__ void gather_row_alone(const float4* __restrict__ rec_n, const int* __restrict__ st_n, const __half* __restrict__ dyt,
                                              const __half* __restrict__ w, __half* __restrict__ dx, const LineGeom& lg, int n, int c, int r, int w0,
                                              unsigned wanted) {
  const Geom& g = lg.g;
  const char* yl = reinterpret_cast<const char*>(dyt) + (c >> 6) * lg.yu + (size_t)n * g.P * kLine + (c & 63) * 2;
  const int lane = threadIdx.x & 31;
  unsigned bank[36];  // both channels, the first one's in the low halves: 4 x 4 cells with a border of zeros
#pragma unroll
  for (int k = 0; k < 36; ++k) {
    const int a = k / 6 - 1, b = k - (k / 6) * 6 - 1;
    bank[k] = a >= 0 && a < 4 && b >= 0 && b < 4 ? chans2(w, c, a * 4 + b, g) : 0u;
  }
  float2 sum[10];  // columns w0 - 1 .. w0 + 8
#pragma unroll
  for (int k = 0; k < 10; ++k) sum[k] = make_float2(0.f, 0.f);
  for (int h0 = r - 1; h0 <= r; ++h0) {
    const int* s = st_n + (h0 + 1) * (g.W + 1) + w0;
    const int last = s[min(9, g.W + 1 - w0)];
    int cur = 0;  // records come by column: the sums of two neighbours stay in registers
    float2 left = sum[0], right = sum[1];
    for (int i0 = s[0]; i0 < last; i0 += 32) {
      Sample q;  // a record per lane
      q.u0 = q.v0 = 0, q.lu = q.lv = 0.f;
      float lw = 0.f, row = 0.f;
      int col = 0, px = 0;
      if (i0 + lane < last) {
        const float4 rec = __ldg(rec_n + i0 + lane);
        const unsigned id = __float_as_uint(rec.w), r2 = __float_as_uint(rec.z);
        bank_point(q, id >> 27, lo2f(r2), hi2f(r2), g);
        const float fl = floorf(rec.x);
        lw = rec.x - fl, row = h0 == r ? 1.f - rec.y : rec.y, col = (int)fl - w0, px = id & 0x7ffffffu;
      }
      const int at = ((q.u0 + 1) * 6 + q.v0 + 1) << 4 | (col + 1), cnt = min(32, last - i0);
      const float cl = row * (1.f - lw), cr = row * lw;
      auto line = [&](int k) { return __ldg(reinterpret_cast<const unsigned*>(yl + (size_t)__shfl_sync(0xffffffffu, px, k) * kLine)); };
      unsigned y0 = line(0), y1 = line(1), y2 = line(2), y3 = line(3);
      // not unrolled: a body of eight records took twice as long, two thirds of it waiting for instructions
#pragma unroll 1
      for (int k = 0; k < cnt; ++k) {
        const unsigned y = y0;
        y0 = y1, y1 = y2, y2 = y3, y3 = line((k + 4) & 31);
        const int o = __shfl_sync(0xffffffffu, at, k);
        const float u = __shfl_sync(0xffffffffu, q.lu, k), t = __shfl_sync(0xffffffffu, q.lv, k);
        const float l = __shfl_sync(0xffffffffu, cl, k), m = __shfl_sync(0xffffffffu, cr, k);
        const unsigned* b = bank + (o >> 4);
        float a0 = 0.f, a1 = 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float h = (e >> 1 ? u : 1.f - u) * (e & 1 ? t : 1.f - t);
          const unsigned cell = b[(e >> 1) * 6 + (e & 1)];
          a0 += h * lo2f(cell), a1 += h * hi2f(cell);
        }
        const float v0 = a0 * lo2f(y), v1 = a1 * hi2f(y);
        while (cur < (o & 15)) sum[cur++] = left, left = right, right = sum[cur + 1];
        left.x += l * v0, left.y += l * v1;
        right.x += m * v0, right.y += m * v1;
      }
    }
    sum[cur] = left, sum[cur + 1] = right;
  }
  __half* o = dx + ((size_t)n * g.C + c) * g.HW + (size_t)r * g.W + w0;
  for (int k = 0; k < 8; ++k) {
    if (w0 + k >= g.W) break;
    if (c < g.C && (wanted >> (k >> 1) & 1)) o[k] = __float2half_rn(sum[k + 1].x);
    if (c + 1 < g.C && (wanted >> (4 + (k >> 1)) & 1)) o[g.HW + k] = __float2half_rn(sum[k + 1].y);
  }
}

// A block has 8 columns of R rows of dx and up to four units of 64 channels, a warp each.  It walks over the rows of cells that
// reach them; the samples of the cells of such a row that touch the columns are one run of the sorted records.  For 16 of
// them at a time: K^T [channel][sample] = W beta^T, times dy, is the first operand of dx^T [channel][column] += (K dy) coef, where
// the coefficients are the bilinear weights of the columns (two pieces of fp16 each, 22 bits), for the upper and the lower row.
__global__ void __launch_bounds__(128, 4) line_gather_kernel(const __half* __restrict__ dyt, const int* __restrict__ starts,
                                                             const float4* __restrict__ recs, const __half* __restrict__ w,
                                                             __half* __restrict__ dx, const __grid_constant__ LineGeom lg,
                                                             const GatherPlan pl, const bool pairs) {
  const Geom& g = lg.g;
  __shared__ uint4 beta[kChunk * 2], chi[kChunk * 2 + 1], clo[kChunk * 2 + 1];  // the last piece takes what is outside the columns
  __shared__ __align__(16) unsigned at[kChunk];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gq = lane >> 2, t = lane & 3;
  const int band = blockIdx.x % pl.bands, rest = blockIdx.x / pl.bands, win = rest % pl.windows, n = rest / pl.windows;
  const int r0 = band * pl.R, rows = min(pl.R, g.H - r0), w0 = win * 8;
  const int c0 = (blockIdx.y * pl.warps + warp) * 64;
  const unsigned none = (unsigned)(g.N * g.P) * kLine;
  const bool active = c0 < g.C;
  unsigned wa[4][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = c0 + 8 * (gq >> 1) + 2 * j + (gq & 1);
    wa[j][0] = cells2(w, c, 2 * t, g);
    wa[j][1] = cells2(w, c + 32, 2 * t, g);
    wa[j][2] = cells2(w, c, 2 * t + 8, g);
    wa[j][3] = cells2(w, c + 32, 2 * t + 8, g);
  }
  const char* yb = reinterpret_cast<const char*>(dyt) + (c0 >> 6) * lg.yu + (lane & 7) * 16;
  const int* st_n = starts + (size_t)n * (pl.bins + 1);
  const float4* rec_n = recs + (size_t)n * kLineTaps * g.P;
  float acc[2][4][4];  // [this row | the next][tile of 16 channels]
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[0][j][k] = acc[1][j][k] = 0.f;
  // ldmatrix: rows of the hat products (samples 0-7: cells 0-7, 8-15; samples 8-15 likewise), rows of the coefficients (samples 0-7, 8-15: upper; lower)
  const unsigned b_at = saddr(beta + swz((lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1));
  const unsigned h_at = saddr(chi + swz(lane & 15, lane >> 4)), l_at = saddr(clo + swz(lane & 15, lane >> 4));
  const int span = min(9, g.W + 1 - w0);
  const int* s = st_n + r0 * (g.W + 1) + w0;
  int next_first = __ldg(s), next_last = __ldg(s + span);
  const float4 nothing = make_float4(-1e30f, 0.f, 0.f, 0.f);
  float4 ahead = nothing;  // the record that the thread turns into operands first in the next chunk
  if (next_first + (int)threadIdx.x < next_last) ahead = __ldg(rec_n + next_first + threadIdx.x);
  for (int i = 0; i <= rows; ++i) {
    const int h0 = r0 - 1 + i;
    const bool up = i > 0, low = i < rows;
    const int first = next_first, last = next_last;
    if (low) s += g.W + 1, next_first = __ldg(s), next_last = __ldg(s + span);
    if (first >= last) {
      ahead = nothing;
      if (low && next_first + (int)threadIdx.x < next_last) ahead = __ldg(rec_n + next_first + threadIdx.x);
    }
    for (int at0 = first; at0 < last; at0 += kChunk) {
      const int cnt = min(kChunk, last - at0), steps = (cnt + 15) >> 4;
      __syncthreads();
      for (int e = threadIdx.x; e < steps * 16; e += blockDim.x) {
        const bool in = e < cnt;
        const int row = (e & ~15) + ((e & 2) << 2) + ((e >> 1) & 6) + (e & 1);  // the k-slot of sample 4 q + i
        const uint4 z = make_uint4(0, 0, 0, 0);
        chi[row * 2] = chi[row * 2 + 1] = clo[row * 2] = clo[row * 2 + 1] = z;
        Sample q;
        float4 rec = e < (int)blockDim.x ? ahead : nothing;
        if (in && e >= (int)blockDim.x) rec = __ldg(rec_n + at0 + e);
        const unsigned id = __float_as_uint(rec.w), r2 = __float_as_uint(rec.z);
        bank_point(q, id >> 27, lo2f(r2), hi2f(r2), g);
        const float fl = floorf(rec.x), lw = rec.x - fl;
        const int col = in ? (int)fl - w0 : -2;
        __half* hi = reinterpret_cast<__half*>(chi);
        __half* lo = reinterpret_cast<__half*>(clo);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int cc = col + (k & 1);
          const float v = (k >> 1 ? rec.y : 1.f - rec.y) * (k & 1 ? lw : 1.f - lw);
          const __half vh = __float2half_rn(v);
          const int o = (unsigned)cc < 8u ? swz(row, k >> 1) * 8 + cc : kChunk * 16;
          hi[o] = vh;
          lo[o] = __float2half_rn(v - __half2float(vh));
        }
        put_beta(beta, row, in, q);
        at[e] = in ? ((unsigned)(n * g.P) + (id & 0x7ffffffu)) * kLine : none;
      }
      {
        const bool more = at0 + kChunk < last;
        const int from = (more ? at0 + kChunk : next_first) + threadIdx.x, to = more ? last : next_last;
        ahead = nothing;
        if ((more || low) && from < to) ahead = __ldg(rec_n + from);
      }
      __syncthreads();
      if (active) {
        uint4 y[4];
        auto fetch = [&](int k) {
          const uint4 s = *reinterpret_cast<const uint4*>(at + k * 16 + (lane >> 3) * 4);
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = line16(yb + word(s, i));
        };
        fetch(0);
#pragma unroll 1
        for (int k = 0; k < steps; ++k) {
          unsigned b[4], ch[4], cl[4], a[4][4];
          ldsm4(b, b_at + k * 512);
          ldsm4t(ch, h_at + k * 512);
          ldsm4t(cl, l_at + k * 512);
          // samples 4 q + i of a half of the channels each -> two channels of the lane's k-slots, the samples 4 t + i
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const unsigned m0 = movmatrix_trans(word(y[0], j)), m1 = movmatrix_trans(word(y[1], j));
            const unsigned m2 = movmatrix_trans(word(y[2], j)), m3 = movmatrix_trans(word(y[3], j));
            a[j][0] = __byte_perm(m0, m1, 0x5410), a[j][1] = __byte_perm(m0, m1, 0x7632);
            a[j][2] = __byte_perm(m2, m3, 0x5410), a[j][3] = __byte_perm(m2, m3, 0x7632);
          }
          if (k + 1 < steps) fetch(k + 1);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            unsigned k0[2], k1[2];
            mul16h(k0, wa[j], b[0], b[1]);
            mul16h(k1, wa[j], b[2], b[3]);
            a[j][0] = hmul2u(k0[0], a[j][0]);
            a[j][1] = hmul2u(k0[1], a[j][1]);
            a[j][2] = hmul2u(k1[0], a[j][2]);
            a[j][3] = hmul2u(k1[1], a[j][3]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (up) mad16(acc[0][j], a[j][0], a[j][1], a[j][2], a[j][3], cl[0], cl[1]);
            if (low) mad16(acc[1][j], a[j][0], a[j][1], a[j][2], a[j][3], cl[2], cl[3]);
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (up) mad16(acc[0][j], a[j][0], a[j][1], a[j][2], a[j][3], ch[0], ch[1]);
            if (low) mad16(acc[1][j], a[j][0], a[j][1], a[j][2], a[j][3], ch[2], ch[3]);
          }
        }
      }
    }
    if (up && active) {
      const int col = w0 + 2 * t;
      bool all = true;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = c0 + 8 * (gq >> 1) + 2 * j + (gq & 1) + 32 * h;
          if (c < g.C && col < g.W) {
            const float v0 = acc[0][j][2 * h], v1 = acc[0][j][2 * h + 1];
            all &= fabsf(v0) < INFINITY && fabsf(v1) < INFINITY;
            __half* o = dx + ((size_t)n * g.C + c) * g.HW + (size_t)h0 * g.W + col;
            if (pairs) {
              *reinterpret_cast<unsigned*>(o) = pack2(v0, v1);
            } else {
              o[0] = __float2half_rn(v0);
              if (col + 1 < g.W) o[1] = __float2half_rn(v1);
            }
          }
        }
      if (__any_sync(0xffffffffu, !all)) {
        unsigned wanted = 0;  // the lane's channels there: c0 + 2 lane, + 1
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const unsigned b = __ballot_sync(0xffffffffu, !(fabsf(acc[0][j][2 * h]) < INFINITY && fabsf(acc[0][j][2 * h + 1]) < INFINITY));
            if ((lane & 3) == j && (lane >> 4) == h) wanted = b >> (lane & 12) * 2 & 0xffu;
          }
        __syncwarp();  // the stores above come first
        gather_row_alone(rec_n, st_n, dyt, w, dx, lg, n, c0 + 2 * lane, h0, w0, wanted);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[0][j][k] = acc[1][j][k], acc[1][j][k] = 0.f;
  }
}

// ------------------------------------------------------------------ host side
size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

bool lines_shape(const Geom& g) {
  if (g.kH != 3 || g.kW != 3 || g.dH != 1 || g.dW != 1 || g.pH != 1 || g.pW != 1) return false;
  if (g.sH != g.sW || (g.sH != 1 && g.sH != 2)) return false;
  if (g.G != 1 || g.scH > 4 || g.scW > 4 || (g.C & 15)) return false;
  const long long lines = (long long)(g.H + 2) * (g.W + 2) * g.N + g.W + 2;  // at least those of dy
  // lines are addressed with 32 bits of bytes, elements of y with 32 bits, the sort's numbers with 27 and 31
  return g.N <= 65535 && g.C < 64 * 30000 && lines * kLine < 0xf0000000LL && (long long)g.N * g.C * g.P < 0xf0000000LL && g.P < (1 << 27) && (long long)g.N * g.P < 0x3fffffffLL &&
         (long long)g.N * g.P * 18 < 0xf0000000LL;
}

struct LinePlan {
  LineGeom lg;
  CoordPlan c;
  GatherPlan gt;
  int share;
  size_t xt, dyt, starts, recs, sums, bank, bytes, sort_smem;
};

void line_plan(const Geom& g, LinePlan& p) {
  LineGeom& lg = p.lg;
  lg.g = g;
  lg.P = make_div(g.P), lg.strip = make_div(kStrip * g.Ho), lg.last = make_div(g.Wo % kStrip ? g.Wo % kStrip : 1), lg.Wo = make_div(g.Wo), lg.W = make_div(g.W);
  lg.units = (g.C + 63) / 64;
  lg.xs = (g.H + 2) * (g.W + 2);
  lg.xu = ((size_t)g.N * lg.xs + g.W + 2) * kLine;
  lg.yu = ((size_t)g.N * g.P + 1) * kLine;
  const int sms = device_sm_count();
  CoordPlan& c = p.c;
  c.units = lg.units;
  c.sets = (c.units + 3) / 4;
  c.upb = (c.units + c.sets - 1) / c.sets;
  c.streams = 4 / c.upb;
  const int npx = 16 * c.streams;
  const long long total = (long long)g.N * g.P;
  c.tiles = (int)((total + npx - 1) / npx);
  int blocks = 3 * sms / c.sets;
  if (blocks < 1) blocks = 1;
  if (blocks > c.tiles) blocks = c.tiles;
  // runs of equal length up to one; short ones take the fewest blocks that are no slower, each lays down bank sums (64 x 256 of 56 x 56, runs of 28 and 29
  // instead of 29: 1341 -> 1324 us; 128 x 160 of 8 x 7, runs of 1 and 2 instead of 2: 99.8 -> 102.4)
  const int run = (c.tiles + blocks - 1) / blocks;
  c.blocks = run >= 8 ? blocks : (c.tiles + run - 1) / run;
  const int warps = c.upb * c.streams;
  c.smem = (size_t)kLineTaps * npx * 76 + npx * 12 + (size_t)c.upb * 2048 + (size_t)warps * (kLineTaps * 160 + kGridCells * kGridPitch) * 4;
  const size_t red = (size_t)warps * 1024 * 4;
  if (c.smem < red) c.smem = red;
  GatherPlan& t = p.gt;
  t.windows = (g.W + 7) / 8;
  const int units = lg.units;
  t.sets = (units + 3) / 4;
  t.warps = (units + t.sets - 1) / t.sets;
  t.bins = (g.H + 1) * (g.W + 1);
  // rows of a band: a row of cells more than rows, and about one more for what a block does besides; 16 warps on an SM
  long long best = -1;
  const long long slots = (long long)sms * (16 / t.warps);
  for (int bands = 1; bands <= g.H; ++bands) {
    const int R = (g.H + bands - 1) / bands;
    const long long nb = (long long)g.N * t.windows * ((g.H + R - 1) / R) * t.sets, cost = (nb + slots - 1) / slots * (R + 2);
    if (best < 0 || cost < best) best = cost, t.R = R, t.bands = (g.H + R - 1) / R;
  }
  p.share = (kLineTaps * g.P + kSortBlocks - 1) / kSortBlocks;
  p.sort_smem = ((size_t)2 * t.bins + 1 + p.share) * 4;
  p.xt = round256(lg.units * lg.xu);
  p.dyt = round256(lg.units * lg.yu);
  p.starts = round256((size_t)g.N * (t.bins + 1) * 4);
  p.recs = round256((size_t)total * kLineTaps * 16);
  p.sums = c.sets > 1 ? round256((size_t)c.sets * kLineTaps * 4 * total * 4) : 0;
  p.bank = round256((size_t)c.blocks * g.C * g.cells * 4);
  p.bytes = p.xt + p.dyt + p.starts + p.recs + p.sums + p.bank;
}

// lines are read and written 16 bytes at a time; the kernels without them take scratch at any word
bool lines_fit(const void* ws) { return (reinterpret_cast<uintptr_t>(ws) & 15) == 0; }

int to_lines(const __half* x, __half* xt, const __half* dy, __half* dyt, const LineGeom& lg, cudaStream_t s) {
  const Geom& g = lg.g;
  auto job = [&](const __half* src, __half* dst, int P) { return LineJob{src, dst, P, (P & 7) == 0 && ptr_mode(src) == 2}; };
  const LineJob jx = job(x, xt, g.HW), jy = job(dy, dyt, g.P);
  const int most = x && g.HW > (dy ? g.P : 0) ? g.HW : g.P;
  lines_kernel<<<dim3((most + 63) / 64, lg.units * ((x != nullptr) + (dy != nullptr)) + 1, g.N), 256, 0, s>>>(jx, jy, lg);
  return check_launch();
}

}  // namespace

bool deform_lines_shape(const Geom& g) { return lines_shape(g); }

size_t deform_lines_forward_workspace(const Geom& g) {
  if (!lines_shape(g)) return 0;
  LinePlan p;
  line_plan(g, p);
  return p.xt;
}

int deform_lines_forward(const __half* x, const __half* off, const __half* rot, const __half* w, __half* y, const Geom& g, void* ws,
                         size_t ws_bytes, cudaStream_t s) {
  if (!lines_shape(g)) return DK_ERR_UNSUPPORTED;
  LinePlan p;
  line_plan(g, p);
  if (ws == nullptr || ws_bytes < p.xt || !lines_fit(ws)) return DK_ERR_UNSUPPORTED;
  __half* xt = reinterpret_cast<__half*>(ws);
  if (int rc = to_lines(x, xt, nullptr, nullptr, p.lg, s)) return rc;
  const int units = p.lg.units, tiles = (int)(((long long)g.N * g.P + kFwdPixels - 1) / kFwdPixels);
  int split = 1;
  while (split < units && (long long)tiles * split < 3 * device_sm_count()) ++split;
  if (int rc = enable_smem(line_forward_kernel, sizeof(FwdSmem))) return rc;
  // neighbouring pixels that are stored together
  const int run = (g.Wo & 3) == 0 && (reinterpret_cast<uintptr_t>(y) & 7) == 0 ? 4 : (g.Wo & 1) == 0 && ptr_mode(y) >= 1 ? 2 : 1;
  line_forward_kernel<<<dim3(tiles, split), 128, sizeof(FwdSmem), s>>>(xt, off, rot, w, y, p.lg, run);
  return check_launch();
}

size_t deform_lines_backward_workspace(const Geom& g) {
  if (!lines_shape(g)) return 0;
  LinePlan p;
  line_plan(g, p);
  return p.bytes;
}

// the wanted gradients (null: not wanted)
int deform_lines_backward(const __half* dy, const __half* x, const __half* off, const __half* rot, const __half* w, __half* dx, __half* doff,
                          __half* drot, __half* dw, const Geom& g, void* ws, size_t ws_bytes, cudaStream_t s) {
  if (!lines_shape(g)) return DK_ERR_UNSUPPORTED;
  LinePlan p;
  line_plan(g, p);
  if (p.sort_smem > 200 * 1024 || ws == nullptr || ws_bytes < p.bytes || !lines_fit(ws)) return DK_ERR_UNSUPPORTED;
  const bool coords = doff || drot || dw;
  char* at = reinterpret_cast<char*>(ws);
  auto take = [&](size_t bytes) {
    char* r = at;
    at += bytes;
    return r;
  };
  __half* xt = reinterpret_cast<__half*>(take(p.xt));
  __half* dyt = reinterpret_cast<__half*>(take(p.dyt));
  int* starts = reinterpret_cast<int*>(take(p.starts));
  float4* recs = reinterpret_cast<float4*>(take(p.recs));
  float* sums = reinterpret_cast<float*>(take(p.sums));
  float* bank = reinterpret_cast<float*>(take(p.bank));
  if (int rc = to_lines(coords ? x : nullptr, xt, dy, dyt, p.lg, s)) return rc;
  if (dx) {
    if (int rc = enable_smem(line_sort_kernel, p.sort_smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g.N * kSortBlocks);
    cfg.blockDim = dim3(kSortThreads);
    cfg.dynamicSmemBytes = p.sort_smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = kSortBlocks, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, line_sort_kernel, off, rot, starts, recs, p.lg, p.gt.bins, p.share);
    if (e != cudaSuccess) {
      set_last_cuda_error(e);
      return DK_ERR_CUDA;
    }
    if (int rc = check_launch()) return rc;
    const bool pairs = (g.W & 1) == 0 && ptr_mode(dx) >= 1;
    line_gather_kernel<<<dim3((unsigned)(g.N * p.gt.windows * p.gt.bands), p.gt.sets), 32 * p.gt.warps, 0, s>>>(dyt, starts, recs, w, dx, p.lg,
                                                                                                            p.gt, pairs);
    if (int rc = check_launch()) return rc;
  }
  if (coords) {
    auto kern = rot ? line_coords_kernel<true> : line_coords_kernel<false>;
    if (int rc = enable_smem(kern, p.c.smem)) return rc;
    kern<<<dim3(p.c.blocks, p.c.sets), 32 * p.c.upb * p.c.streams, p.c.smem, s>>>(dyt, xt, off, rot, w, doff, drot, sums, dw ? bank : nullptr, p.lg, p.c);
    if (int rc = check_launch()) return rc;
    const int NK = rot ? 4 : 2;
    if (p.c.sets > 1 && (doff || drot)) {
      line_coord_sums_kernel<<<dim3((unsigned)((g.N * g.P + 255) / 256), kLineTaps * NK), 256, 0, s>>>(sums, doff, drot, p.lg, p.c.sets, NK);
      if (int rc = check_launch()) return rc;
    }
    if (dw) return reduce_bank<__half>(bank, dw, g.C * g.cells, p.c.blocks, s);
  }
  return DK_OK;
}

}  // namespace dk
