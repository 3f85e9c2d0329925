// Local deformable kernel on the fifth-generation tensor cores (tcgen05 + TMEM), fp16 and fp32 storage.
//
// The resampled kernel is a contraction with hat products, K[c, p, tap] = sum_cell W[c, cell] * beta[p, tap, cell]
// (dk_local_mma.cu).  Here the channels are the 128 rows of a tcgen05.mma: W stays in TMEM, the hat products of a step's 64
// pixels and the three taps of one kernel row are the 192 columns in shared memory, and the result is read back one channel
// per lane.  A lane then owns 8 consecutive pixels of ONE channel: its source window is one 16-byte shared-memory load per
// row plus the two edge values, shared by nine taps.
//
// With mma.sync fragments (8 channels x 2 pixels per lane) the same step executes 166 warp-instructions per 128 outputs: 27
// loads of 4 bytes, 45 for the hat products that every warp builds for itself, 9 mma, 36 multiply-adds, 30 for indices and
// waits.  Here hat products are built once per block by warps of their own, the mma are issued by one warp, and a consumer
// warp is left with 72 multiply-adds, 15 loads and the stores per 256 outputs.
//
// fp16: K leaves the tensor cores rounded to fp16 (relative 2^-11, like the tensors themselves) and meets x in the
// mixed-precision multiply-add (exact product, fp32 sum), as in dk_local_ring.cu and dk_local_mma.cu, whose calls these are.  Calls
// that those do not take (channels no multiple of 16) keep K in fp32: W is exact in one piece, the hat products take two.
// fp32: W is split into three fp16 pieces and the hat products into two, scaled by powers of two (W per channel, its last piece
// by 2^15 more; the hat products by 2^15).  The pieces hold W to 24 bits down to 2^-30 of the channel's largest value, below that
// to 2^-55 of it, and the hat products to 23 bits down to 2^-15, below that to 2^-40.  Five products, the small ones first: the
// tensor cores truncate each sum, and only the last one is at full size (kUnbias).  Error against fp64, 2-norm, N(0, 1) data, 56 x 56:
// 1.36e-7, most of it the rounding of the coordinates (four gathered fp32 products and additions before: 1.40e-7; two pieces of W, large
// products first: 1.94e-7).
//
// A block walks through a contiguous range of 8-pixel segments of the destination rows (sample, row, column octet, in
// memory order) for up to CG channels; 8 segments are a step.  Roles:
//   16 consumer warps  team j (4 warps, one per quarter of the TMEM lanes) takes segments 2j, 2j + 1 of every step: waits
//                      for the accumulators of one kernel row, multiplies, leaves the results in shared memory
//   1 MMA warp         issues the tcgen05.mma, two sets of accumulators
//   1 or 3 loaders     source rows through a ring of row slots: TMA where rows are multiples of 16 bytes (out-of-range
//                      elements arrive as zeros = the convolution padding), else cp.async pieces or elements, 3 warps
//   6 or 4 hat warps   lane = destination pixel: offsets, taps of 16 hat products each, written as the B operand
//   4 store warps      results of a step from shared memory, consecutive pixels on consecutive lanes (written straight from
//                      the consumers' registers, one channel per lane, every store touches 32 lines)
// Every hand-over is an mbarrier used once per step (or per set of accumulators) by the same warps, in order.
#include <atomic>
#include <cstring>
#include <type_traits>

#include "dk_tc.cuh"

namespace dk {

using namespace ring;
using namespace tc;
using mma::hat;

namespace {

__device__ int g_tc_error;  // set when a bounded wait ran out

constexpr int kTeams = 4;
constexpr int kConsumers = 16;
constexpr int kHelpers = 12;  // MMA, loaders, hat products, stores
constexpr int kThreads = 32 * (kConsumers + kHelpers);
// Registers per thread: 72 at launch, then more for the four consumer warpgroups than for the three of the helpers.  Consumers of
// fp16 kernel values hold two items; of fp32 values (FULL) one, and with one loader the hat products get what that leaves (with
// three, 88 / 48 is the faster split: 32 x 384 of 14 x 14 47 -> 45 us).
constexpr int kRegsLaunch = 72;
template <bool FULL, int NL>
__host__ __device__ constexpr int consumer_regs() {
  return FULL && NL == 1 ? 80 : 88;
}
template <bool FULL, int NL>
__host__ __device__ constexpr int helper_regs() {
  return FULL && NL == 1 ? 56 : 48;
}
static_assert(kConsumers * consumer_regs<true, 1>() + kHelpers * helper_regs<true, 1>() <= (kConsumers + kHelpers) * kRegsLaunch &&
                  kConsumers * consumer_regs<false, 1>() + kHelpers * helper_regs<false, 1>() <= (kConsumers + kHelpers) * kRegsLaunch,
              "register shares");
constexpr int kLoaders = 3;                         // warps that fetch rows without TMA
constexpr int kStepSegs = 8;
constexpr int kSlotCols = 48;                       // three taps x 16 pixels
constexpr int kSetCols = kTeams * kSlotCols;        // one set of accumulators
constexpr int kBankCol = 2 * kSetCols;              // the bank behind the two sets
constexpr int kDepth = 4;                           // steps in flight, as seen by the row ring
constexpr int kPairRow = 6 * 256;                   // hat products of two segments and one kernel row: 48 columns x 32 bytes
constexpr int kPiece = 3 * kTeams * kPairRow;       // of a step: [kernel row][pair][segment, tap: 8 columns][two halves of the cells]
constexpr int kMinSmem = 120 * 1024;                // one block per SM: it takes all of TMEM

// Hat products: two buffers, each with two or three warps of its own, so that a warp sees every reuse of its buffer (a barrier's phase
// can only be told from the one before it).  Two warps take half of a step's pixels each; three, where there is one loader, a kernel
// row each (three buffers with two warps: fp16, 128 x 96 of 112 x 112 285 / 328 us against 268 / 264; two with two: fp32, 64 x 144 of
// 56 x 56 178 / 178 against 150 / 148).
constexpr int kBufs = 2;
constexpr int kBars = 2 * kDepth + 2 * kBufs + 6;
__host__ __device__ constexpr int warps_per_buffer(int loaders) { return loaders == 1 ? 3 : 2; }

template <typename T>
__host__ __device__ constexpr int bank_piece_count() {
  return sizeof(T) == 2 ? 1 : 3;
}

enum Mode { kFwd1 = 0, kFwd2 = 1, kData1 = 2, kData2 = 3 };  // forward, grad-input; stride 1, 2

struct ConvParams {
  int N, C;
  int Hs, Ws;  // source plane
  int Hg, Wg;  // plane of the segments: destination (kData2: grad-output)
  int Hd, Wd;  // destination plane
  int Ho, Wo;  // plane of the offsets
  int nseg;    // segments per row
  int L;       // stream rows per sample
  int R;       // slots in the row ring
  int pitch;   // bytes per channel row in a slot: an odd multiple of 16
  int CG;      // channels per block
  int box_c;   // channels per TMA box
  int full;    // quads of 32-channel groups
  int rest;    // groups beyond them
  int segs;    // N * Hg * nseg
  int steps_per_cta;
  unsigned magic_seg, magic_row;  // ceil(2^32 / nseg), ceil(2^32 / Hg)
  int scW, cells;
  float uh0, uw0;
  int store;  // bytes per store of a result row: 16, 4 or 2
};

struct SegPos {
  int n, g, s;
};
__device__ __forceinline__ SegPos seg_pos(int b, const ConvParams& p) {
  SegPos r;
  const int row = p.nseg == 1 ? b : (int)__umulhi((unsigned)b, p.magic_seg);
  r.s = b - row * p.nseg;
  r.n = p.Hg == 1 ? row : (int)__umulhi((unsigned)row, p.magic_row);
  r.g = row - r.n * p.Hg;
  return r;
}

template <int MODE> struct Walk {
  static constexpr int S = MODE == kFwd2 ? 2 : 1;        // stream rows per segment row
  static constexpr int rows = MODE == kData2 ? 2 : 3;    // stream rows a segment reads
  static constexpr int first = MODE == kData2 ? 0 : -1;  // source row of a sample's first stream row
  static constexpr int xs = MODE == kFwd2 ? 2 : 1;       // source columns per segment column
};

// ------------------------------------------------------------------ consumers' operands
// One item = one segment (8 pixels) and one kernel row of the lane's channel: 24 kernel values (tap-major; pixels p and
// p + 4 in adjacent columns) and the source window.
template <typename T, int MODE, bool FULL> struct Item;

template <int MODE> struct Item<__half, MODE, false> {
  static constexpr int NW = MODE == kFwd2 ? 8 : 4;
  unsigned k[12];        // fp16 pairs (p, p + 4)
  unsigned w[NW];        // source columns 0 .. 7 (15) of the segment
  unsigned left, right;  // columns -1 and 8
  __device__ __forceinline__ void load(unsigned tmem, const char* row) {
    ld24(k, tmem);
    const __half* x = reinterpret_cast<const __half*>(row);
#pragma unroll
    for (int i = 0; i < NW / 4; ++i) {
      const uint4 q = *reinterpret_cast<const uint4*>(x + 8 * i);
      w[4 * i] = q.x, w[4 * i + 1] = q.y, w[4 * i + 2] = q.z, w[4 * i + 3] = q.w;
    }
    if (MODE != kData2) left = *reinterpret_cast<const unsigned short*>(x - 1);
    if (MODE != kFwd2) right = *reinterpret_cast<const unsigned short*>(x + 8);
  }
  // a += source column I * half KH of kk
  template <int I, int KH> __device__ __forceinline__ void mac(float& a, unsigned kk) const {
    if constexpr (I < 0) mma::fma_hh<0, KH>(a, left, kk);
    else if constexpr (I >= 2 * NW) mma::fma_hh<0, KH>(a, right, kk);
    else mma::fma_hh<I & 1, KH>(a, w[I / 2], kk);
  }
  template <int LO, int HI, int Q> __device__ __forceinline__ void tap(float& a, float& b) const {
    mac<LO, 0>(a, k[Q]);
    mac<HI, 1>(b, k[Q]);
  }
};

template <typename T, int MODE> struct Item<T, MODE, true> {
  static constexpr int NW = MODE == kFwd2 ? 16 : 8;
  unsigned k[24];
  float w[NW], left, right;
  __device__ __forceinline__ void load(unsigned tmem, const char* row) {
    ld24(k, tmem);
    const T* x = reinterpret_cast<const T*>(row);
    if constexpr (sizeof(T) == 4) {
#pragma unroll
      for (int i = 0; i < NW / 4; ++i) {
        const float4 q = *reinterpret_cast<const float4*>(x + 4 * i);
        w[4 * i] = q.x, w[4 * i + 1] = q.y, w[4 * i + 2] = q.z, w[4 * i + 3] = q.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < NW / 8; ++i) {
        const uint4 q = *reinterpret_cast<const uint4*>(x + 8 * i);
        const unsigned h[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) w[8 * i + 2 * j] = mma::lo2f(h[j]), w[8 * i + 2 * j + 1] = mma::hi2f(h[j]);
      }
    }
    if (MODE != kData2) left = static_cast<float>(x[-1]);
    if (MODE != kFwd2) right = static_cast<float>(x[8]);
  }
  template <int I> __device__ __forceinline__ float at() const {
    if constexpr (I < 0) return left;
    else if constexpr (I >= NW) return right;
    else return w[I];
  }
  template <int LO, int HI, int Q> __device__ __forceinline__ void tap(float& a, float& b) const {
    a = fmaf(at<LO>(), __uint_as_float(k[2 * Q]), a);
    b = fmaf(at<HI>(), __uint_as_float(k[2 * Q + 1]), b);
  }
};

// acc += window * kernel row.  Source column of tap t and pixel p: p xs + t - 1 (kData2: p, and p + 1 for the third tap);
// kData2 keeps the even destination columns in acc[0..8) and the odd ones in acc[8..16).
template <typename T, int MODE, bool FULL, int N>
__device__ __forceinline__ void multiply(float (&acc)[N], const Item<T, MODE, FULL>& it) {
  constexpr int XS = Walk<MODE>::xs;
  constexpr bool D = MODE == kData2;
#define DK_TAP(t, p)                                                                                             \
  it.template tap<D ? p + (t == 2) : p * XS + t - 1, D ? p + 4 + (t == 2) : (p + 4) * XS + t - 1, t * 4 + p>( \
      acc[(D && t ? 8 : 0) + p], acc[(D && t ? 8 : 0) + p + 4]);
#define DK_TAPS(t) DK_TAP(t, 0) DK_TAP(t, 1) DK_TAP(t, 2) DK_TAP(t, 3)
  DK_TAPS(0) DK_TAPS(1) DK_TAPS(2)
#undef DK_TAPS
#undef DK_TAP
}

// `count` consecutive values v[0..count) of one channel row to global memory (kData2)
template <typename T, int NV>
__device__ __forceinline__ void store_row(T* __restrict__ d, const float (&v)[NV], int count, bool vec) {
  constexpr int V = 16 / sizeof(T);
#pragma unroll
  for (int i = 0; i < NV; i += V) {
    if (vec && count >= i + V) {
      if constexpr (sizeof(T) == 2)
        *reinterpret_cast<uint4*>(d + i) = make_uint4(mma::pack2(v[i], v[i + 1]), mma::pack2(v[i + 2], v[i + 3]),
                                                      mma::pack2(v[i + 4], v[i + 5]), mma::pack2(v[i + 6], v[i + 7]));
      else
        *reinterpret_cast<float4*>(d + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
    } else {
#pragma unroll
      for (int k = i; k < i + V; ++k)
        if (k < count) st<T, float>(d + k, v[k]);
    }
  }
}

// ------------------------------------------------------------------ bank in TMEM
// A tiles: `full` quads of groups in order, then four variants of the remaining 1 to 3 groups.  Variant v puts them on the
// quarters of the lanes (= consumer warps) that pair (v - step) mod 4 of a step uses, so that over four pairs every quarter
// gets the same number of groups.  Index of the remaining group on quarter q, -1: none.
__device__ __forceinline__ int rest_index(int rest, int v, int q) {
  if (rest == 1) return q == v ? 0 : -1;
  if (rest == 2) return (q >> 1) == (v & 1) ? (q & 1) : -1;
  return q == v ? -1 : q - (q > v);
}

// The tensor cores truncate a sum to 24 bits: 1/2 of the last place too low on average, 2^-24 / 1.44 of the value over a binade.
// Banks are larger by that much; the truncation takes it off again (a sum of one term comes out exact: less than one place was added).
constexpr float kUnbias = 4.1e-8f;

// The 16 cells of one channel into the columns at `a` as fp16 pieces of 8 columns (two cells each): the values, or for fp32 their
// upper and lower parts and, scaled by 2^15, what those leave.  Returns what undoes the scaling of fp32 banks and of the hat
// products they meet; `finite` is cleared where a value is not.
template <typename T>
__device__ __forceinline__ float bank_to_tmem(unsigned a, const T* __restrict__ w, int cells, bool ok, bool& finite) {
  float v[16], inv = 1.f;
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    v[i] = ok && i < cells ? ld<float>(w + i) : 0.f;
    finite &= fabsf(v[i]) < INFINITY;
  }
  if constexpr (std::is_same<T, float>::value) {
    float top = 0.f;
#pragma unroll
    for (int i = 0; i < 16; ++i) top = fmaxf(top, fabsf(v[i]));
    int e = 0;
    if (top > 0.f && top < INFINITY) frexpf(top, &e);
    const int shift = min(15 - e, 111);  // largest magnitude in [2^14, 2^15), or less where `inv` would be subnormal
    const float sc = ldexpf(1.f, shift);
    inv = ldexpf(1.f, -15 - shift);
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] *= sc;
  }
  unsigned top_part[8];
#pragma unroll
  for (int piece = 0; piece < bank_piece_count<T>(); ++piece) {
    unsigned r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (piece == 2) {
        v[2 * i] = 32768.f * fmaf(kUnbias, mma::lo2f(top_part[i]), v[2 * i]);
        v[2 * i + 1] = 32768.f * fmaf(kUnbias, mma::hi2f(top_part[i]), v[2 * i + 1]);
      }
      r[i] = mma::pack2(v[2 * i], v[2 * i + 1]);
      if (piece == 0) top_part[i] = r[i];
      v[2 * i] -= mma::lo2f(r[i]), v[2 * i + 1] -= mma::hi2f(r[i]);
    }
    st8(a + 8 * piece, r);
  }
  return inv;
}

// ------------------------------------------------------------------ hat products
// Tap column t of kernel row v of segment pixel (g, x): the offsets' pixel (qh, qw) and the tap (fh, fw).
template <int MODE>
__device__ __forceinline__ void tap_of(int v, int t, int g, int x, int& qh, int& qw, int& fh, int& fw) {
  if (MODE == kFwd1 || MODE == kFwd2) {
    qh = g, qw = x, fh = v, fw = t;
  } else if (MODE == kData1) {
    qh = g + v - 1, qw = x + t - 1, fh = 2 - v, fw = 2 - t;
  } else {  // 2 x 2 patch: (0, tap 1) -> even row; (0, tap 2), (1, tap 0) -> odd row; columns alike
    qh = g + (v == 2), qw = x + (t == 2), fh = v == 0 ? 1 : (v == 1 ? 2 : 0), fw = t == 0 ? 1 : (t == 1 ? 2 : 0);
  }
}

// 16 hat products of one tap: cells (2i, 2i + 1) in hi[i].  SPLIT (fp32): scaled by 2^15, and what hi leaves of the unrounded
// products in lo[i].  Products in packed pairs only where nothing else is done with them: before the subtraction the pairs have to be
// moved into place (forward of N = 64, C = 144, 56 x 56 170 us, 156 without).
template <bool SC44, bool SPLIT>
__device__ __forceinline__ void hat_products(unsigned (&hi)[8], unsigned (&lo)[8], float u, float v, bool ok, int scW, int cells) {
  constexpr float kScale = SPLIT ? 32768.f : 1.f;
  if constexpr (SC44) {
    float hv[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) hv[a] = hat(v - (float)a);
    if constexpr (SPLIT) {
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float hu = ok ? kScale * hat(u - (float)a) : 0.f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float h0 = hv[2 * k], h1 = hv[2 * k + 1];
          const unsigned h = hi[2 * a + k] = mma::pack2(hu * h0, hu * h1);
          lo[2 * a + k] = mma::pack2(fmaf(hu, h0, -mma::lo2f(h)), fmaf(hu, h1, -mma::hi2f(h)));
        }
      }
    } else {
      float hu[4], b[16];
#pragma unroll
      for (int a = 0; a < 4; ++a) hu[a] = ok ? hat(u - (float)a) : 0.f;
      const unsigned long long v01 = pair(hv[0], hv[1]), v23 = pair(hv[2], hv[3]);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const unsigned long long uu = pair(hu[a], hu[a]);
        const float2 r = unpair(mul2(uu, v01)), q = unpair(mul2(uu, v23));
        b[4 * a] = r.x, b[4 * a + 1] = r.y, b[4 * a + 2] = q.x, b[4 * a + 3] = q.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) hi[i] = mma::pack2(b[2 * i], b[2 * i + 1]);
    }
  } else {
    int a = 0, c = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float hu[2], hv[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        hu[k] = ok && 2 * i + k < cells ? kScale * hat(u - (float)a) : 0.f;
        hv[k] = hat(v - (float)c);
        if (++c == scW) c = 0, ++a;
      }
      hi[i] = mma::pack2(hu[0] * hv[0], hu[1] * hv[1]);
      if (SPLIT) lo[i] = mma::pack2(fmaf(hu[0], hv[0], -mma::lo2f(hi[i])), fmaf(hu[1], hv[1], -mma::hi2f(hi[i])));
    }
  }
}

__device__ __forceinline__ void sts16(unsigned a, unsigned x, unsigned y, unsigned z, unsigned w) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// What a beta warp does in a step, WPB warps sharing it: 18 / WPB pieces of 32 pixels (lane = pixel: segment lane / 8, column lane % 8)
// and one tap.  Offsets as they lie in memory, (vertical, horizontal); absent ones read as zero.
template <typename T, int WPB> struct Offsets {
  static constexpr int kPieces = 18 / WPB;
  T r[kPieces][2];
  unsigned ok;  // taps whose offsets exist
};
template <int WPB>
__device__ __forceinline__ void piece_of(int i, int w, int& half, int& v, int& t) {
  half = WPB == 3 ? i / 3 : w, v = WPB == 3 ? w : i / 3, t = i % 3;
}

template <typename T, int MODE, int WPB>
__device__ __forceinline__ void fetch_offsets(Offsets<T, WPB>& o, const T* __restrict__ rot, int seg, int hi_seg, const ConvParams& p,
                                              int w, int lane) {
  const int P = p.Ho * p.Wo;
  SegPos sp;
  int x = 0;
  const T* rn = rot;
  bool live = false;
  o.ok = 0;
#pragma unroll
  for (int i = 0; i < Offsets<T, WPB>::kPieces; ++i) {
    int half, v, t, qh, qw, fh, fw;
    piece_of<WPB>(i, w, half, v, t);
    if (i == 0 || (WPB == 3 && i == 3)) {
      const int b = seg + half * 4 + (lane >> 3);
      sp = seg_pos(min(b, hi_seg - 1), p);
      x = sp.s * 8 + (lane & 7);
      live = b < hi_seg && x < p.Wg;
      rn = rot + (size_t)sp.n * 18 * P;
    }
    tap_of<MODE>(v, t, sp.g, x, qh, qw, fh, fw);
    const bool ok = live && qh >= 0 && qh < p.Ho && qw >= 0 && qw < p.Wo;
    o.ok |= (unsigned)ok << i;
    const T* a = rn + ((fh * 3 + fw) * 2) * P + qh * p.Wo + qw;
    o.r[i][0] = ok ? __ldg(a) : T(0.f);
    o.r[i][1] = ok ? __ldg(a + P) : T(0.f);
  }
}

template <typename T, int MODE, bool SC44, bool SPLIT, int WPB>
__device__ __forceinline__ void write_hats(unsigned buf, const Offsets<T, WPB>& o, const ConvParams& p, int w, int lane) {
  const int sl = lane >> 3, px = lane & 7;
  // row of this pixel inside its 8-row core matrix: pixels p and p + 4 are neighbours
  const unsigned dst = buf + (sl >> 1) * kPairRow + (sl & 1) * (3 * 256) + ((px & 3) * 2 + (px >> 2)) * 16;
#pragma unroll
  for (int i = 0; i < Offsets<T, WPB>::kPieces; ++i) {
    int half, v, t, qh, qw, fh, fw;
    piece_of<WPB>(i, w, half, v, t);
    tap_of<MODE>(v, t, 0, 0, qh, qw, fh, fw);
    const float ru = static_cast<float>(o.r[i][0]), rv = static_cast<float>(o.r[i][1]);
    // fp32: one rounding, tap + (scope - kernel) / 2 is exact; with fp16 offsets the reference's order is, too
    const float u0 = SPLIT ? ru + ((float)fh + p.uh0) : ((float)fh + ru) + p.uh0, v0 = SPLIT ? rv + ((float)fw + p.uw0) : ((float)fw + rv) + p.uw0;
    unsigned hi[8], lo[8];
    hat_products<SC44, SPLIT>(hi, lo, u0, v0, (o.ok >> i) & 1, p.scW, p.cells);
    const unsigned a = dst + v * (kTeams * kPairRow) + half * (2 * kPairRow) + t * 256;
    sts16(a, hi[0], hi[1], hi[2], hi[3]);
    sts16(a + 128, hi[4], hi[5], hi[6], hi[7]);
    if (SPLIT) {
      sts16(a + kPiece, lo[0], lo[1], lo[2], lo[3]);
      sts16(a + kPiece + 128, lo[4], lo[5], lo[6], lo[7]);
    }
  }
}

// ------------------------------------------------------------------ source rows without TMA
// Loader warp lw of NL: source row `row` of channels c0 .. c0 + cg - 1 of sample n into a slot.
template <typename T, int NL>
__device__ __forceinline__ void copy_row(char* slot, const T* __restrict__ src, int n, int c0, int cg, int row, const ConvParams& p,
                                         int lw, int lane) {
  const int bytes = p.Ws * (int)sizeof(T);
  if (row < 0 || row >= p.Hs) {  // a row of the padding
    for (int c = lw; c < cg; c += NL) {
      uint4* d = reinterpret_cast<uint4*>(slot + (size_t)c * p.pitch);
      for (int i = lane; i < p.pitch / 16; i += 32) d[i] = make_uint4(0, 0, 0, 0);
    }
    return;
  }
  const size_t plane = (size_t)p.Hs * bytes;
  const char* g0 = reinterpret_cast<const char*>(src) + ((size_t)n * p.C + c0) * plane + (size_t)row * bytes;
  char* d0 = slot + 16;
  const unsigned align = (unsigned)(reinterpret_cast<uintptr_t>(src) | (unsigned)bytes);
  const int unit = (align & 7) == 0 ? 8 : ((align & 3) == 0 ? 4 : 2);
  const int per = bytes / unit;  // copies per channel row
  // a lane keeps its piece of the row and walks down the channels, several channels per step where rows are short
  const int chs = per <= 16 ? 32 / per : 1;
  for (int i = lane; i < (per <= 16 ? chs * per : per); i += 32) {
    const int sub = per <= 16 ? i / per : 0, first = lw * chs + sub, step = NL * chs;
    const int pc = i - sub * per;
    const char* g = g0 + (size_t)first * plane + pc * unit;
    char* d = d0 + first * p.pitch + pc * unit;
    const size_t gs = (size_t)step * plane;
    const int ds = step * p.pitch;
    if (unit == 8) {
#pragma unroll 4
      for (int c = first; c < cg; c += step, g += gs, d += ds) cp_async8(d, g);
    } else if (unit == 4) {
#pragma unroll 4
      for (int c = first; c < cg; c += step, g += gs, d += ds) mma::cp_async4(d, g);
    } else {
      for (int c = first; c < cg; c += 8 * step, g += 8 * gs, d += 8 * ds) {  // eight independent loads in flight
        unsigned short v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (c + k * step < cg) v[k] = __ldg(reinterpret_cast<const unsigned short*>(g + k * gs));
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (c + k * step < cg) *reinterpret_cast<unsigned short*>(d + k * ds) = v[k];
      }
    }
  }
}

// ------------------------------------------------------------------ banks with values that are not finite
// Products with a hat of zero would carry such a value to every output of its channel.  A block that finds one among its
// channels' cells gathers the four cells of a sample instead, a lane per output.
template <typename T, int MODE>
__device__ __noinline__ void gather_block(const T* __restrict__ src, const T* __restrict__ rot, const T* __restrict__ bank,
                                          T* __restrict__ dst, const ConvParams& p, int c0, int cg, int lo, int hi) {
  constexpr bool kData = MODE == kData1 || MODE == kData2;
  constexpr int S = MODE == kFwd2 || MODE == kData2 ? 2 : 1, PX = MODE == kData2 ? 32 : 8;  // destination pixels of a segment
  const int scH = p.cells / p.scW, px = (hi - lo) * PX, P = p.Ho * p.Wo;
#pragma unroll 1
  for (int c = c0; c < c0 + cg; ++c) {
    const T* w = bank + (size_t)c * p.cells;
#pragma unroll 1
    for (int i = threadIdx.x; i < px; i += kThreads) {
      const SegPos sp = seg_pos(lo + i / PX, p);
      const int k = i % PX, oh = MODE == kData2 ? 2 * sp.g + (k >> 4) : sp.g, ow = MODE == kData2 ? 16 * sp.s + (k & 15) : 8 * sp.s + k;
      if (oh >= p.Hd || ow >= p.Wd) continue;
      const T* plane = src + ((size_t)sp.n * p.C + c) * p.Hs * p.Ws;
      float acc = 0.f;
#pragma unroll 1
      for (int tap = 0; tap < 9; ++tap) {
        const int fh = tap / 3, fw = tap - fh * 3;
        int sh = kData ? oh + 1 - fh : oh * S - 1 + fh, sw = kData ? ow + 1 - fw : ow * S - 1 + fw;
        if (sh < 0 || sw < 0 || (kData && S == 2 && ((sh | sw) & 1))) continue;
        if (kData && S == 2) sh >>= 1, sw >>= 1;
        if (sh >= p.Hs || sw >= p.Ws) continue;
        const T* r = rot + ((size_t)sp.n * 18 + 2 * tap) * P + (kData ? sh * p.Wo + sw : oh * p.Wo + ow);
        const float u = ld<float>(r) + ((float)fh + p.uh0), v = ld<float>(r + P) + ((float)fw + p.uw0);
        float kv = 0.f;
        if (u > -1.f && v > -1.f && u < (float)scH && v < (float)p.scW) {
          const float fu = floorf(u), fv = floorf(v);
#pragma unroll 1
          for (int q = 0; q < 4; ++q) {
            const int a = (int)fu + (q >> 1), b = (int)fv + (q & 1);
            if (a >= 0 && a < scH && b >= 0 && b < p.scW) kv = fmaf(hat(u - (float)a) * hat(v - (float)b), ld<float>(w + a * p.scW + b), kv);
          }
        }
        acc = fmaf(ld<float>(plane + (size_t)sh * p.Ws + sw), kv, acc);
      }
      st<T, float>(dst + (((size_t)sp.n * p.C + c) * p.Hd + oh) * p.Wd + ow, acc);
    }
  }
}

// ------------------------------------------------------------------ forward and grad-input
// d = bank at a (its pieces 8 columns apart) * hat products at b (kPiece apart), the smallest products first
template <typename T, bool FULL>
__device__ __forceinline__ void products(unsigned d, unsigned a, uint64_t b, unsigned idesc) {
  const uint64_t b_lo = b + (kPiece >> 4);
  if constexpr (sizeof(T) == 4) {
    mma_ts(d, a + 16, b, idesc, false);
    mma_ts_scaled<15>(d, a + 8, b_lo, idesc);
    mma_ts(d, a + 8, b, idesc, true);
    mma_ts(d, a, b_lo, idesc, true);
    mma_ts(d, a, b, idesc, true);
  } else {
    if (FULL) mma_ts(d, a, b_lo, idesc, false);
    mma_ts(d, a, b, idesc, FULL);
  }
}

// staged results: [channel][64 pixels], an odd number of 16-byte units per channel (lanes = channels write 16 bytes each)
template <typename T> __host__ __device__ constexpr int out_pitch() { return kStepSegs * 8 * (int)sizeof(T) + 16; }

struct ConvSmem {  // byte offsets behind the row ring
  unsigned beta, inv, out, segs, bars, total;
};
template <typename T, int MODE, bool FULL>
__host__ __device__ inline ConvSmem conv_smem(unsigned ring_bytes, int groups) {
  ConvSmem m;
  m.beta = (ring_bytes + 32 + 127) & ~127u;  // 32: what the last channel row's right edge may read
  m.inv = m.beta + kBufs * kPiece * (FULL ? 2 : 1);
  m.out = m.inv + (sizeof(T) == 4 ? groups * 128 : 0);
  m.segs = m.out + (MODE == kData2 ? 0 : groups * 32 * out_pitch<T>());
  m.bars = m.segs + kDepth * kStepSegs * 16;
  m.total = m.bars + kBars * 8 + 16;
  return m;
}

// FULL: the kernel values leave the tensor cores as fp32 (fp32 tensors always)
template <typename T, int MODE, bool SC44, int NL, bool FULL>
__device__ __forceinline__ void tc_conv(const CUtensorMap& tm, const T* __restrict__ src, const T* __restrict__ rot,
                                        const T* __restrict__ bank, T* __restrict__ dst, const ConvParams& p) {
  extern __shared__ __align__(1024) char smem[];
  using Wk = Walk<MODE>;
  constexpr bool STAGED = MODE != kData2, SCALED = sizeof(T) == 4;
  constexpr int PIECES = FULL ? 2 : 1, E = sizeof(T), TILE = 8 * bank_piece_count<T>();  // columns of 128 channels' bank
  constexpr int WPB = warps_per_buffer(NL), NB = kBufs * WPB, NS = kHelpers - 1 - NL - NB;
  constexpr int kOutPitch = out_pitch<T>();
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int c0 = blockIdx.y * p.CG, cg = min(p.CG, p.C - c0);
  const int groups = p.full * 4 + p.rest, rounds = p.full + (p.rest ? 1 : 0);
  const unsigned slot_bytes = (unsigned)p.CG * p.pitch, ring_bytes = slot_bytes * p.R;
  const ConvSmem sm = conv_smem<T, MODE, FULL>(ring_bytes, groups);
  const unsigned base = smem_u32(smem);
  const unsigned x_full = base + sm.bars, step_done = x_full + 8 * kDepth, b_full = step_done + 8 * kDepth;
  const unsigned b_free = b_full + 8 * kBufs, t_full = b_free + 8 * kBufs, t_empty = t_full + 16, o_full = t_empty + 16,
                 o_free = o_full + 8;
  float* inv_s = reinterpret_cast<float*>(smem + sm.inv);
  volatile int* tail = reinterpret_cast<volatile int*>(smem + sm.bars + kBars * 8);  // TMEM address, abort flag, a bank that is not finite

  const int lo = blockIdx.x * p.steps_per_cta * kStepSegs, hi = min(lo + p.steps_per_cta * kStepSegs, p.segs);
  const int steps = (hi - lo + kStepSegs - 1) / kStepSegs;
  const SegPos s_lo = seg_pos(lo, p);
  const int j_first = s_lo.n * p.L + s_lo.g * Wk::S;  // first stream row
  const unsigned magic_r = (unsigned)((0x100000000ull + (unsigned)p.R - 1) / (unsigned)p.R);

  // ---- set-up: the padding that no copy writes is zero
  if (NL == 1) {
    for (int i = threadIdx.x; i < p.R * p.CG; i += kThreads) *reinterpret_cast<uint4*>(smem + (size_t)i * p.pitch) = make_uint4(0, 0, 0, 0);
  } else {
    for (unsigned i = threadIdx.x * 16; i < ring_bytes; i += kThreads * 16) *reinterpret_cast<uint4*>(smem + i) = make_uint4(0, 0, 0, 0);
  }
  if (threadIdx.x < 2) *reinterpret_cast<uint4*>(smem + ring_bytes + threadIdx.x * 16) = make_uint4(0, 0, 0, 0);
  fence_proxy_async();
  if (threadIdx.x == 0) {
    for (int i = 0; i < kDepth; ++i) {
      mbar_init(x_full + 8 * i, NL == 1 ? 1 : 64 * NL);
      mbar_init(step_done + 8 * i, kConsumers);
    }
    for (int i = 0; i < kBufs; ++i) {
      mbar_init(b_full + 8 * i, WPB);
      mbar_init(b_free + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(t_full + 8 * i, 1);
      mbar_init(t_empty + 8 * i, kConsumers);
    }
    mbar_init(o_full, kConsumers);
    mbar_init(o_free, NS);
    fence_barrier_init();
    tail[1] = tail[2] = 0;
  }
  if (warp == kConsumers) tmem_alloc_all(smem_u32(const_cast<int*>(tail)));
  fence_before();
  __syncthreads();
  fence_after();
  const unsigned tmem = __shfl_sync(0xffffffffu, (unsigned)tail[0], 0);
  volatile int* abort_flag = tail + 1;
  if (warp < kConsumers) {  // bank -> TMEM
    const int q = warp & 3, tiles = p.full + (p.rest ? 4 : 0);
    for (int i = warp >> 2; i < tiles; i += kTeams) {
      int grp = i * 4 + q;
      if (i >= p.full) {
        const int k = rest_index(p.rest, i - p.full, q);
        grp = k < 0 ? -1 : p.full * 4 + k;
      }
      const int ch = grp * 32 + lane;
      const bool ok = grp >= 0 && ch < cg;
      bool finite = true;
      const float inv = bank_to_tmem<T>(tmem + ((unsigned)(q * 32) << 16) + kBankCol + i * TILE, bank + (size_t)(c0 + (ok ? ch : 0)) * p.cells,
                                        p.cells, ok, finite);
      if (SCALED && grp >= 0) inv_s[grp * 32 + lane] = inv;
      if (FULL && !finite) tail[2] = 1;
    }
    wait_st();
  }
  fence_before();
  __syncthreads();
  fence_after();

  if (FULL && tail[2]) {
    gather_block<T, MODE>(src, rot, bank, dst, p, c0, cg, lo, hi);
  } else if (warp < kConsumers) {
    // ================================================================ consumers
    regs_inc<consumer_regs<FULL, NL>()>();
    const int q = warp & 3, team = warp >> 2;
    const unsigned lanes = (unsigned)(q * 32) << 16;
    const bool vec = p.store == 16;
    constexpr int NA = MODE == kData2 ? 16 : 8;
    int use = 0;
    for (int s = 0; s < steps; ++s) {
      if (!wait_bar(x_full + 8 * (s & (kDepth - 1)), (s / kDepth) & 1, abort_flag)) break;
      // this pair's two segments, as the first loader left them: offsets of the source windows in the ring, and where the
      // segment lies (worked out by every consumer warp for itself, this was a third of all instructions at 96 channels)
      int4 sd[2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
        sd[h] = *reinterpret_cast<const int4*>(smem + sm.segs + ((s & (kDepth - 1)) * kStepSegs + team * 2 + h) * 16);
      bool ok = true, out_free = s == 0;
      for (int rd = 0; rd < rounds; ++rd) {
        int grp = rd * 4 + q;
        if (rd == p.full) {
          const int k = rest_index(p.rest, (team + s) & 3, q);
          grp = k < 0 ? -1 : p.full * 4 + k;
        }
        if (grp < 0) {  // no group for this quarter: only keep step with the sets of accumulators
          for (int v = 0; v < 3; ++v, ++use) {
            ok = wait_bar(t_full + 8 * (use & 1), (use >> 1) & 1, abort_flag);
            if (!ok) break;
            if (lane == 0) mbar_arrive(t_empty + 8 * (use & 1));
          }
          if (!ok) break;
          continue;
        }
        const int ch = grp * 32 + lane;
        const char* xc = smem + ch * p.pitch;
        const float inv = SCALED ? inv_s[ch] : FULL ? 1.f / 32768.f : 1.f;
        float acc[2][NA];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int i = 0; i < NA; ++i) acc[h][i] = 0.f;
        // items (kernel row, segment) in order; fp16 fetches the next item while it multiplies this one
        constexpr int NI = FULL ? 1 : 2;
        Item<T, MODE, FULL> item[NI];
        auto fetch = [&](Item<T, MODE, FULL>& it, int i) -> bool {
          const int v = i >> 1, h = i & 1, set = (use + v) & 1;
          if (h == 0) {
            if (!wait_bar(t_full + 8 * set, ((use + v) >> 1) & 1, abort_flag)) return false;
            fence_after();
            __syncwarp();
          }
          constexpr int row_of[3] = {0, MODE == kData2 ? 0 : 1, MODE == kData2 ? 1 : 2};
          it.load(tmem + lanes + set * kSetCols + team * kSlotCols + h * 24, xc + (row_of[v] == 0 ? sd[h].x : row_of[v] == 1 ? sd[h].y : sd[h].z));
          return true;
        };
        auto fetched = [&](Item<T, MODE, FULL>& it, int i) {
          wait_ld(it.k);
          if (i & 1) {  // both segments' accumulators of this kernel row are in registers
            fence_before();
            if (lane == 0) mbar_arrive(t_empty + 8 * ((use + (i >> 1)) & 1));
          }
        };
        if (NI == 2) {
          ok = fetch(item[0], 0);
          if (!ok) break;
          fetched(item[0], 0);
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) {
          if (NI == 2) {
            if (i < 5) {
              ok = fetch(item[(i + 1) % NI], i + 1);
              if (!ok) break;
            }
            multiply<T, MODE, FULL>(acc[i & 1], item[i % NI]);
            if (i < 5) fetched(item[(i + 1) % NI], i + 1);
          } else {
            ok = fetch(item[0], i);
            if (!ok) break;
            fetched(item[0], i);
            multiply<T, MODE, FULL>(acc[i & 1], item[0]);
          }
          if (MODE == kData2 && (i < 2 || i > 3)) {  // kernel row 0 completes the even row of the patch, 2 the odd one
            const int h = i & 1, row = 2 * (sd[h].w >> 8) + (i > 3), col = 16 * (sd[h].w & 255);
            if (sd[h].w >= 0 && ch < cg && row < p.Hd) {
              float o[16];
#pragma unroll
              for (int k = 0; k < 8; ++k) o[2 * k] = acc[h][k] * inv, o[2 * k + 1] = acc[h][NA - 8 + k] * inv;
              store_row<T, 16>(dst + (((size_t)sd[h].z * p.C + c0 + ch) * p.Hd + row) * p.Wd + col, o, p.Wd - col, vec);
            }
#pragma unroll
            for (int k = 0; k < NA; ++k) acc[h][k] = 0.f;
          }
        }
        if (!ok) break;
        use += 3;
        if (STAGED) {
          if (!out_free) {  // the results of the step before are on their way
            ok = wait_bar(o_free, (s - 1) & 1, abort_flag);
            if (!ok) break;
            out_free = true;
          }
          char* o = smem + sm.out + ch * kOutPitch + team * (16 * E);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if constexpr (E == 2) {
              unsigned r[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) r[k] = mma::pack2(acc[h][2 * k] * inv, acc[h][2 * k + 1] * inv);
              *reinterpret_cast<uint4*>(o + 16 * h) = make_uint4(r[0], r[1], r[2], r[3]);
            } else {
#pragma unroll
              for (int k = 0; k < 8; k += 4)
                *reinterpret_cast<float4*>(o + 32 * h + 4 * k) =
                    make_float4(acc[h][k] * inv, acc[h][k + 1] * inv, acc[h][k + 2] * inv, acc[h][k + 3] * inv);
            }
          }
        }
      }
      if (STAGED && ok && !out_free) ok = wait_bar(o_free, (s - 1) & 1, abort_flag);  // a step without a group for this warp
      if (!ok) break;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(step_done + 8 * (s & (kDepth - 1)));
        if (STAGED) mbar_arrive(o_full);
      }
    }
  } else if (warp == kConsumers) {
    // ================================================================ MMA
    regs_dec<helper_regs<FULL, NL>()>();
    constexpr unsigned idesc_all = idesc_f16(128, kSetCols, false, false, FULL), idesc_pair = idesc_f16(128, kSlotCols, false, false, FULL);
    int use = 0;
    bool ok = true;
    for (int s = 0, bi = 0, turn = 0; s < steps && ok; ++s) {
      ok = wait_bar(b_full + 8 * bi, turn & 1, abort_flag);
      if (!ok) break;
      fence_after();
      const unsigned buf = base + sm.beta + bi * (PIECES * kPiece);
      for (int rd = 0; rd < rounds && ok; ++rd) {
        for (int v = 0; v < 3; ++v, ++use) {
          const int set = use & 1;
          if (use >= 2) {
            ok = wait_bar(t_empty + 8 * set, ((use >> 1) - 1) & 1, abort_flag);
            if (!ok) break;
            fence_after();
          }
          const unsigned d = tmem + set * kSetCols;
          const uint64_t b = sdesc(buf + v * (kTeams * kPairRow), 128, 256);
          if (elect_one()) {
            if (rd < p.full) {
              products<T, FULL>(d, tmem + kBankCol + rd * TILE, b, idesc_all);
            } else {  // the remaining groups sit on other lanes for every pair
#pragma unroll
              for (int j = 0; j < kTeams; ++j) {
                products<T, FULL>(d + j * kSlotCols, tmem + kBankCol + (p.full + ((j + s) & 3)) * TILE, b + j * (kPairRow >> 4), idesc_pair);
              }
            }
            commit(t_full + 8 * set);
          }
          __syncwarp();
        }
      }
      if (ok && elect_one()) commit(b_free + 8 * bi);
      __syncwarp();
      if (++bi == kBufs) bi = 0, ++turn;
    }
  } else if (warp <= kConsumers + NL) {
    // ================================================================ source rows
    regs_dec<helper_regs<FULL, NL>()>();
    const int lw = warp - kConsumers - 1;
    int next = 0, done = 0;
    bool ok = true;
    for (int s = 0; s < steps && ok; ++s) {
      const SegPos e = seg_pos(min(lo + s * kStepSegs + kStepSegs - 1, hi - 1), p);
      const int last = e.n * p.L + e.g * Wk::S + Wk::rows - 1 - j_first;
      // steps that must be over: those that read the rows about to be overwritten, and the last user of this step's barrier
      while (done < s) {
        const SegPos f = seg_pos(lo + done * kStepSegs, p);
        const int first_row = f.n * p.L + f.g * Wk::S - j_first;
        if (done > s - kDepth && (next > last || first_row > last - p.R)) break;
        ok = wait_bar(step_done + 8 * (done & (kDepth - 1)), (done / kDepth) & 1, abort_flag);
        if (!ok) break;
        ++done;
      }
      if (!ok) break;
      const unsigned bar = x_full + 8 * (s & (kDepth - 1));
      if (lw == 0 && lane < kStepSegs) {
        // {ring offsets of the rows it reads; kData2: two of them, sample, segment row and column (negative: no segment)}
        const int b = lo + s * kStepSegs + lane;
        const SegPos q = seg_pos(min(b, hi - 1), p);
        const int k = q.n * p.L + q.g * Wk::S - j_first;
        int o[3];
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const int kk = k + (v < Wk::rows ? v : 0), sl = kk - (int)__umulhi((unsigned)kk, magic_r) * p.R;
          o[v] = sl * (int)slot_bytes + 16 + q.s * (8 * Wk::xs * E);
        }
        *reinterpret_cast<int4*>(smem + sm.segs + ((s & (kDepth - 1)) * kStepSegs + lane) * 16) =
            MODE == kData2 ? make_int4(o[0], o[1], q.n, b < hi ? q.g * 256 + q.s : -1) : make_int4(o[0], o[1], o[2], 0);
      }
      __syncwarp();
      if (NL == 1) {
        if (lane == 0) {
          if (last >= next) mbar_arrive_expect_tx(bar, (unsigned)(last - next + 1) * slot_bytes);
          else mbar_arrive(bar);
        }
        __syncwarp();
      }
      for (; next <= last; ++next) {
        const int sl = next - (int)__umulhi((unsigned)next, magic_r) * p.R;
        const int j = j_first + next, n = j / p.L, row = j - n * p.L + Wk::first;
        if (NL == 1) {
          if (lane == 0)
            for (int c = 0; c < p.CG; c += p.box_c)
              tma_load_3d(base + sl * slot_bytes + c * p.pitch, &tm, -(16 / E), row, n * p.C + c0 + c, bar);
        } else {
          copy_row<T, NL>(smem + (size_t)sl * slot_bytes, src, n, c0, cg, row, p, lw, lane);
        }
      }
      if (NL != 1) {
        cp_async_arrive_noinc(bar);
        mbar_arrive(bar);
      }
    }
  } else if (warp <= kConsumers + NL + NB) {
    // ================================================================ hat products
    regs_dec<helper_regs<FULL, NL>()>();
    const int w = (warp - kConsumers - 1 - NL) % WPB, bi = (warp - kConsumers - 1 - NL) / WPB;
    Offsets<T, WPB> off;
    if (bi < steps) fetch_offsets<T, MODE, WPB>(off, rot, lo + bi * kStepSegs, hi, p, w, lane);
    for (int s = bi, turn = 0; s < steps; s += kBufs, ++turn) {
      if (turn > 0 && !wait_bar(b_free + 8 * bi, (turn - 1) & 1, abort_flag)) break;
      write_hats<T, MODE, SC44, FULL, WPB>(base + sm.beta + bi * (PIECES * kPiece), off, p, w, lane);
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(b_full + 8 * bi);
      if (s + kBufs < steps) fetch_offsets<T, MODE, WPB>(off, rot, lo + (s + kBufs) * kStepSegs, hi, p, w, lane);
    }
  } else {
    // ================================================================ results to memory
    regs_dec<helper_regs<FULL, NL>()>();
    const int w = warp - kConsumers - 1 - NL - NB;
    const size_t plane = (size_t)p.Hd * p.Wd;
    for (int s = 0; s < steps && STAGED; ++s) {
      const int seg = lo + s * kStepSegs;
      // where this lane's share of a channel's 64 staged values goes: `store` bytes of a segment
      if (p.store == 16) {
        constexpr int PC = kStepSegs * 8 * E / 16, PS = PC / kStepSegs;  // 16-byte pieces per channel, per segment
        const int i = lane % PC, b = seg + i / PS;
        const SegPos sp = seg_pos(min(b, hi - 1), p);
        const int col = 8 * sp.s + (i % PS) * (16 / E);
        T* d = dst + ((size_t)sp.n * p.C + c0) * plane + (size_t)sp.g * p.Wd + col;
        const char* o = smem + sm.out + i * 16;
        if (!wait_bar(o_full, s & 1, abort_flag)) break;
        if (b < hi && col < p.Wd) {
#pragma unroll 4
          for (int c = w * (32 / PC) + lane / PC; c < cg; c += NS * (32 / PC))
            *reinterpret_cast<uint4*>(d + c * plane) = *reinterpret_cast<const uint4*>(o + c * kOutPitch);
        }
      } else {
        if (!wait_bar(o_full, s & 1, abort_flag)) break;
        const int per = 8 * E / p.store;
        for (int i = lane; i < kStepSegs * per; i += 32) {
          const int b = seg + i / per;
          const SegPos sp = seg_pos(min(b, hi - 1), p);
          const int col = 8 * sp.s + (i % per) * (p.store / E);
          if (b < hi && col < p.Wd) {
            T* d = dst + ((size_t)sp.n * p.C + c0) * plane + (size_t)sp.g * p.Wd + col;
            const char* o = smem + sm.out + i * p.store;
            if (p.store == 4) {
#pragma unroll 4
              for (int c = w; c < cg; c += NS) *reinterpret_cast<unsigned*>(d + c * plane) = *reinterpret_cast<const unsigned*>(o + c * kOutPitch);
            } else {
#pragma unroll 4
              for (int c = w; c < cg; c += NS)
                *reinterpret_cast<unsigned short*>(d + c * plane) = *reinterpret_cast<const unsigned short*>(o + c * kOutPitch);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(o_free);
    }
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  if (*abort_flag) {
    // a wait ran out: report it, and leave the shared memory that copies may still write to for a while
    if (threadIdx.x == 0) atomicExch(&g_tc_error, 2);
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  if (warp == kConsumers) {
    fence_after();
    tmem_free_all(tmem);
  }
}

template <typename T, int MODE, bool SC44, int NL>
__global__ void __launch_bounds__(kThreads, 1)
    tc_conv_kernel(const __grid_constant__ CUtensorMap tm, const T* __restrict__ src, const T* __restrict__ rot,
                   const T* __restrict__ bank, T* __restrict__ dst, const __grid_constant__ ConvParams p) {
  tc_conv<T, MODE, SC44, NL, true>(tm, src, rot, bank, dst, p);
}
template <int MODE, bool SC44, int NL>
__global__ void __launch_bounds__(kThreads, 1)
    tc_conv_rounded_kernel(const __grid_constant__ CUtensorMap tm, const __half* __restrict__ src, const __half* __restrict__ rot,
                           const __half* __restrict__ bank, __half* __restrict__ dst, const ConvParams p) {
  tc_conv<__half, MODE, SC44, NL, false>(tm, src, rot, bank, dst, p);
}

// ------------------------------------------------------------------ host side
bool tc_shape(const Geom& g) {
  if (g.kH != 3 || g.kW != 3 || g.dH != 1 || g.dW != 1 || g.pH != 1 || g.pW != 1) return false;
  if (g.sH != g.sW || (g.sH != 1 && g.sH != 2)) return false;
  return g.G == 1 && g.cells <= 16;
}

// most stream rows that `segments` consecutive segments can read
int step_rows(int nseg, int Hg, int S, int L, int rows, int segments) {
  const int span = (nseg - 1 + segments - 1) / nseg;      // segment rows beyond the first
  const int crossings = span ? (span + Hg - 1) / Hg : 0;  // samples beyond the first
  return span * S + crossings * (L - Hg * S) + rows;
}

struct ConvPlan {
  bool ok;
  bool tma;
  int ctas, splits;
  size_t smem;
  ConvParams p;
};

template <typename T, int MODE, bool FULL>
ConvPlan plan_conv(const Geom& g, const void* src, const void* dst) {
  using Wk = Walk<MODE>;
  ConvPlan pl;
  pl.ok = false;
  ConvParams& p = pl.p;
  constexpr bool kData = MODE == kData1 || MODE == kData2;
  constexpr int E = sizeof(T);
  p.N = g.N, p.C = g.C, p.Ho = g.Ho, p.Wo = g.Wo;
  p.Hs = kData ? g.Ho : g.H, p.Ws = kData ? g.Wo : g.W;
  p.Hd = kData ? g.H : g.Ho, p.Wd = kData ? g.W : g.Wo;
  p.Hg = MODE == kData2 ? g.Ho : p.Hd, p.Wg = MODE == kData2 ? g.Wo : p.Wd;
  p.nseg = (p.Wg + 7) / 8;
  p.L = MODE == kFwd2 ? 2 * g.Ho + 1 : (MODE == kData2 ? g.Ho + 1 : p.Hs + 2);
  const long long rows = (long long)g.N * p.Hg, segs = rows * p.nseg;
  if (segs > 0x3fffffffLL || (long long)g.N * p.L > 0x3fffffffLL) return pl;
  // the divisions by nseg, Hg and the ring depth are multiplications that need these products below 2^32
  if (segs * p.nseg > 0xffffffffLL || rows * p.Hg > 0xffffffffLL) return pl;
  p.segs = (int)segs;
  p.magic_seg = (unsigned)((0x100000000ull + p.nseg - 1) / p.nseg);
  p.magic_row = (unsigned)((0x100000000ull + p.Hg - 1) / p.Hg);
  p.scW = g.scW, p.cells = g.cells;
  p.uh0 = 0.5f * (g.scH - 3), p.uw0 = 0.5f * (g.scW - 3);
  p.store = E;
  if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (p.Wd * E) % 16 == 0) p.store = 16;
  else if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0 && (p.Wd * E) % 4 == 0) p.store = 4;
  // padded row: 16 bytes in front; the column behind the last segment is the next row's front
  p.pitch = ((1 + (p.nseg * 8 * Wk::xs * E) / 16) | 1) * 16;
  if (p.pitch < 16 + p.Ws * E || p.pitch > 1152 || p.Hg >= (1 << 22)) return pl;
  pl.tma = (reinterpret_cast<uintptr_t>(src) & 15) == 0 && (p.Ws * E) % 16 == 0 && p.pitch / E <= 256;
  const int need = step_rows(p.nseg, p.Hg, Wk::S, p.L, Wk::rows, kStepSegs);
  const int want = step_rows(p.nseg, p.Hg, Wk::S, p.L, Wk::rows, kStepSegs * kDepth);
  const int groups = (g.C + 31) / 32, steps = (p.segs + kStepSegs - 1) / kStepSegs, sms = device_sm_count();
  const size_t budget = (size_t)device_smem_optin();
  long long best = -1;
  for (int per = groups; per >= 1; --per) {  // groups per block
    const int splits = (groups + per - 1) / per;
    if ((groups + splits - 1) / splits != per || splits > 65535) continue;  // as many blocks with a better balance exist
    const int full = per / 4, rest = per % 4;
    if ((full + (rest ? 4 : 0)) * 8 * bank_piece_count<T>() > 512 - kBankCol) continue;
    int cg = splits == 1 ? (g.C + 7) & ~7 : per * 32;
    const int boxes = (cg + 255) / 256;
    cg = (cg + 8 * boxes - 1) / (8 * boxes) * (8 * boxes);  // boxes start on 128 bytes
    if (splits > 1 && cg != per * 32) continue;
    const size_t slot = (size_t)cg * p.pitch, fixed = conv_smem<T, MODE, FULL>(0, per).total + 160;
    if (fixed + slot * (need + 1) > budget) continue;
    int R = (int)((budget - fixed) / slot);
    if (R > want + 2) R = want + 2;
    const bool shallow = R < need + 2 * Wk::S + 1;
    long long cx = sms / splits > 0 ? sms / splits : 1;
    if (cx > steps) cx = steps;
    const int spc = (int)((steps + cx - 1) / cx);
    const long long waves = ((long long)((steps + spc - 1) / spc) * splits + sms - 1) / sms;
    // time of a block ~ steps x (groups + the hat products, about one group's work), plus its set-up
    const long long cost = waves * ((long long)(spc + 2) * (per + 1) * (shallow ? 5 : 4));
    if (best < 0 || cost < best) {
      best = cost;
      pl.ok = true;
      p.CG = cg, p.box_c = cg / boxes, p.full = full, p.rest = rest, p.R = R;
      p.steps_per_cta = spc;
      pl.ctas = (steps + spc - 1) / spc, pl.splits = splits;
      pl.smem = conv_smem<T, MODE, FULL>((unsigned)(slot * R), per).total;
      if (pl.smem < kMinSmem) pl.smem = kMinSmem;
    }
  }
  return pl;
}

// Registers per thread that a launch of KERN allocates; -1: the query failed.
template <auto KERN>
int launch_registers() {
  cudaFuncAttributes at;
  const cudaError_t e = cudaFuncGetAttributes(&at, KERN);
  if (e == cudaSuccess) return at.numRegs;
  (void)cudaGetLastError();
  return -1;
}
// setmaxnreg.inc waits for registers that the launch did not allocate for ever: a kernel that was compiled to fewer than the
// roles' shares add up to is not launched.  One answer per kernel (the kernels of a template share a pointer type, so KERN is
// a template argument); a failed query is not kept.
template <auto KERN>
bool shares_fit() {
  static std::atomic<int> regs{-1};
  int r = regs.load(std::memory_order_relaxed);
  if (r < 0) {
    r = launch_registers<KERN>();
    regs.store(r, std::memory_order_relaxed);
  }
  return r >= kRegsLaunch;
}

template <auto KERN, typename T>
int run_conv(const ConvPlan& pl, const CUtensorMap& tm, const T* src, const T* rot, const T* w, T* dst, cudaStream_t s) {
  if (!shares_fit<KERN>()) return DK_ERR_UNSUPPORTED;
  const int rc = enable_smem(KERN, pl.smem);
  if (rc) return rc;
  KERN<<<dim3(pl.ctas, pl.splits), kThreads, pl.smem, s>>>(tm, src, rot, w, dst, pl.p);
  return check_launch();
}
template <typename T, int MODE, bool SC44, int NL, bool FULL>
constexpr auto conv_kernel() {
  if constexpr (FULL) return &tc_conv_kernel<T, MODE, SC44, NL>;
  else return &tc_conv_rounded_kernel<MODE, SC44, NL>;
}

template <typename T, int MODE, bool FULL>
int launch_conv(const T* src, const T* rot, const T* w, T* dst, const Geom& g, cudaStream_t s) {
  const ConvPlan pl = plan_conv<T, MODE, FULL>(g, src, dst);
  if (!pl.ok) return DK_ERR_UNSUPPORTED;
  CUtensorMap tm;
  std::memset(&tm, 0, sizeof(tm));
  if (pl.tma && !make_plane_row_map(&tm, src, sizeof(T), pl.p.Ws, pl.p.Hs, (long long)g.N * g.C, pl.p.pitch / (int)sizeof(T), pl.p.box_c))
    return DK_ERR_UNSUPPORTED;
  const bool sc44 = g.scH == 4 && g.scW == 4;
  if (pl.tma)
    return sc44 ? run_conv<conv_kernel<T, MODE, true, 1, FULL>()>(pl, tm, src, rot, w, dst, s)
                : run_conv<conv_kernel<T, MODE, false, 1, FULL>()>(pl, tm, src, rot, w, dst, s);
  return sc44 ? run_conv<conv_kernel<T, MODE, true, kLoaders, FULL>()>(pl, tm, src, rot, w, dst, s)
              : run_conv<conv_kernel<T, MODE, false, kLoaders, FULL>()>(pl, tm, src, rot, w, dst, s);
}

template <typename T, int MODE, bool SC44, int NL, bool FULL>
void add_registers(long long out[8]) {
  const int r = launch_registers<conv_kernel<T, MODE, SC44, NL, FULL>()>();
  ++out[0];
  if (out[1] < 0 || r < out[1]) out[1] = r;
}
template <typename T, int MODE, bool FULL>
void add_registers_of(long long out[8]) {
  add_registers<T, MODE, true, 1, FULL>(out), add_registers<T, MODE, false, 1, FULL>(out);
  add_registers<T, MODE, true, kLoaders, FULL>(out), add_registers<T, MODE, false, kLoaders, FULL>(out);
}
template <typename T, bool FULL>
void add_registers_of(long long out[8]) {
  add_registers_of<T, kFwd1, FULL>(out), add_registers_of<T, kFwd2, FULL>(out), add_registers_of<T, kData1, FULL>(out),
      add_registers_of<T, kData2, FULL>(out);
}

template <typename T, bool FULL>
int launch_conv(const T* src, const T* rot, const T* w, T* dst, const Geom& g, bool transposed, cudaStream_t s) {
  if (!tc_shape(g)) return DK_ERR_UNSUPPORTED;
  if (!transposed) return g.sH == 1 ? launch_conv<T, kFwd1, FULL>(src, rot, w, dst, g, s) : launch_conv<T, kFwd2, FULL>(src, rot, w, dst, g, s);
  return g.sH == 1 ? launch_conv<T, kData1, FULL>(src, rot, w, dst, g, s) : launch_conv<T, kData2, FULL>(src, rot, w, dst, g, s);
}

}  // namespace

template <typename T>
int local_conv_tc(const T* src, const T* rot, const T* w, T* dst, const Geom& g, bool transposed, cudaStream_t s) {
  return launch_conv<T, true>(src, rot, w, dst, g, transposed, s);
}
template int local_conv_tc<float>(const float*, const float*, const float*, float*, const Geom&, bool, cudaStream_t);
template int local_conv_tc<__half>(const __half*, const __half*, const __half*, __half*, const Geom&, bool, cudaStream_t);

int local_conv_tc_rounded(const __half* src, const __half* rot, const __half* w, __half* dst, const Geom& g, bool transposed,
                          cudaStream_t s) {
  return launch_conv<__half, false>(src, rot, w, dst, g, transposed, s);
}

int tc_register_query(long long out[8]) {
  for (int i = 0; i < 8; ++i) out[i] = 0;
  out[1] = -1, out[2] = kRegsLaunch;
  add_registers_of<float, true>(out), add_registers_of<__half, false>(out), add_registers_of<__half, true>(out);
  return out[1] < 0 ? DK_ERR_CUDA : DK_OK;
}

int tc_error_status() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)) != cudaSuccess) return -1;
  return v;
}

}  // namespace dk
