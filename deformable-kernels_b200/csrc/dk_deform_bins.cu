// Gradients of DK + DCN where the tensor-core kernels do not apply (fp32; fp16 with channels that are no multiple of 16, other
// scopes, planes beyond 56 x 56), one offset group.
//
// The scatter of dy * k into the four corners of every sample point is 36 float additions to colliding addresses per output,
// and shared memory adds floats with a compare-and-swap loop: 0.25 ms for 16 x 192 channels of 28 x 28 (350 G additions / s),
// as slow as additions in L2.  But where a sample lands does not depend on the channel.  So the samples (pixel, tap) are first
// sorted by the cell of the input grid they fall into, once for all channels (dcn_bins_kernel), and then a warp walks through
// the cells of a row with 32 channels on its lanes and the four corner sums in registers: no atomics, no collisions, one
// multiply-add per corner (dcn_gather_kernel).  16 x 192 of 28 x 28: 245 -> 71 us (19 of them the sort); 13 x 96 of 80 x 80:
// 985 -> 281, in fp16 912 -> 281; 64 x 384 of 14 x 14: 640 -> 111; 32 x 72 of 56 x 56, stride 2: 124 -> 101.  The gather is
// bound by latency: 1.6 instructions per cycle and SM (40 % of the issue slots) from one dependent walk per warp, 192 blocks of eight
// warps on 148 SMs for 16 x 192 of 28 x 28; the sort by the latency of its five steps.
#include <cooperative_groups.h>

#include <type_traits>

#include "dk_common.cuh"

namespace dk {
namespace {

namespace cg = cooperative_groups;

constexpr int kSortBlocks = 8, kSortThreads = 1024;  // a cluster of 8 blocks sorts one sample
constexpr int kGatherWarps = 8, kMovePixels = 128;

struct BinPlan {
  int bins, rec_per_n, Cp, groups;  // (H + 1) x (W + 1) cells; taps * P samples; channels rounded up to those of a block
  int movers, sorted;               // first block that transposes; samples to sort (N or none)
  int V, R, bands, segs;               // destination rows of a block, blocks per plane, pieces of a row of cells
  int bank_blocks;                  // partial bank gradients
  bool sorts;                       // the sort's table and the gather's sums fit: grad-input, which no other pass needs
  size_t starts_bytes, recs_bytes, dyt_bytes, bytes, xt_bytes, bankt_bytes, all_bytes, sort_smem, gather_smem;
};

// The bank in channel order: [scH + 2][scW + 2] cells with a border of zeros, and behind them as many zeros as the four cells of a
// sample span, for samples that are not used (zero weights alone would let a cell that is not finite through).
__host__ __device__ inline int bank_unused_cell(const Geom& g) { return (g.scH + 2) * (g.scW + 2); }
__host__ __device__ inline int bank_cells(const Geom& g) { return bank_unused_cell(g) + g.scW + 4; }

// Without kernel-space offsets (rot null) the sampled kernel is the same at every pixel: in place of the bank its value per (tap,
// channel) is laid out, and one read stands for four and their multiply-adds; the bank gradient meets the cells once per tap.  16 x 192
// of 28 x 28, 3 x 3 scope: forward 39 -> 25 us, gather 53 -> 44, offsets 43 -> 31, bank 42 -> 33; 13 x 88 of 80 x 80 in fp16, all, 848 -> 646.
// The unused cell keeps its zeros; samples that are not used meet their tap's value with zeros, and where that leaves sums that are not finite
// they are formed again with zero selected in its place.
__host__ __device__ inline bool fixed_kernel(const Geom& g, const void* rot) { return rot == nullptr && g.taps <= bank_unused_cell(g); }

// one sample point: corner coefficients of the image and of the bank, {bank cell * 32, column of the cell, pixel * Cp, 0}
struct Rec {
  float4 ci, cb;
  int4 at;
};

// where sample (n, tap, p) falls in the image and in the bank (rot may be null: zeros): upper left corner (-1 .. last) and the fractions
struct Point {
  int h0, w0, u0, v0;
  float lh, lw, lu, lv;
};

template <typename T>
__device__ __forceinline__ bool sample_point(int n, int tap, int p, const T* __restrict__ off, const T* __restrict__ rot, const Geom& g,
                                             Point& q) {
  const int fh = tap / g.kW, fw = tap - fh * g.kW, oh = p / g.Wo, ow = p - oh * g.Wo;
  const size_t o = ((size_t)n * g.taps + tap) * 2 * g.P + p;
  const float ph = (float)(oh * g.sH - g.pH + fh * g.dH) + ld<float>(off + o);
  const float pw = (float)(ow * g.sW - g.pW + fw * g.dW) + ld<float>(off + o + g.P);
  const float u = ((float)fh + (rot ? ld<float>(rot + o) : 0.f)) + (float)(g.scH - g.kH) * 0.5f;
  const float v = ((float)fw + (rot ? ld<float>(rot + o + g.P) : 0.f)) + (float)(g.scW - g.kW) * 0.5f;
  // written so that NaN fails; what passes is in range for the conversions below
  if (!(ph > -1.f && pw > -1.f && ph < (float)g.H && pw < (float)g.W)) return false;
  if (!(u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW)) return false;
  const float fph = floorf(ph), fpw = floorf(pw), fu = floorf(u), fv = floorf(v);
  q.h0 = (int)fph, q.w0 = (int)fpw, q.u0 = (int)fu, q.v0 = (int)fv;
  q.lh = ph - fph, q.lw = pw - fpw, q.lu = u - fu, q.lv = v - fv;
  return true;
}

// cell of sample i = tap * P + p, or -1 where it adds nothing
template <typename T>
__device__ __forceinline__ int sample_cell(int i, int n, const T* __restrict__ off, const T* __restrict__ rot, const Geom& g, Rec* rec,
                                           int Cp) {
  const int tap = i / g.P, p = i - tap * g.P;
  Point q;
  if (!sample_point(n, tap, p, off, rot, g, q)) return -1;
  if (rec != nullptr) {
    const float hh = 1.f - q.lh, hw = 1.f - q.lw, hu = 1.f - q.lu, hv = 1.f - q.lv;
    rec->ci = make_float4(hh * hw, hh * q.lw, q.lh * hw, q.lh * q.lw);
    rec->cb = make_float4(hu * hv, hu * q.lv, q.lu * hv, q.lu * q.lv);
    rec->at = make_int4((fixed_kernel(g, rot) ? tap : (q.u0 + 1) * (g.scW + 2) + q.v0 + 1) * 32, q.w0 + 1, p * Cp, 0);
  }
  return (q.h0 + 1) * (g.W + 1) + q.w0 + 1;
}

template <typename T>
__device__ __forceinline__ float fixed_kernel_value(int tap, int c, const T* __restrict__ w, const Geom& g) {
  const int fh = tap / g.kW, fw = tap - fh * g.kW;
  Bilinear<float> b;
  float k = 0.f;
  if (bank_setup<float>(0.f, 0.f, fh, fw, g, b)) {
    const float t[4] = {b.hh, b.hh, b.lh, b.lh}, u[4] = {b.hw, b.lw, b.hw, b.lw};
    for (int e = 0; e < 4; ++e)
      if (b.m[e]) k += t[e] * u[e] * ld<float>(w + (size_t)c * g.cells + b.idx[e]);
  }
  return k;
}

template <typename T>
__device__ __forceinline__ void move_channels(const T* __restrict__ src, T* __restrict__ dst, int P, const Geom& g, const BinPlan& t,
                                              float* tile) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tiles_p = (P + 1 + kMovePixels - 1) / kMovePixels, per_n = t.Cp / 32 * tiles_p;
  for (int k = blockIdx.x - t.movers; k >= 0 && k < g.N * per_n; k += gridDim.x - t.movers) {
    const int m = k / per_n, r = k - m * per_n, grp = r / tiles_p, p0 = (r - grp * tiles_p) * kMovePixels;
    const T* from = src + ((size_t)m * g.C + min(grp * 32 + warp, g.C - 1)) * P;
    const bool has = grp * 32 + warp < g.C;
    float v[kMovePixels / 32];
#pragma unroll
    for (int e = 0; e < kMovePixels / 32; ++e)
      v[e] = has && p0 + e * 32 + lane < P ? ld<float>(from + p0 + e * 32 + lane) : 0.f;
    __syncthreads();
#pragma unroll
    for (int e = 0; e < kMovePixels / 32; ++e) tile[(e * 32 + lane) * 33 + warp] = v[e];
    __syncthreads();
    T* to = dst + ((size_t)m * (P + 1) + p0 + warp) * t.Cp + grp * 32 + lane;
#pragma unroll
    for (int e = 0; e < kMovePixels / 32; ++e)
      if (p0 + warp + e * 32 <= P) st<T, float>(to + (size_t)e * 32 * t.Cp, tile[(warp + e * 32) * 33 + lane]);
  }
}

// Counting sort of the samples of one (n) by cell: every block of the cluster counts its share in shared memory, the blocks
// share the prefix sums (an eighth of the cells each, through distributed shared memory), then every block places its samples.
// The clusters beyond the first (or, where they are few, all blocks before they sort) bring dy, x and the bank into the order
// in which the channels of a pixel or cell are neighbours: [P + 1][Cp] and [H W + 1][Cp] with a last pixel of zeros, and
// [bank_cells][Cp].  x and the bank only where the other gradients want them.
template <typename T>
__global__ void __launch_bounds__(kSortThreads, 2) dcn_bins_kernel(const T* __restrict__ dy, const T* __restrict__ off,
                                                                const T* __restrict__ rot, int* __restrict__ starts,
                                                                Rec* __restrict__ recs, T* __restrict__ dyt,
                                                                const T* __restrict__ x, T* __restrict__ xt, const T* __restrict__ w,
                                                                float* __restrict__ bankt, const Geom g, const BinPlan t) {
  extern __shared__ __align__(16) int hist[];
  __shared__ int slices[kSortBlocks], warp_sum[32];
  __shared__ float tile[kMovePixels * 33];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = blockIdx.x / kSortBlocks, rank = blockIdx.x - n * kSortBlocks;
  if (dyt != nullptr) move_channels(dy, dyt, g.P, g, t, tile);
  if (xt != nullptr) {
    move_channels(x, xt, g.HW, g, t, tile);
    const int cells = bank_cells(g);
    for (int i = (blockIdx.x - t.movers) * kSortThreads + tid; i >= 0 && i < cells * t.Cp; i += (gridDim.x - t.movers) * kSortThreads) {
      const int cell = i / t.Cp, c = i - cell * t.Cp, a = cell / (g.scW + 2) - 1, b = cell - (a + 1) * (g.scW + 2) - 1;
      if (fixed_kernel(g, rot)) bankt[i] = c < g.C && cell < g.taps ? fixed_kernel_value<T>(cell, c, w, g) : 0.f;
      else bankt[i] = c < g.C && a >= 0 && a < g.scH && b >= 0 && b < g.scW ? ld<float>(w + (size_t)c * g.cells + a * g.scW + b) : 0.f;
    }
  }
  if (n >= t.sorted) return;
  cg::cluster_group cluster = cg::this_cluster();
  for (int i = tid; i < t.bins; i += kSortThreads) hist[i] = 0;
  __syncthreads();
  for (int i = rank * kSortThreads + tid; i < t.rec_per_n; i += kSortBlocks * kSortThreads) {
    const int cell = sample_cell<T>(i, n, off, rot, g, nullptr, 0);
    if (cell >= 0) atomicAdd(&hist[cell], 1);
  }
  cluster.sync();
  const int per = (t.bins + kSortBlocks - 1) / kSortBlocks, q = (per + kSortThreads - 1) / kSortThreads;
  const int hi = min((rank + 1) * per, t.bins), lo = rank * per + tid * q, end = min(lo + q, hi);
  int sum = 0;
  for (int b = lo; b < end; ++b)
#pragma unroll
    for (int k = 0; k < kSortBlocks; ++k) sum += cluster.map_shared_rank(hist, k)[b];
  int scan = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, scan, d);
    if (lane >= d) scan += o;
  }
  if (lane == 31) warp_sum[warp] = scan;
  __syncthreads();
  int base = 0, total = 0;
  for (int w = 0; w < kSortThreads / 32; ++w) {
    if (w < warp) base += warp_sum[w];
    total += warp_sum[w];
  }
  if (tid < kSortBlocks) cluster.map_shared_rank(slices, tid)[rank] = total;
  cluster.sync();
  int run = base + scan - sum, before = 0;
  for (int k = 0; k < rank; ++k) before += slices[k];
  run += before;
  int* out = starts + (size_t)n * (t.bins + 1);
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
  if (rank == kSortBlocks - 1 && tid == 0) out[t.bins] = before + total;
  cluster.sync();
  Rec* to = recs + (size_t)n * t.rec_per_n;
  for (int i = rank * kSortThreads + tid; i < t.rec_per_n; i += kSortBlocks * kSortThreads) {
    Rec r;
    const int cell = sample_cell<T>(i, n, off, rot, g, &r, t.Cp);
    if (cell >= 0) to[atomicAdd(&hist[cell], 1)] = r;
  }
}

// one or two neighbouring channels
template <typename T, int V>
__device__ __forceinline__ void get(const T* p, float (&v)[V]) {
  if constexpr (V == 1) {
    v[0] = static_cast<float>(*p);
  } else if constexpr (sizeof(T) == 4) {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x, v[1] = q.y;
  } else {
    const float2 q = __half22float2(*reinterpret_cast<const __half2*>(p));
    v[0] = q.x, v[1] = q.y;
  }
}
// the same at a byte offset: one addition and no 64-bit address per load
template <typename T, int V>
__device__ __forceinline__ void get_at(const T* base, unsigned off, float (&v)[V]) {
  get<T, V>(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off), v);
}
template <int V>
__device__ __forceinline__ void put(float* p, const float (&v)[V]) {
  if constexpr (V == 1) *p = v[0];
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}

// Block = 32 V channels of R rows of dx, V channels on a lane.  A unit of a warp is a piece of a row of cells: the samples of a cell add to
// S00 .. S11, which at the end of the cell go to its four corners; the right-hand pair is carried to the next cell.  Even rows
// of cells write their two rows of dx first, then the odd rows add theirs, so no element has two writers.  What a piece
// carries past its end waits in `seam`.  A sample costs four shared loads of its record, one line of dy, four bank reads
// and nine multiplications or multiply-adds per channel.
template <typename T, int V, bool FIXED>
__global__ void __launch_bounds__(32 * kGatherWarps, 3) dcn_gather_kernel(const T* __restrict__ dyt, const int* __restrict__ starts,
                                                                       const Rec* __restrict__ recs, const T* __restrict__ w,
                                                                       T* __restrict__ dx, const Geom g, const BinPlan t) {
  constexpr int CB = 32 * V, PITCH = V == 1 ? 33 : 66;
  extern __shared__ __align__(16) float4 smem4[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x / t.bands, r0 = (blockIdx.x - n * t.bands) * t.R, rows = min(t.R, g.H - r0);
  const int c0 = blockIdx.y * CB, n_c = min(CB, g.C - c0), bw = g.scW + 2, W1 = g.W + 1;
  float4* stage = smem4 + warp * 96;                                   // [32 records]
  float* bank = reinterpret_cast<float*>(smem4 + kGatherWarps * 96);   // [cell of the zero-bordered bank][channel]
  float* seam = bank + bank_cells(g) * CB;                          // [row of cells][piece][upper | lower][channel]
  float* acc = seam + (t.R + 1) * t.segs * 2 * CB;                     // [row][column][PITCH]
  for (int i = threadIdx.x; i < bank_cells(g) * CB; i += 32 * kGatherWarps) {
    const int cell = i / CB, a = cell / bw - 1, b = cell - (a + 1) * bw - 1, c = i % CB;
    if (FIXED) bank[i] = c < n_c && cell < g.taps ? fixed_kernel_value<T>(cell, c0 + c, w, g) : 0.f;
    else bank[i] = (c < n_c && a >= 0 && a < g.scH && b >= 0 && b < g.scW) ? ld<float>(w + (size_t)(c0 + c) * g.cells + a * g.scW + b) : 0.f;
  }
  __syncthreads();
  const T* yl = dyt + (size_t)n * (g.P + 1) * t.Cp + c0 + V * lane;
  const int* st_n = starts + (size_t)n * (t.bins + 1);
  const float4* rc_n = reinterpret_cast<const float4*>(recs + (size_t)n * t.rec_per_n);
  const float* bl = bank + V * lane;
  const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int phase = 0; phase < 2; ++phase) {
    const int n_rows = (rows + 2 - phase) >> 1;  // rows of cells r0 - 1 .. r0 + rows - 1, every other one
    for (int unit = warp; unit < n_rows * t.segs; unit += kGatherWarps) {
      const int k = unit / t.segs, seg = unit - k * t.segs, i = 2 * k + phase;  // row r0 - 1 + i of the plane
      const int b0 = seg * W1 / t.segs, b1 = (seg + 1) * W1 / t.segs;
      const int* sr = st_n + (r0 + i) * W1;
      const int first = __ldg(sr + b0), last = __ldg(sr + b1);
      float* up = i >= 1 ? acc + (i - 1) * g.W * PITCH + V * lane : nullptr;
      float* low = i < rows ? acc + i * g.W * PITCH + V * lane : nullptr;
      int cur = b0;
      float s00[V] = {}, s01[V] = {}, s10[V] = {}, s11[V] = {}, cu[V] = {}, cl[V] = {};
      auto flush = [&]() {
        if (cur > 0) {
          const int o = (cur - 1) * PITCH;
#pragma unroll
          for (int j = 0; j < V; ++j) cu[j] += s00[j], cl[j] += s10[j];
          if (up) {
            if (phase)
              for (int j = 0; j < V; ++j) cu[j] += up[o + j];
            put<V>(up + o, cu);
          }
          if (low) {
            if (phase)
              for (int j = 0; j < V; ++j) cl[j] += low[o + j];
            put<V>(low + o, cl);
          }
        }
#pragma unroll
        for (int j = 0; j < V; ++j) cu[j] = s01[j], cl[j] = s11[j], s00[j] = s01[j] = s10[j] = s11[j] = 0.f;
        ++cur;
      };
      // records beyond the last one: no weight, the zero pixel, zero cells of the bank, no new cell
      float4 next[3];
      auto fetch = [&](int at) {
        const int lim = (last - at) * 3;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const int e = lane + 32 * j;
          next[j] = e < lim ? __ldg(rc_n + (size_t)at * 3 + e) : none;
          if (e >= lim && e % 3 == 2) next[j].x = __int_as_float(bank_unused_cell(g) * 32), next[j].z = __int_as_float(g.P * t.Cp);
        }
      };
      if (first < last) fetch(first);
      for (int at = first; at < last; at += 32) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 3; ++j) stage[lane + 32 * j] = next[j];
        __syncwarp();
        if (at + 32 < last) fetch(at + 32);
        const int cnt = min(32, last - at);
        for (int k0 = 0; k0 < cnt; k0 += 8) {
          float yv[8][V];
#pragma unroll
          for (int j = 0; j < 8; ++j) get<T, V>(yl + reinterpret_cast<const int*>(stage + (k0 + j) * 3 + 2)[2], yv[j]);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float4 ci = stage[(k0 + j) * 3], cb = FIXED ? none : stage[(k0 + j) * 3 + 1];
            const int2 at2 = *reinterpret_cast<const int2*>(stage + (k0 + j) * 3 + 2);
            while (cur < at2.y) flush();
            const float* bk = bl + at2.x * V;
            float b0v[V], b1v[V], b2v[V], b3v[V];
            get<float, V>(bk, b0v);
            if (!FIXED) get<float, V>(bk + CB, b1v), get<float, V>(bk + bw * CB, b2v), get<float, V>(bk + bw * CB + CB, b3v);
#pragma unroll
            for (int e = 0; e < V; ++e) {
              const float kv = FIXED ? b0v[e] : cb.x * b0v[e] + cb.y * b1v[e] + cb.z * b2v[e] + cb.w * b3v[e];
              const float v = kv * yv[j][e];
              s00[e] += ci.x * v, s01[e] += ci.y * v, s10[e] += ci.z * v, s11[e] += ci.w * v;
            }
          }
        }
      }
      while (cur < b1) flush();
      put<V>(seam + ((i * t.segs + seg) * 2) * CB + V * lane, cu);
      put<V>(seam + ((i * t.segs + seg) * 2 + 1) * CB + V * lane, cl);
    }
    __syncthreads();
  }
  if (t.segs > 1) {
    for (int u = warp; u < rows * (t.segs - 1); u += kGatherWarps) {
      const int d = u / (t.segs - 1), seg = u - d * (t.segs - 1), b = (seg + 1) * W1 / t.segs;
      for (int j = lane; j < CB; j += 32)
        acc[(d * g.W + b - 1) * PITCH + j] += seam[(((d + 1) * t.segs + seg) * 2) * CB + j] + seam[((d * t.segs + seg) * 2 + 1) * CB + j];
    }
    __syncthreads();
  }
  const int span = rows * g.W;
  for (int c = warp; c < n_c; c += kGatherWarps) {
    T* o = dx + ((size_t)n * g.C + c0 + c) * g.HW + (size_t)r0 * g.W;
    for (int e = lane; e < span; e += 32) st<T, float>(o + e, acc[e * PITCH + c]);
  }
}

// ------------------------------------------------------------------ the other gradients, channels on the lanes
// With x, dy and the bank in channel order a corner of a sample is one line for 32 (64) channels instead of one line per lane, and
// the corner indices and fractions, worked out by one lane per sample, are shared by all channels.  Corners outside the image
// read the zero pixel, cells outside the bank its zero border, so nothing is masked.  A unit of a warp is 32 pixels of a tap.
// Offsets, with x and dy brought into channel order for it alone: 16 x 192 of 28 x 28 120 -> 70 us, 8 x 960 of 7 x 7 222 -> 33; bank
// 167 -> 62.  All gradients from one preparation: 16 x 192 of 28 x 28 531 -> 183 us, 13 x 96 of 80 x 80 2704 -> 773, fp16 13 x 88
// of 80 x 80 2424 -> 713, 64 x 384 of 14 x 14 1061 -> 300, 32 x 72 of 56 x 56 at stride 2 551 -> 265.  Bound by the load
// pipe (70 %, the forward 82 %): nine lines for 28 (14) multiply-adds; the bank gradient by the latency of five at 16 accumulators'
// registers (FMA pipe 54 %).
constexpr int kRowWarps = 8;

// byte offsets of the four corners; {1 - lh, lh, 1 - lw, lw}; for the coordinates the same of the bank and {dy, bank cell}, for the bank
// the hat functions of its rows and columns and {dy}
struct TapRec {
  int4 idx;
  float4 im, a, b;
  int4 at;
};

template <typename T, bool BANK>
__device__ __forceinline__ void tap_record(int flat, int total, int tap, const T* __restrict__ off, const T* __restrict__ rot, const Geom& g,
                                           int Cp, TapRec* to) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  TapRec r;
  const unsigned px_bytes = Cp * (unsigned)sizeof(T);
  const int nothing = (int)(g.HW * px_bytes);  // the zero pixels of the first sample
  r.idx = make_int4(nothing, nothing, nothing, nothing), r.im = r.a = r.b = zero, r.at = make_int4((int)(g.P * px_bytes), bank_unused_cell(g) * Cp * (int)sizeof(float), 0, 0);
  if (flat < total) {
    const int n = flat / g.P, p = flat - n * g.P;
    Point q;
    if (sample_point(n, tap, p, off, rot, g, q)) {
      const int base = n * (g.HW + 1);
      const bool r0 = q.h0 >= 0, r1 = q.h0 + 1 < g.H, k0 = q.w0 >= 0, k1 = q.w0 + 1 < g.W;
      const int px = q.h0 * g.W + q.w0;
      r.idx.x = (int)((base + (r0 && k0 ? px : g.HW)) * px_bytes), r.idx.y = (int)((base + (r0 && k1 ? px + 1 : g.HW)) * px_bytes);
      r.idx.z = (int)((base + (r1 && k0 ? px + g.W : g.HW)) * px_bytes), r.idx.w = (int)((base + (r1 && k1 ? px + g.W + 1 : g.HW)) * px_bytes);
      r.im = make_float4(1.f - q.lh, q.lh, 1.f - q.lw, q.lw);
      r.at.x = (int)((n * (g.P + 1) + p) * px_bytes);
      if (BANK) {
        float* hu = reinterpret_cast<float*>(&r.a);
        float* hv = reinterpret_cast<float*>(&r.b);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          hu[k] = k >= g.scH ? 0.f : k == q.u0 ? 1.f - q.lu : k == q.u0 + 1 ? q.lu : 0.f;
          hv[k] = k >= g.scW ? 0.f : k == q.v0 ? 1.f - q.lv : k == q.v0 + 1 ? q.lv : 0.f;
        }
      } else {
        r.a = make_float4(1.f - q.lu, q.lu, 1.f - q.lv, q.lv);
        r.at.y = ((q.u0 + 1) * (g.scW + 2) + q.v0 + 1) * Cp * (int)sizeof(float);
      }
    }
  }
  *to = r;
}

// Forward: a block takes 32 pixels and all their taps, a warp four of the pixels, two at a time; results pass through shared memory so that
// they are stored along the pixels.  14 multiply-adds per sample and channel.
constexpr int kForwardTaps = 9;

template <typename T, int V, bool FIXED>
__global__ void __launch_bounds__(32 * kRowWarps, 3) dcn_forward_kernel(const T* __restrict__ xt, const float* __restrict__ bankt,
                                                                        const T* __restrict__ off, const T* __restrict__ rot,
                                                                        T* __restrict__ y, const Geom g, const int Cp) {
  constexpr int CB = 32 * V;
  __shared__ TapRec recs[kForwardTaps][32];
  __shared__ float out[CB][33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, total = g.N * g.P, flat0 = blockIdx.x * 32;
  for (int i = threadIdx.x; i < g.taps * 32; i += 32 * kRowWarps)
    tap_record<T, false>(flat0 + (i & 31), total, i >> 5, off, rot, g, Cp, &recs[i >> 5][i & 31]);
  __syncthreads();
  const unsigned cell = Cp * sizeof(float), row = (g.scW + 2) * cell;
  const bool live = flat0 + lane < total;
  const int n = (flat0 + lane) / g.P, p = flat0 + lane - n * g.P;
  for (int c0 = blockIdx.y * CB; c0 < Cp; c0 += gridDim.y * CB) {
    const int c = c0 + V * lane;
    const unsigned cb = c * (unsigned)sizeof(T), ck = c * (unsigned)sizeof(float);
#pragma unroll 1
    for (int j = warp * 4; j < warp * 4 + 4; j += 2) {
      float acc[2][V] = {};
      auto taps = [&](auto select) {
#pragma unroll 1
        for (int tap = 0; tap < g.taps; ++tap) {
          float x[2][4][V], k[2][4][V];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const TapRec& r = recs[tap][j + h];
            const int4 idx = r.idx;
            const unsigned bk = r.at.y + ck;
            get_at<T, V>(xt, idx.x + cb, x[h][0]), get_at<T, V>(xt, idx.y + cb, x[h][1]), get_at<T, V>(xt, idx.z + cb, x[h][2]), get_at<T, V>(xt, idx.w + cb, x[h][3]);
            if (FIXED) {
              if (h == 0) get_at<float, V>(bankt, tap * cell + ck, k[0][0]);
            } else {
              get_at<float, V>(bankt, bk, k[h][0]), get_at<float, V>(bankt, bk + cell, k[h][1]);
              get_at<float, V>(bankt, bk + row, k[h][2]), get_at<float, V>(bankt, bk + row + cell, k[h][3]);
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 im = recs[tap][j + h].im, b = recs[tap][j + h].a;
            const bool used = !decltype(select)::value || im.x + im.y > 0.f;  // the two are 1 - lh and lh, or zeros
#pragma unroll
            for (int e = 0; e < V; ++e) {
              const float xs = im.x * (im.z * x[h][0][e] + im.w * x[h][1][e]) + im.y * (im.z * x[h][2][e] + im.w * x[h][3][e]);
              if (FIXED) acc[h][e] += xs * (used ? k[0][0][e] : 0.f);
              else acc[h][e] += xs * (b.x * (b.z * k[h][0][e] + b.w * k[h][1][e]) + b.y * (b.z * k[h][2][e] + b.w * k[h][3][e]));
            }
          }
        }
      };
      taps(std::false_type());
      if constexpr (FIXED) {
        bool finite = true;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int e = 0; e < V; ++e) finite &= fabsf(acc[h][e]) < INFINITY;
        if (!finite) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int e = 0; e < V; ++e) acc[h][e] = 0.f;
          taps(std::true_type());
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int e = 0; e < V; ++e) out[V * lane + e][j + h] = acc[h][e];
    }
    __syncthreads();
    if (live) {
      T* to = y + ((size_t)n * g.C + c0) * g.P + p;
      for (int ch = warp; ch < min(CB, g.C - c0); ch += kRowWarps) st<T, float>(to + (size_t)ch * g.P, out[ch][lane]);
    }
    __syncthreads();
  }
}

// Both offset gradients.  S warps share the channels of a unit; the sum over the lanes leaves a quarter of the four sums on each.
// 28 multiplications and additions per sample and channel, nine loads of a line.
template <typename T, int V, bool ROT, bool FIXED>
__global__ void __launch_bounds__(32 * kRowWarps, 3) dcn_coords_kernel(const T* __restrict__ dyt, const T* __restrict__ xt,
                                                                       const float* __restrict__ bankt, const T* __restrict__ off,
                                                                       const T* __restrict__ rot, T* __restrict__ doff,
                                                                       T* __restrict__ drot, const Geom g, const int Cp, const int S) {
  __shared__ TapRec recs[kRowWarps][32];
  __shared__ __align__(16) float out[kRowWarps][32][4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, share = warp % S;
  const int total = g.N * g.P, tiles = (total + 31) / 32, u = blockIdx.x * (kRowWarps / S) + warp / S;
  const int tap = u / tiles, flat0 = (u - tap * tiles) * 32, cnt = tap < g.taps ? min(32, total - flat0) : 0;
  if (cnt > 0) tap_record<T, false>(flat0 + lane, total, tap, off, rot, g, Cp, &recs[warp][lane]);
  __syncwarp();
  const unsigned cell = Cp * sizeof(float), row = (g.scW + 2) * cell;
  for (int j = 0; j < cnt; j += 2) {
    float s[2][4] = {};
    auto channels = [&](auto select) {
#pragma unroll 1
      for (int c = (share * 32 + lane) * V; c < Cp; c += S * 32 * V) {
        const unsigned cb = c * (unsigned)sizeof(T);
        float x[2][4][V], k[2][4][V], y[2][V];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const TapRec& r = recs[warp][j + h];
          const int4 idx = r.idx;
          const int2 at = *reinterpret_cast<const int2*>(&r.at);
          get_at<T, V>(xt, idx.x + cb, x[h][0]), get_at<T, V>(xt, idx.y + cb, x[h][1]), get_at<T, V>(xt, idx.z + cb, x[h][2]), get_at<T, V>(xt, idx.w + cb, x[h][3]);
          get_at<T, V>(dyt, at.x + cb, y[h]);
          const unsigned bk = at.y + c * (unsigned)sizeof(float);
          if (FIXED) {
            if (h == 0) get_at<float, V>(bankt, tap * cell + c * (unsigned)sizeof(float), k[0][0]);
          } else {
            get_at<float, V>(bankt, bk, k[h][0]), get_at<float, V>(bankt, bk + cell, k[h][1]);
            get_at<float, V>(bankt, bk + row, k[h][2]), get_at<float, V>(bankt, bk + row + cell, k[h][3]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 im = recs[warp][j + h].im, b = recs[warp][j + h].a;
          const bool used = !decltype(select)::value || im.x + im.y > 0.f;
#pragma unroll
          for (int e = 0; e < V; ++e) {
            const float top = im.z * x[h][0][e] + im.w * x[h][1][e], low = im.z * x[h][2][e] + im.w * x[h][3][e];
            const float ktop = FIXED ? 0.f : b.z * k[h][0][e] + b.w * k[h][1][e], klow = FIXED ? 0.f : b.z * k[h][2][e] + b.w * k[h][3][e];
            const float yk = y[h][e] * (FIXED ? (used ? k[0][0][e] : 0.f) : b.x * ktop + b.y * klow);
            s[h][0] += yk * (low - top);
            s[h][1] += yk * (im.x * (x[h][1][e] - x[h][0][e]) + im.y * (x[h][3][e] - x[h][2][e]));
            if (ROT) {
              const float yx = y[h][e] * (im.x * top + im.y * low);
              s[h][2] += yx * (klow - ktop);
              s[h][3] += yx * (b.x * (k[h][1][e] - k[h][0][e]) + b.y * (k[h][3][e] - k[h][2][e]));
            }
          }
        }
      }
    };
    channels(std::false_type());
    if (FIXED && !(fabsf(s[0][0]) < INFINITY && fabsf(s[0][1]) < INFINITY && fabsf(s[1][0]) < INFINITY && fabsf(s[1][1]) < INFINITY)) {
      s[0][0] = s[0][1] = s[1][0] = s[1][1] = 0.f;
      channels(std::true_type());
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float a, b;
      if (ROT) {
        const bool up = lane & 16;
        a = (up ? s[h][2] : s[h][0]) + __shfl_xor_sync(0xffffffffu, up ? s[h][0] : s[h][2], 16);
        b = (up ? s[h][3] : s[h][1]) + __shfl_xor_sync(0xffffffffu, up ? s[h][1] : s[h][3], 16);
      } else {
        a = s[h][0] + __shfl_xor_sync(0xffffffffu, s[h][0], 16);
        b = s[h][1] + __shfl_xor_sync(0xffffffffu, s[h][1], 16);
      }
      a = (lane & 8 ? b : a) + __shfl_xor_sync(0xffffffffu, lane & 8 ? a : b, 8);
      a += __shfl_xor_sync(0xffffffffu, a, 4);
      a += __shfl_xor_sync(0xffffffffu, a, 2);
      a += __shfl_xor_sync(0xffffffffu, a, 1);
      if ((lane & 7) == 0) out[warp][j + h][lane >> 3] = a;
    }
  }
  __syncthreads();
  if (share == 0 && lane < cnt) {
    float4 sum = *reinterpret_cast<const float4*>(out[warp][lane]);
    for (int k = 1; k < S; ++k) {
      const float4 o = *reinterpret_cast<const float4*>(out[warp + k][lane]);
      sum.x += o.x, sum.y += o.y, sum.z += o.z, sum.w += o.w;
    }
    const int n = (flat0 + lane) / g.P, p = flat0 + lane - n * g.P;
    const size_t o = ((size_t)n * g.taps + tap) * 2 * g.P + p;
    if (doff) st<T, float>(doff + o, sum.x), st<T, float>(doff + o + g.P, sum.y);
    if (ROT) st<T, float>(drot + o, sum.z), st<T, float>(drot + o + g.P, sum.w);
  }
}

// The units of a warp of dcn_bank_kernel again, each product to the four cells of its sample only: what a block whose sums are not
// finite does, because products that are not finite would reach all cells (times a hat of zero).  acc: [cell][channel], the lane's.
template <typename T, int V>
__device__ __noinline__ void rows_bank_by_cells(float* acc, const T* __restrict__ dyt, const T* __restrict__ xt, const T* __restrict__ off,
                                                const T* __restrict__ rot, const Geom& g, int Cp, int c, int warp) {
  constexpr int CB = 32 * V;
  for (int i = 0; i < 16; ++i)
    for (int e = 0; e < V; ++e) acc[i * CB + e] = 0.f;
  const int total = g.N * g.P, tiles = (total + 31) / 32;
  for (int u = blockIdx.x * kRowWarps + warp; u < g.taps * tiles; u += gridDim.x * kRowWarps) {
    const int tap = u / tiles, flat0 = (u - tap * tiles) * 32, cnt = min(32, total - flat0);
    for (int j = 0; j < cnt; ++j) {
      const int n = (flat0 + j) / g.P, pix = flat0 + j - n * g.P;
      Point q;
      if (!sample_point(n, tap, pix, off, rot, g, q)) continue;
      for (int e = 0; e < V; ++e) {
        float xs = 0.f;
        for (int k = 0; k < 4; ++k) {
          const int ih = q.h0 + (k >> 1), iw = q.w0 + (k & 1);
          if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W)
            xs = fmaf((k >> 1 ? q.lh : 1.f - q.lh) * (k & 1 ? q.lw : 1.f - q.lw),
                      static_cast<float>(xt[((size_t)n * (g.HW + 1) + ih * g.W + iw) * Cp + c + e]), xs);
        }
        const float dk = static_cast<float>(dyt[((size_t)n * (g.P + 1) + pix) * Cp + c + e]) * xs;
        for (int k = 0; k < 4; ++k) {
          const int a = q.u0 + (k >> 1), b = q.v0 + (k & 1);
          if (a >= 0 && a < g.scH && b >= 0 && b < g.scW)
            acc[(a * 4 + b) * CB + e] += (k >> 1 ? q.lu : 1.f - q.lu) * (k & 1 ? q.lv : 1.f - q.lv) * dk;
        }
      }
    }
  }
}

// Bank gradient without kernel-space offsets: the samples of a tap go to the same cells at every pixel, so their products are summed per tap and
// only the nine sums meet the cells.  A warp takes a run of units (32 pixels of a tap) and lays a sum down where the tap changes.
template <typename T, int V>
__global__ void __launch_bounds__(32 * kRowWarps, 3) dcn_fixed_bank_kernel(const T* __restrict__ dyt, const T* __restrict__ xt,
                                                                           const T* __restrict__ off, float* __restrict__ partial,
                                                                           const __grid_constant__ Geom g, const int Cp) {
  constexpr int CB = 32 * V;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = blockIdx.y * CB, cb = (c0 + V * lane) * (int)sizeof(T);
  TapRec* recs = reinterpret_cast<TapRec*>(smem) + warp * 32;
  float* sums = reinterpret_cast<float*>(reinterpret_cast<TapRec*>(smem) + kRowWarps * 32);  // [warp][tap][CB]
  float* mine = sums + warp * g.taps * CB + V * lane;
  for (int tap = 0; tap < g.taps; ++tap)
    for (int e = 0; e < V; ++e) mine[tap * CB + e] = 0.f;
  const int total = g.N * g.P, tiles = (total + 31) / 32, units = g.taps * tiles, runs = gridDim.x * kRowWarps, run = blockIdx.x * kRowWarps + warp;
  const int first = (int)((long long)units * run / runs), last = (int)((long long)units * (run + 1) / runs);
  float acc[V] = {};
  for (int u = first; u < last; ++u) {
    const int tap = u / tiles, flat0 = (u - tap * tiles) * 32, cnt = min(32, total - flat0);
    __syncwarp();
    tap_record<T, false>(flat0 + lane, total, tap, off, (const T*)nullptr, g, Cp, recs + lane);
    __syncwarp();
    float part[V] = {};
    for (int j = 0; j < cnt; j += 4) {
      float x[4][4][V], y[4][V];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int4 idx = recs[j + h].idx;
        get_at<T, V>(xt, idx.x + cb, x[h][0]), get_at<T, V>(xt, idx.y + cb, x[h][1]), get_at<T, V>(xt, idx.z + cb, x[h][2]), get_at<T, V>(xt, idx.w + cb, x[h][3]);
        get_at<T, V>(dyt, recs[j + h].at.x + cb, y[h]);
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float4 im = recs[j + h].im;
#pragma unroll
        for (int e = 0; e < V; ++e)
          part[e] += y[h][e] * (im.x * (im.z * x[h][0][e] + im.w * x[h][1][e]) + im.y * (im.z * x[h][2][e] + im.w * x[h][3][e]));
      }
    }
#pragma unroll
    for (int e = 0; e < V; ++e) acc[e] += part[e];
    if (u + 1 == last || (u + 1) / tiles != tap) {
#pragma unroll
      for (int e = 0; e < V; ++e) mine[tap * CB + e] = acc[e], acc[e] = 0.f;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < g.taps * CB; i += 32 * kRowWarps) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < kRowWarps; ++k) s += sums[k * g.taps * CB + i];
    sums[i] = s;  // in the first warp's room, which this thread alone has read at i
  }
  __syncthreads();
  for (int i = threadIdx.x; i < g.cells * CB; i += 32 * kRowWarps) {
    const int cell = i / CB, a = cell / g.scW, b = cell - a * g.scW, ch = i % CB;
    if (c0 + ch >= g.C) continue;
    float s = 0.f;
    for (int tap = 0; tap < g.taps; ++tap) {
      const int fh = tap / g.kW, fw = tap - fh * g.kW;
      const float u = (float)fh + (float)(g.scH - g.kH) * 0.5f, v = (float)fw + (float)(g.scW - g.kW) * 0.5f;
      const int da = a - (int)floorf(u), db = b - (int)floorf(v);  // one of the four cells of the tap's samples?
      if (da < 0 || da > 1 || db < 0 || db > 1 || !(u > -1.f && v > -1.f && u < (float)g.scH && v < (float)g.scW)) continue;
      s += (1.f - fabsf(u - (float)a)) * (1.f - fabsf(v - (float)b)) * sums[tap * CB + ch];
    }
    partial[((size_t)blockIdx.x * g.C + c0 + ch) * g.cells + cell] = s;
  }
}

// Bank gradient, dense in up to 4 x 4 cells (deform_bank_kernel with the samples taken by the lanes that use them).
template <typename T, int V>
__global__ void __launch_bounds__(32 * kRowWarps, 2) dcn_bank_kernel(const T* __restrict__ dyt, const T* __restrict__ xt,
                                                                     const T* __restrict__ off, const T* __restrict__ rot,
                                                                     float* __restrict__ partial, const __grid_constant__ Geom g, const int Cp) {
  constexpr int CB = 32 * V;
  __shared__ __align__(16) float room[kRowWarps * 16 * CB > kRowWarps * 32 * 20 ? kRowWarps * 16 * CB : kRowWarps * 32 * 20];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c0 = blockIdx.y * CB, cb = (c0 + V * lane) * (int)sizeof(T);
  TapRec* recs = reinterpret_cast<TapRec*>(room) + warp * 32;
  const int total = g.N * g.P, tiles = (total + 31) / 32;
  unsigned long long acc[V][2][4] = {};
  for (int u = blockIdx.x * kRowWarps + warp; u < g.taps * tiles; u += gridDim.x * kRowWarps) {
    const int tap = u / tiles, flat0 = (u - tap * tiles) * 32, cnt = min(32, total - flat0);
    __syncwarp();
    tap_record<T, true>(flat0 + lane, total, tap, off, rot, g, Cp, recs + lane);
    __syncwarp();
    for (int j = 0; j < cnt; j += 4) {
      float x[4][4][V], y[4][V];
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int4 idx = recs[j + h].idx;
        get_at<T, V>(xt, idx.x + cb, x[h][0]), get_at<T, V>(xt, idx.y + cb, x[h][1]), get_at<T, V>(xt, idx.z + cb, x[h][2]), get_at<T, V>(xt, idx.w + cb, x[h][3]);
        get_at<T, V>(dyt, recs[j + h].at.x + cb, y[h]);
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float4 im = recs[j + h].im, hv = recs[j + h].b;
        const ulonglong2 hu = *reinterpret_cast<const ulonglong2*>(&recs[j + h].a);
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float dk = y[h][e] * (im.x * (im.z * x[h][0][e] + im.w * x[h][1][e]) + im.y * (im.z * x[h][2][e] + im.w * x[h][3][e]));
          const float bb[4] = {dk * hv.x, dk * hv.y, dk * hv.z, dk * hv.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const unsigned long long w2 = pair(bb[k], bb[k]);
            fma2(acc[e][0][k], hu.x, w2);
            fma2(acc[e][1][k], hu.y, w2);
          }
        }
      }
    }
  }
  bool finite = true;
#pragma unroll
  for (int e = 0; e < V; ++e)
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float2 v = unpair(acc[e][i >> 2][i & 3]);
      finite &= fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY;
    }
  if (__syncthreads_or(!finite)) {
    rows_bank_by_cells<T, V>(room + warp * 16 * CB + V * lane, dyt, xt, off, rot, g, Cp, c0 + V * lane, warp);
  } else {
#pragma unroll
    for (int e = 0; e < V; ++e)
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float2 v = unpair(acc[e][i >> 2][i & 3]);
        const int cell = (i >> 2) * 8 + (i & 3);
        room[(warp * 16 + cell) * CB + V * lane + e] = v.x;
        room[(warp * 16 + cell + 4) * CB + V * lane + e] = v.y;
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 16 * CB; i += 32 * kRowWarps) {
    const int cell = i / CB, a = cell >> 2, b = cell & 3, ch = c0 + i % CB;
    if (ch < g.C && a < g.scH && b < g.scW) {
      float sum = 0.f;
#pragma unroll
      for (int k = 0; k < kRowWarps; ++k) sum += room[k * 16 * CB + i];
      partial[((size_t)blockIdx.x * g.C + ch) * g.cells + a * g.scW + b] = sum;
    }
  }
}

// ------------------------------------------------------------------ host side
size_t round256(size_t v) { return (v + 255) & ~(size_t)255; }

bool bin_plan(const Geom& g, size_t elem, BinPlan& t) {
  const long long bins = (long long)(g.H + 1) * (g.W + 1), recs = (long long)g.taps * g.P;
  // Two channels on a lane share the record and the walk through the cells (1.3 times the time of one).  A block walks R + 1
  // rows of cells, half of them at a time, in pieces so that every warp gets one; what it does besides costs about three
  // rows.  Up to 72 KB of sums, two blocks on an SM.  16 x 192 of 28 x 28: (V, R) = (1, 3) 94, (1, 7) 76, (2, 3) 75, (2, 7)
  // 75 us; 64 x 384 of 14 x 14: 219, 146, 144, 112; 4 x 64 of 50 x 84: 83, 126, 93, -, and (2, 1) 71.
  const int sms = device_sm_count();
  long long best = -1;
  for (int V = 1; V <= (g.C > 32 ? 2 : 1); ++V) {
    for (int R = 1; R < kGatherWarps; R = 2 * R + 1) {
      const int groups = (g.C + 32 * V - 1) / (32 * V), held = R < g.H ? R : g.H;
      if ((long long)held * g.W * (V == 1 ? 33 : 66) * 4 > 72 * 1024) continue;
      const long long blocks = (long long)g.N * groups * ((g.H + R - 1) / R), cost = (blocks + 2 * sms - 1) / (2 * sms) * (R + 4) * (V == 1 ? 10 : 13);
      if (best >= 0 && cost >= best) continue;
      best = cost;
      t.V = V, t.groups = groups, t.R = held, t.bands = (g.H + R - 1) / R;
      t.segs = 2 * kGatherWarps / (R + 1);
    }
  }
  t.sorts = best >= 0;
  if (!t.sorts) {
    t.V = g.C > 32 ? 2 : 1, t.groups = (g.C + 32 * t.V - 1) / (32 * t.V);
    t.R = t.bands = t.segs = 1;
  }
  if (t.segs > (g.W + 1) / 4) t.segs = (g.W + 1) / 4 > 0 ? (g.W + 1) / 4 : 1;
  const int row = g.W * (t.V == 1 ? 33 : 66) * 4;
  t.Cp = 32 * t.V * t.groups;
  if (g.G != 1 || recs > 0x3fffffff || ((long long)g.P + 1) * t.Cp > 0x7fffffff || t.groups > 65535) return false;
  if ((long long)g.N * (t.Cp / 32) * (g.P / kMovePixels + 1) > 0x3fffffff) return false;
  t.sorts = t.sorts && bins * 4 <= 160 * 1024;
  t.bins = t.sorts ? (int)bins : 0, t.rec_per_n = t.sorts ? (int)recs : 0;
  t.sort_smem = (size_t)t.bins * 4;
  t.gather_smem = (size_t)kGatherWarps * 1536 + ((size_t)bank_cells(g) * 32 * t.V + (size_t)(t.R + 1) * t.segs * 64 * t.V) * 4 + (size_t)t.R * row;
  if (t.gather_smem > 110 * 1024 || (long long)g.N * t.bands > 0x7fffffff || (long long)g.N * kSortBlocks > 0x3fffffff)
    t.sorts = false, t.bins = t.rec_per_n = 0;
  t.starts_bytes = t.sorts ? round256((size_t)g.N * (t.bins + 1) * sizeof(int)) : 0;
  t.recs_bytes = round256((size_t)g.N * t.rec_per_n * sizeof(Rec));
  t.dyt_bytes = round256((size_t)g.N * (g.P + 1) * t.Cp * elem);
  t.bytes = t.starts_bytes + t.recs_bytes + t.dyt_bytes;
  const int V = t.Cp % 64 == 0 ? 2 : 1;
  const long long units = (long long)g.taps * (((long long)g.N * g.P + 31) / 32), most = (units + kRowWarps - 1) / kRowWarps;
  t.bank_blocks = 2 * sms / (t.Cp / (32 * V));
  if (t.bank_blocks < 1) t.bank_blocks = 1;
  if (t.bank_blocks > most) t.bank_blocks = (int)most;
  t.xt_bytes = round256((size_t)g.N * (g.HW + 1) * t.Cp * elem);
  t.bankt_bytes = round256((size_t)bank_cells(g) * t.Cp * sizeof(float));
  t.all_bytes = t.bytes + t.xt_bytes + t.bankt_bytes + (size_t)t.bank_blocks * g.C * g.cells * sizeof(float);
  return true;
}
// the kernels above address all samples of x and dy with 32 bits of bytes
bool rows_shape(const Geom& g, const BinPlan& t) {
  return t.xt_bytes < 0xf0000000u && t.dyt_bytes < 0xf0000000u && (long long)g.N * g.P * g.taps < 0x3fffffff;
}

}  // namespace

bool deform_rows_gathers(const Geom& g, size_t elem) {
  BinPlan t;
  return bin_plan(g, elem, t) && t.sorts;
}
size_t deform_rows_workspace(const Geom& g, size_t elem) {
  BinPlan t;
  return bin_plan(g, elem, t) && rows_shape(g, t) ? t.all_bytes : 0;
}

template <typename T>
static int launch_bins(const T* dy, const T* x, const T* off, const T* rot, const T* w, bool sort, int* starts, Rec* recs, T* dyt, T* xt,
                       float* bankt, const Geom& g, BinPlan& t, cudaStream_t s) {
  const size_t smem = sort ? t.sort_smem : 0;
  const int rc = enable_smem(dcn_bins_kernel<T>, smem);
  if (rc) return rc;
  t.sorted = sort ? g.N : 0;
  long long tiles = dyt != nullptr ? (long long)g.N * (t.Cp / 32) * (g.P / kMovePixels + 1) : 0;
  if (xt != nullptr) tiles += (long long)g.N * (t.Cp / 32) * (g.HW / kMovePixels + 1);
  long long clusters = t.sorted + (tiles + kSortBlocks - 1) / kSortBlocks;
  if (clusters > 2 * device_sm_count() / kSortBlocks) clusters = 2 * device_sm_count() / kSortBlocks;
  if (clusters < t.sorted) clusters = t.sorted;
  if (clusters < 1) clusters = 1;
  t.movers = 3 * clusters >= 4 * (long long)t.sorted ? t.sorted * kSortBlocks : 0;
  if (clusters * kSortBlocks <= t.movers) t.movers = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * kSortBlocks));
  cfg.blockDim = dim3(kSortThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kSortBlocks, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, dcn_bins_kernel<T>, dy, off, rot, starts, recs, dyt, x, xt, w, bankt, g, t);
  if (e != cudaSuccess) {
    set_last_cuda_error(e);
    return DK_ERR_CUDA;
  }
  return check_launch();
}

template <typename T>
static int launch_gather(const T* dyt, const int* starts, const Rec* recs, const T* w, T* dx, const Geom& g, const BinPlan& t, bool fixed,
                         cudaStream_t s) {
  auto gather = fixed ? (t.V == 1 ? dcn_gather_kernel<T, 1, true> : dcn_gather_kernel<T, 2, true>)
                      : (t.V == 1 ? dcn_gather_kernel<T, 1, false> : dcn_gather_kernel<T, 2, false>);
  const int rc = enable_smem(gather, t.gather_smem);
  if (rc) return rc;
  gather<<<dim3((unsigned)(g.N * t.bands), t.groups), 32 * kGatherWarps, t.gather_smem, s>>>(dyt, starts, recs, w, dx, g, t);
  return check_launch();
}

// The wanted gradients (null: not wanted) from one pass that brings the operands into channel order.  The bank gradient, where
// the scope is larger than 4 x 4, is left to the caller (*bank_done).
template <typename T>
int deform_backward_rows(const T* dy, const T* x, const T* off, const T* rot, const T* w, T* dx, T* doff, T* drot, T* dw, const Geom& g,
                         void* ws, size_t ws_bytes, cudaStream_t s, bool* bank_done) {
  BinPlan t;
  *bank_done = false;
  const bool bank = dw != nullptr && g.scH <= 4 && g.scW <= 4, coords = doff != nullptr || drot != nullptr;
  if (!bin_plan(g, sizeof(T), t) || !rows_shape(g, t) || ws == nullptr || ws_bytes < t.all_bytes || (dx && !t.sorts)) return DK_ERR_UNSUPPORTED;
  // One gradient alone has to pay for bringing x and dy into channel order.  us, without -> with, image offsets / kernel offsets / bank:
  // 16 x 64 of 28 x 28 47 -> 34 / 75 -> 38 / 75 -> 38, 64 x 40 101 -> 107 / 162 -> 118 / 149 -> 91; stride 2, 32 x 72 of 56 x 56 101 -> 110 / 132 -> 116 /
  // 171 -> 106, 32 x 40 71 -> 75 / 94 -> 79 / 95 -> 69.  Bank alone with few pixels: 32 x 192 of 7 x 7 28 -> 28, 48 x 192 30 -> 32, 1 x 960 12 -> 19.
  if (!dx && !(coords && bank) && (g.C < 64 || (!coords && (long long)g.N * g.P < 2048))) return DK_ERR_UNSUPPORTED;
  if (!dx && !coords && !bank) return DK_ERR_UNSUPPORTED;
  char* at = reinterpret_cast<char*>(ws);
  int* starts = reinterpret_cast<int*>(at);
  Rec* recs = reinterpret_cast<Rec*>(at + t.starts_bytes);
  T* dyt = reinterpret_cast<T*>(at + t.starts_bytes + t.recs_bytes);
  T* xt = reinterpret_cast<T*>(at + t.bytes);
  float* bankt = reinterpret_cast<float*>(at + t.bytes + t.xt_bytes);
  float* partial = reinterpret_cast<float*>(at + t.bytes + t.xt_bytes + t.bankt_bytes);
  int rc = launch_bins<T>(dy, x, off, rot, w, dx != nullptr, starts, recs, dyt, coords || bank ? xt : nullptr, bankt, g, t, s);
  if (rc) return rc;
  const bool fixed = fixed_kernel(g, rot);
  if (dx && (rc = launch_gather<T>(dyt, starts, recs, w, dx, g, t, fixed, s))) return rc;
  const int V = t.Cp % 64 == 0 ? 2 : 1, groups = t.Cp / (32 * V), units = g.taps * ((g.N * g.P + 31) / 32);
  if (coords) {
    // warps share a unit's channels until there are 16 on every SM
    int S = 1;
    while (S < kRowWarps && 2 * S <= groups && (long long)units * S < 16 * device_sm_count()) S *= 2;
    auto kern = fixed ? (V == 2 ? dcn_coords_kernel<T, 2, false, true> : dcn_coords_kernel<T, 1, false, true>)
                : V == 2 ? (drot ? dcn_coords_kernel<T, 2, true, false> : dcn_coords_kernel<T, 2, false, false>)
                         : (drot ? dcn_coords_kernel<T, 1, true, false> : dcn_coords_kernel<T, 1, false, false>);
    const int per_block = kRowWarps / S;
    kern<<<(units + per_block - 1) / per_block, 32 * kRowWarps, 0, s>>>(dyt, xt, bankt, off, rot, doff, drot, g, t.Cp, S);
    if ((rc = check_launch())) return rc;
  }
  if (bank) {
    const size_t fixed_smem = kRowWarps * (32 * sizeof(TapRec) + (size_t)g.taps * 32 * V * sizeof(float));
    if (fixed && fixed_smem <= 100 * 1024) {
      auto kern = V == 2 ? dcn_fixed_bank_kernel<T, 2> : dcn_fixed_bank_kernel<T, 1>;
      if ((rc = enable_smem(kern, fixed_smem))) return rc;
      kern<<<dim3(t.bank_blocks, groups), 32 * kRowWarps, fixed_smem, s>>>(dyt, xt, off, partial, g, t.Cp);
    } else {
      auto kern = V == 2 ? dcn_bank_kernel<T, 2> : dcn_bank_kernel<T, 1>;
      kern<<<dim3(t.bank_blocks, groups), 32 * kRowWarps, 0, s>>>(dyt, xt, off, rot, partial, g, t.Cp);
    }
    if ((rc = check_launch())) return rc;
    if ((rc = reduce_bank<T>(partial, dw, g.C * g.cells, t.bank_blocks, s))) return rc;
    *bank_done = true;
  }
  return DK_OK;
}
// Forward: x and the bank into channel order, then a lane per channel.  Not where most lanes stay empty in a large call.  Lane per
// pixel -> per channel, us: 16 x 192 of 28 x 28 90 -> 56, 64 x 24 64 -> 50, 64 x 16 55 -> 50, 64 x 8 39 -> 48, 128 x 16 of 56 x 56 274 -> 296,
// 8 x 16 of 32 x 32 50 -> 22; stride 2: 32 x 128 of 56 x 56 152 -> 106, 32 x 64 102 -> 59, 32 x 40 53 -> 60, 32 x 32 59 -> 40.
static bool forward_rows(const Geom& g, size_t elem, BinPlan& t) {
  if (g.taps > kForwardTaps || !bin_plan(g, elem, t) || !rows_shape(g, t)) return false;
  return g.C >= 24 || (long long)g.N * g.P < 16384;
}
size_t deform_forward_rows_workspace(const Geom& g, size_t elem) {
  BinPlan t;
  return forward_rows(g, elem, t) ? t.xt_bytes + t.bankt_bytes : 0;
}
template <typename T>
int deform_forward_rows(const T* x, const T* off, const T* rot, const T* w, T* y, const Geom& g, void* ws, size_t ws_bytes, cudaStream_t s) {
  BinPlan t;
  if (!forward_rows(g, sizeof(T), t)) return DK_ERR_UNSUPPORTED;
  if (ws == nullptr || ws_bytes < t.xt_bytes + t.bankt_bytes) return DK_ERR_WORKSPACE;
  T* xt = reinterpret_cast<T*>(ws);
  float* bankt = reinterpret_cast<float*>(reinterpret_cast<char*>(ws) + t.xt_bytes);
  const int rc = launch_bins<T>(nullptr, x, off, rot, w, false, nullptr, nullptr, nullptr, xt, bankt, g, t, s);
  if (rc) return rc;
  const int V = t.Cp % 64 == 0 ? 2 : 1, groups = t.Cp / (32 * V), tiles = (g.N * g.P + 31) / 32;
  int split = (3 * device_sm_count() + tiles - 1) / tiles;  // blocks share the channels until there are three on every SM
  if (split > groups) split = groups;
  auto kern = fixed_kernel(g, rot) ? (V == 2 ? dcn_forward_kernel<T, 2, true> : dcn_forward_kernel<T, 1, true>)
                                   : (V == 2 ? dcn_forward_kernel<T, 2, false> : dcn_forward_kernel<T, 1, false>);
  kern<<<dim3(tiles, split), 32 * kRowWarps, 0, s>>>(xt, bankt, off, rot, y, g, t.Cp);
  return check_launch();
}
template int deform_forward_rows<float>(const float*, const float*, const float*, const float*, float*, const Geom&, void*, size_t, cudaStream_t);
template int deform_forward_rows<__half>(const __half*, const __half*, const __half*, const __half*, __half*, const Geom&, void*, size_t,
                                         cudaStream_t);
template int deform_backward_rows<float>(const float*, const float*, const float*, const float*, const float*, float*, float*, float*, float*,
                                        const Geom&, void*, size_t, cudaStream_t, bool*);
template int deform_backward_rows<__half>(const __half*, const __half*, const __half*, const __half*, const __half*, __half*, __half*, __half*,
                                         __half*, const Geom&, void*, size_t, cudaStream_t, bool*);

}  // namespace dk
