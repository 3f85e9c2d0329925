// The global deformable kernel with a 1x1 depthwise kernel as two calls (forward, backward) instead of the ~35
// launches of its PyTorch composition (reference: modules/deform_kernel.py:76-118):
//
//   gap[n, c]   = mean over the plane of x[n, c]                                  (global average pool)
//   raw[n, d]   = fc_weight[d, :] . gap[n, :] + fc_bias[d] + tap_bias[d]           (coordinate head, D = bank dims)
//   coord[n, d] = clamp(raw[n, d], 0, shape[0] - 1)                               (the reference clamps every dim by shape[0])
//   scale[n, c] = N-d linear sample of bank[c] at coord[n]                         (dk_nd.cu semantics)
//   y[n, c]     = x[n, c] * scale[n, c]
//
// and its gradient wrt x, the bank and the head's weight and bias.  The head runs in fp32 whatever the dtype of x.
#include "dk_nd_common.cuh"

namespace dk {

namespace {

template <typename T>
__global__ void gdk_pool_kernel(const T* __restrict__ x, float* __restrict__ gap, long long planes, int hw, float inv_hw) {
  const int lane = threadIdx.x & 31;
  const long long plane = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const T* xp = x + plane * hw;
  float acc = 0.f;
  for (int i = lane; i < hw; i += 32) acc += ld<float>(xp + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) gap[plane] = acc * inv_hw;
}

// one block per sample: coordinates, then the sampled scale of every channel
__global__ void __launch_bounds__(256) gdk_head_fwd_kernel(const float* __restrict__ gap, const float* __restrict__ fc_w,
                                                           const float* __restrict__ fc_b, const float* __restrict__ tap_bias,
                                                           const float* __restrict__ bank, float* __restrict__ raw,
                                                           float* __restrict__ coord, float* __restrict__ scale, int C, int D,
                                                           int prod, const NdShape sh, float cmax) {
  __shared__ float red[8][kMaxNdDims];
  __shared__ float cs[kMaxNdDims];
  const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* g = gap + (size_t)n * C;
  float part[kMaxNdDims];
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) part[d] = 0.f;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    const float gv = g[c];
#pragma unroll
    for (int d = 0; d < kMaxNdDims; ++d)
      if (d < D) part[d] += fc_w[(size_t)d * C + c] * gv;
  }
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) {
    if (d < D) {
      float v = part[d];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][d] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < D) {
    const int d = threadIdx.x;
    float v = 0.f;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) v += red[k][d];
    v = v + fc_b[d] + tap_bias[d];
    const float cl = fminf(fmaxf(v, 0.f), cmax);
    raw[(size_t)n * D + d] = v;
    coord[(size_t)n * D + d] = cl;
    cs[d] = cl;
  }
  __syncthreads();
  NdPoint<float> pt;
  nd_point<float, float, false>(cs, D, sh, pt);
  for (int c = threadIdx.x; c < C; c += blockDim.x)
    scale[(size_t)n * C + c] = pt.valid ? nd_gather<float, float>(bank + (size_t)c * prod, D, sh, pt, -1) : 0.f;
}

template <typename T>
__global__ void gdk_apply_kernel(const T* __restrict__ x, const float* __restrict__ scale, T* __restrict__ y, long long planes,
                                 int hw) {
  const int lane = threadIdx.x & 31;
  const long long plane = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const float kv = scale[plane];
  const T* xp = x + plane * hw;
  T* yp = y + plane * hw;
  for (int i = lane; i < hw; i += 32) st<T, float>(yp + i, ld<float>(xp + i) * kv);
}

template <typename T>
__global__ void gdk_dscale_kernel(const T* __restrict__ dy, const T* __restrict__ x, float* __restrict__ dscale,
                                  long long planes, int hw) {
  const int lane = threadIdx.x & 31;
  const long long plane = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const T* gp = dy + plane * hw;
  const T* xp = x + plane * hw;
  float acc = 0.f;
  for (int i = lane; i < hw; i += 32) acc += ld<float>(gp + i) * ld<float>(xp + i);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) dscale[plane] = acc;
}

// one block per sample: gradient of the (clamped) coordinates, then of the pooled features
__global__ void __launch_bounds__(256) gdk_head_bwd_sample_kernel(const float* __restrict__ dscale, const float* __restrict__ bank,
                                                                  const float* __restrict__ raw, const float* __restrict__ coord,
                                                                  const float* __restrict__ fc_w, float* __restrict__ dcoord,
                                                                  float* __restrict__ dgap, int C, int D, int prod,
                                                                  const NdShape sh, float cmax) {
  __shared__ float red[8][kMaxNdDims];
  __shared__ float dc[kMaxNdDims];
  const int n = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  NdPoint<float> pt;
  nd_point<float, float>(coord + (size_t)n * D, D, sh, pt);
  float part[kMaxNdDims];
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) part[d] = 0.f;
  if (pt.valid) {
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      const float ds = dscale[(size_t)n * C + c];
#pragma unroll
      for (int d = 0; d < kMaxNdDims; ++d)
        if (d < D) part[d] += ds * nd_gather<float, float>(bank + (size_t)c * prod, D, sh, pt, d);
    }
  }
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) {
    if (d < D) {
      float v = part[d];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][d] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < D) {
    const int d = threadIdx.x;
    float v = 0.f;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) v += red[k][d];
    const float r = raw[(size_t)n * D + d];
    if (!(r >= 0.f && r <= cmax)) v = 0.f;  // the clamp passes the gradient inside [0, cmax] only
    dcoord[(size_t)n * D + d] = v;
    dc[d] = v;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int d = 0; d < kMaxNdDims; ++d)
      if (d < D) v += dc[d] * fc_w[(size_t)d * C + c];
    dgap[(size_t)n * C + c] = v;
  }
}

// Sums over the batch in a fixed order, a cluster of blocks per 32 channels: the bank gradient (nd_accumulate_bank), then
// the head's weight gradient (one coordinate per block at a time, the warps split the batch) and, in the first cluster,
// its bias gradient.  32 us as one thread per output walking the batch, 4 us now (C = 256, 2 x 2 cells, 32 samples).
__global__ void __launch_bounds__(256) gdk_head_bwd_param_kernel(const float* __restrict__ dscale, const float* __restrict__ coord,
                                                                 const float* __restrict__ dcoord, const float* __restrict__ gap,
                                                                 float* __restrict__ dbank, float* __restrict__ dfc_w,
                                                                 float* __restrict__ dfc_b, int N, int C, int D, int prod,
                                                                 const NdShape sh) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[8][32];
  const int rank = blockIdx.x % kNdCluster, c0 = blockIdx.x / kNdCluster * 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (dbank)
    nd_accumulate_bank<float, float, true>(reinterpret_cast<float*>(smem_raw), dscale, coord, dbank, rank, c0, N, C, D, prod, sh);
  const int c = c0 + lane;
  for (int d = rank; d < D; d += kNdCluster) {
    if (dfc_w) {
      float acc = 0.f;
      if (c < C)
        for (int n = warp; n < N; n += warps) acc += dcoord[(size_t)n * D + d] * gap[(size_t)n * C + c];
      red[warp][lane] = acc;
      __syncthreads();
      if (warp == 0 && c < C) {
        for (int w = 1; w < warps; ++w) acc += red[w][lane];
        dfc_w[(size_t)d * C + c] = acc;
      }
      __syncthreads();
    }
    if (dfc_b && c0 == 0 && warp == 0) {
      float acc = 0.f;
      for (int n = lane; n < N; n += 32) acc += dcoord[(size_t)n * D + d];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) dfc_b[d] = acc;
    }
  }
}

// The same for banks whose accumulators do not fit in shared memory: bank gradient (thread = channel x cell), head weight
// (thread = dim x channel), head bias (thread = dim), each walking the batch.
__global__ void gdk_head_bwd_param_large_kernel(const float* __restrict__ dscale, const float* __restrict__ coord,
                                                const float* __restrict__ dcoord, const float* __restrict__ gap,
                                                float* __restrict__ dbank, float* __restrict__ dfc_w, float* __restrict__ dfc_b, int N,
                                                int C, int D, int prod, const NdShape sh) {
  const long long tid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long n_bank = (long long)C * prod, n_w = (long long)D * C;
  if (tid < n_bank) {
    if (!dbank) return;
    const int cell = (int)(tid % prod), c = (int)(tid / prod);
    int pos[kMaxNdDims];
    {
      int rem = cell;
#pragma unroll
      for (int d = kMaxNdDims - 1; d >= 0; --d) {
        if (d < D) {
          pos[d] = rem % sh.s[d];
          rem /= sh.s[d];
        }
      }
    }
    float acc = 0.f;
    for (int n = 0; n < N; ++n) {
      NdPoint<float> pt;
      nd_point<float, float>(coord + (size_t)n * D, D, sh, pt);
      if (!pt.valid) continue;
      float wgt = 1.f;
#pragma unroll
      for (int d = 0; d < kMaxNdDims; ++d) {
        if (d < D) {
          const int rel = pos[d] - pt.low[d];
          wgt *= (rel == 0) ? 1.f - pt.frac[d] : (rel == 1 ? pt.frac[d] : 0.f);
        }
      }
      if (wgt != 0.f) acc += wgt * dscale[(size_t)n * C + c];
    }
    dbank[tid] = acc;
  } else if (tid < n_bank + n_w) {
    if (!dfc_w) return;
    const long long i = tid - n_bank;
    const int c = (int)(i % C), d = (int)(i / C);
    float acc = 0.f;
    for (int n = 0; n < N; ++n) acc += dcoord[(size_t)n * D + d] * gap[(size_t)n * C + c];
    dfc_w[i] = acc;
  } else if (tid < n_bank + n_w + D) {
    if (!dfc_b) return;
    const int d = (int)(tid - n_bank - n_w);
    float acc = 0.f;
    for (int n = 0; n < N; ++n) acc += dcoord[(size_t)n * D + d];
    dfc_b[d] = acc;
  }
}

template <typename T>
__global__ void gdk_dx_kernel(const T* __restrict__ dy, const float* __restrict__ scale, const float* __restrict__ dgap,
                              T* __restrict__ dx, long long planes, int hw, float inv_hw) {
  const int lane = threadIdx.x & 31;
  const long long plane = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (plane >= planes) return;
  const float kv = scale[plane], add = dgap[plane] * inv_hw;
  const T* gp = dy + plane * hw;
  T* op = dx + plane * hw;
  for (int i = lane; i < hw; i += 32) st<T, float>(op + i, ld<float>(gp + i) * kv + add);
}

// ---- whole samples on chip: one cluster of blocks per sample, each block a share of its channels
//
// The pool needs every pixel before the first scaled pixel can be written, and the gradient of the pool needs every product
// dy * x before the first pixel of dx: as launches of their own the passes read the feature map twice each way.  Where a
// sample's share fits in shared memory, a block keeps it there, the blocks exchange the head's partial sums (D floats each)
// through distributed shared memory, and the map crosses HBM once, in one launch each way.  Forward 16.2 us in three
// launches, backward 16.5 us in three, N = 32, C = 256, 14 x 14 fp32.
constexpr int kGdkThreads = 512;
constexpr size_t kGdkSmem = 200 * 1024;

__host__ __device__ inline int gdk_share(int C) { return (C + kNdCluster - 1) / kNdCluster; }
// maps: feature maps kept on chip (forward 1, backward 2); 0 bytes: the sample does not fit
template <typename T>
inline size_t gdk_cluster_smem(int C, int hw, int maps) {
  const int cc = gdk_share(C);
  const size_t map = ((size_t)cc * hw * sizeof(T) + 15) & ~(size_t)15;
  const size_t bytes = maps * map + (size_t)2 * cc * sizeof(float);
  return bytes <= kGdkSmem ? bytes : 0;
}

// `count` elements from global to shared memory, 16 bytes at a time where the source allows
template <typename T>
__device__ __forceinline__ void gdk_stage(T* dst, const T* __restrict__ src, int count) {
  constexpr int V = 16 / sizeof(T);
  int done = 0;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    const int nv = count / V;
    const int4* s4 = reinterpret_cast<const int4*>(src);
    int4* d4 = reinterpret_cast<int4*>(dst);
#pragma unroll 4
    for (int i = threadIdx.x; i < nv; i += kGdkThreads) d4[i] = __ldg(s4 + i);
    done = nv * V;
  }
#pragma unroll 4
  for (int i = done + threadIdx.x; i < count; i += kGdkThreads) dst[i] = __ldg(src + i);
}

// out[i] = map[i] * mul + add over one plane, by one warp
template <typename T>
__device__ __forceinline__ void gdk_write_plane(T* __restrict__ out, const T* map, int hw, float mul, float add, int lane) {
  constexpr int V = 16 / sizeof(T);
  if (((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(map)) & 15) == 0 && hw % V == 0) {
    for (int i = lane; i < hw / V; i += 32) {
      union { int4 q; T v[V]; } u;
      u.q = reinterpret_cast<const int4*>(map)[i];
#pragma unroll
      for (int k = 0; k < V; ++k) st<T, float>(&u.v[k], static_cast<float>(u.v[k]) * mul + add);
      reinterpret_cast<int4*>(out)[i] = u.q;
    }
  } else {
    for (int i = lane; i < hw; i += 32) st<T, float>(out + i, static_cast<float>(map[i]) * mul + add);
  }
}

// sum over the block's threads of part[0..D), then over the cluster's blocks in rank order; every thread of every block
// gets the totals in `tot` (shared).  red: [kGdkThreads / 32][kMaxNdDims], mine: this block's sums.
__device__ __forceinline__ void gdk_cluster_sum(float (&part)[kMaxNdDims], int D, float (*red)[kMaxNdDims], float* mine,
                                                float* tot) {
  namespace cg = cooperative_groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) {
    if (d < D) {
      float v = part[d];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp][d] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < D) {
    float v = 0.f;
    for (int k = 0; k < kGdkThreads / 32; ++k) v += red[k][threadIdx.x];
    mine[threadIdx.x] = v;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (threadIdx.x < D) {
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < kNdCluster; ++r) v += cluster.map_shared_rank(mine, r)[threadIdx.x];
    tot[threadIdx.x] = v;
  }
  __syncthreads();
}

template <typename T>
__global__ void __launch_bounds__(kGdkThreads) gdk_fwd_cluster_kernel(
    const T* __restrict__ x, const float* __restrict__ bank, const float* __restrict__ fc_w, const float* __restrict__ fc_b,
    const float* __restrict__ tap_bias, T* __restrict__ y, float* __restrict__ gap, float* __restrict__ raw,
    float* __restrict__ coord, float* __restrict__ scale, int C, int hw, int D, int prod, const NdShape sh, float inv_hw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[kGdkThreads / 32][kMaxNdDims];
  __shared__ float mine[kMaxNdDims], cs[kMaxNdDims];
  const int cc = gdk_share(C), rank = blockIdx.x % kNdCluster, n = blockIdx.x / kNdCluster;
  const int c0 = rank * cc, cnt = max(0, min(cc, C - c0));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T* map = reinterpret_cast<T*>(smem_raw);
  float* pooled = reinterpret_cast<float*>(smem_raw + (((size_t)cc * hw * sizeof(T) + 15) & ~(size_t)15));
  float* ks = pooled + cc;
  const size_t base = (size_t)n * C + c0;
  gdk_stage(map, x + base * hw, cnt * hw);
  __syncthreads();
  for (int j = warp; j < cnt; j += kGdkThreads / 32) {
    float acc = 0.f;
    for (int i = lane; i < hw; i += 32) acc += static_cast<float>(map[(size_t)j * hw + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      pooled[j] = acc * inv_hw;
      gap[base + j] = acc * inv_hw;
    }
  }
  __syncthreads();
  float part[kMaxNdDims];
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) part[d] = 0.f;
  for (int j = threadIdx.x; j < cnt; j += kGdkThreads) {
#pragma unroll
    for (int d = 0; d < kMaxNdDims; ++d)
      if (d < D) part[d] += __ldg(fc_w + (size_t)d * C + c0 + j) * pooled[j];
  }
  gdk_cluster_sum(part, D, red, mine, cs);
  if (threadIdx.x < D) {
    const int d = threadIdx.x;
    const float v = cs[d] + fc_b[d] + tap_bias[d], cl = fminf(fmaxf(v, 0.f), (float)(sh.s[0] - 1));
    cs[d] = cl;
    if (rank == 0) {
      raw[(size_t)n * D + d] = v;
      coord[(size_t)n * D + d] = cl;
    }
  }
  __syncthreads();
  NdPoint<float> pt;
  nd_point<float, float, false>(cs, D, sh, pt);
  for (int j = threadIdx.x; j < cnt; j += kGdkThreads) {
    ks[j] = pt.valid ? nd_gather<float, float>(bank + (size_t)(c0 + j) * prod, D, sh, pt, -1) : 0.f;
    scale[base + j] = ks[j];
  }
  __syncthreads();
  for (int j = warp; j < cnt; j += kGdkThreads / 32)
    gdk_write_plane(y + (base + j) * hw, map + (size_t)j * hw, hw, ks[j], 0.f, lane);
  cooperative_groups::this_cluster().sync();  // no block leaves while another may read its sums
}

template <typename T>
__global__ void __launch_bounds__(kGdkThreads) gdk_bwd_cluster_kernel(
    const T* __restrict__ dy, const T* __restrict__ x, const float* __restrict__ bank, const float* __restrict__ fc_w,
    const float* __restrict__ raw, const float* __restrict__ coord, const float* __restrict__ scale, T* __restrict__ dx,
    float* __restrict__ dscale, float* __restrict__ dcoord, int C, int hw, int D, int prod, const NdShape sh, float inv_hw) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float red[kGdkThreads / 32][kMaxNdDims];
  __shared__ float mine[kMaxNdDims], dc[kMaxNdDims];
  const int cc = gdk_share(C), rank = blockIdx.x % kNdCluster, n = blockIdx.x / kNdCluster;
  const int c0 = rank * cc, cnt = max(0, min(cc, C - c0));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t map_bytes = ((size_t)cc * hw * sizeof(T) + 15) & ~(size_t)15;
  T* gmap = reinterpret_cast<T*>(smem_raw);
  T* xmap = reinterpret_cast<T*>(smem_raw + map_bytes);
  float* ds = reinterpret_cast<float*>(smem_raw + 2 * map_bytes);
  const size_t base = (size_t)n * C + c0;
  gdk_stage(gmap, dy + base * hw, cnt * hw);
  gdk_stage(xmap, x + base * hw, cnt * hw);
  __syncthreads();
  for (int j = warp; j < cnt; j += kGdkThreads / 32) {
    float acc = 0.f;
    for (int i = lane; i < hw; i += 32)
      acc += static_cast<float>(gmap[(size_t)j * hw + i]) * static_cast<float>(xmap[(size_t)j * hw + i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      ds[j] = acc;
      dscale[base + j] = acc;
    }
  }
  __syncthreads();
  NdPoint<float> pt;
  nd_point<float, float>(coord + (size_t)n * D, D, sh, pt);
  float part[kMaxNdDims];
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) part[d] = 0.f;
  if (pt.valid) {
    for (int j = threadIdx.x; j < cnt; j += kGdkThreads) {
#pragma unroll
      for (int d = 0; d < kMaxNdDims; ++d)
        if (d < D) part[d] += ds[j] * nd_gather<float, float>(bank + (size_t)(c0 + j) * prod, D, sh, pt, d);
    }
  }
  gdk_cluster_sum(part, D, red, mine, dc);
  if (threadIdx.x < D) {
    const int d = threadIdx.x;
    const float r = raw[(size_t)n * D + d];
    if (!(r >= 0.f && r <= (float)(sh.s[0] - 1))) dc[d] = 0.f;  // the clamp passes the gradient inside [0, shape[0] - 1] only
    if (rank == 0) dcoord[(size_t)n * D + d] = dc[d];
  }
  __syncthreads();
  if (dx) {
    for (int j = warp; j < cnt; j += kGdkThreads / 32) {
      float dgap = 0.f;
#pragma unroll
      for (int d = 0; d < kMaxNdDims; ++d)
        if (d < D) dgap += dc[d] * __ldg(fc_w + (size_t)d * C + c0 + j);
      gdk_write_plane(dx + (base + j) * hw, gmap + (size_t)j * hw, hw, __ldg(scale + base + j), dgap * inv_hw, lane);
    }
  }
  cooperative_groups::this_cluster().sync();
}

}  // namespace

template <typename T>
int global_dk_forward(const T* x, const float* bank, const float* fc_w, const float* fc_b, const float* tap_bias, T* y,
                      float* gap, float* raw, float* coord, float* scale, int N, int C, int hw, int D, int prod,
                      const NdShape& sh, cudaStream_t s) {
  const long long planes = (long long)N * C;
  const long long blocks = (planes + 7) / 8;
  if (blocks > 0x7fffffffLL) return DK_ERR_UNSUPPORTED;
  if constexpr (sizeof(T) <= 4) {
    const size_t smem = gdk_cluster_smem<T>(C, hw, 1);
    if (smem > 0 && N <= 0x7fffffff / kNdCluster)
      return launch_nd_clusters(gdk_fwd_cluster_kernel<T>, (unsigned)N, kGdkThreads, smem, s, x, bank, fc_w, fc_b, tap_bias, y, gap,
                                raw, coord, scale, C, hw, D, prod, sh, 1.f / (float)hw);
  }
  gdk_pool_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(x, gap, planes, hw, 1.f / (float)hw);
  gdk_head_fwd_kernel<<<N, 256, 0, s>>>(gap, fc_w, fc_b, tap_bias, bank, raw, coord, scale, C, D, prod, sh,
                                        (float)(sh.s[0] - 1));
  gdk_apply_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(x, scale, y, planes, hw);
  return check_launch();
}

template <typename T>
int global_dk_backward(const T* dy, const T* x, const float* bank, const float* fc_w, const float* gap, const float* raw,
                       const float* coord, const float* scale, T* dx, float* dbank, float* dfc_w, float* dfc_b, float* ws,
                       int N, int C, int hw, int D, int prod, const NdShape& sh, cudaStream_t s) {
  const long long planes = (long long)N * C;
  const long long blocks = (planes + 7) / 8;
  if (blocks > 0x7fffffffLL) return DK_ERR_UNSUPPORTED;
  float* dscale = ws;
  float* dgap = dscale + planes;
  float* dcoord = dgap + planes;
  size_t smem = 0;
  if constexpr (sizeof(T) <= 4) smem = N <= 0x7fffffff / kNdCluster ? gdk_cluster_smem<T>(C, hw, 2) : 0;
  if (smem > 0) {
    if constexpr (sizeof(T) <= 4) {
      const int rc = launch_nd_clusters(gdk_bwd_cluster_kernel<T>, (unsigned)N, kGdkThreads, smem, s, dy, x, bank, fc_w, raw, coord,
                                        scale, dx, dscale, dcoord, C, hw, D, prod, sh, 1.f / (float)hw);
      if (rc) return rc;
    }
  } else {
    gdk_dscale_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(dy, x, dscale, planes, hw);
    gdk_head_bwd_sample_kernel<<<N, 256, 0, s>>>(dscale, bank, raw, coord, fc_w, dcoord, dgap, C, D, prod, sh,
                                                 (float)(sh.s[0] - 1));
  }
  if (dbank || dfc_w || dfc_b) {
    const int warps = nd_acc_warps<float>(prod, N);
    if (warps > 0) {
      const int rc = launch_nd_clusters(gdk_head_bwd_param_kernel, (unsigned)((C + 31) / 32), 32 * warps,
                                        (size_t)warps * prod * 32 * sizeof(float), s, (const float*)dscale, coord,
                                        (const float*)dcoord, gap, dbank, dfc_w, dfc_b, N, C, D, prod, sh);
      if (rc) return rc;
    } else {
      const long long work = (long long)C * prod + (long long)D * C + D;
      gdk_head_bwd_param_large_kernel<<<(unsigned)((work + 127) / 128), 128, 0, s>>>(dscale, coord, dcoord, gap, dbank, dfc_w,
                                                                                    dfc_b, N, C, D, prod, sh);
    }
  }
  if (dx && smem == 0) gdk_dx_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(dy, scale, dgap, dx, planes, hw, 1.f / (float)hw);
  return check_launch();
}

#define DK_INSTANTIATE_GLOBAL(T)                                                                                          \
  template int global_dk_forward<T>(const T*, const float*, const float*, const float*, const float*, T*, float*, float*,  \
                                    float*, float*, int, int, int, int, int, const NdShape&, cudaStream_t);                \
  template int global_dk_backward<T>(const T*, const T*, const float*, const float*, const float*, const float*,           \
                                     const float*, const float*, T*, float*, float*, float*, float*, int, int, int, int,  \
                                     int, const NdShape&, cudaStream_t);
DK_INSTANTIATE_GLOBAL(float)
DK_INSTANTIATE_GLOBAL(__half)
DK_INSTANTIATE_GLOBAL(double)

}  // namespace dk
