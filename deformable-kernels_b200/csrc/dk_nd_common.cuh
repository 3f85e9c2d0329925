// Device helpers of the N-d multilinear sampler, shared by the operator kernels (dk_nd.cu) and the fused
// global deformable kernel (dk_global.cu).  Semantics: see dk_nd.cu.
#pragma once
#include <cooperative_groups.h>

#include "dk_common.cuh"

namespace dk {

template <typename A>
struct NdPoint {
  int low[kMaxNdDims];
  A frac[kMaxNdDims];
  bool valid;
};

// LDG = false reads the coordinates with plain loads (for coordinates in shared memory or written by this kernel)
template <typename T, typename A, bool LDG = true>
__device__ __forceinline__ void nd_point(const T* __restrict__ coord, int D, const NdShape& sh, NdPoint<A>& pt) {
  pt.valid = true;
#pragma unroll
  for (int d = 0; d < kMaxNdDims; ++d) {
    if (d < D) {
      const A xv = LDG ? ld<A>(coord + d) : static_cast<A>(coord[d]);
      if (xv <= (A)-1 || xv >= (A)sh.s[d]) pt.valid = false;
      if (!(xv == xv)) pt.valid = false;  // NaN samples nothing
      const A fl = dk_floor(xv);
      pt.low[d] = (int)fmin(fmax(fl, (A)-2), (A)(sh.s[d] + 1));
      pt.frac[d] = xv - fl;
    }
  }
}

// Weighted sum over the corners of one channel; GDIM >= 0 differentiates wrt that dimension.
template <typename T, typename A>
__device__ __forceinline__ A nd_gather(const T* __restrict__ data, int D, const NdShape& sh, const NdPoint<A>& pt,
                                       int gdim) {
  A val = (A)0;
  const unsigned corners = 1u << D;
  for (unsigned i = 0; i < corners; ++i) {
    int offset = 0;
    A wgt = (A)1;
    bool ok = true;
#pragma unroll
    for (int d = 0; d < kMaxNdDims; ++d) {
      if (d < D) {
        const int hi = (i >> d) & 1;
        const int pos = pt.low[d] + hi;
        ok = ok && pos >= 0 && pos <= sh.s[d] - 1;
        offset = offset * sh.s[d] + pos;
        const A f = hi ? pt.frac[d] : (A)1 - pt.frac[d];
        const A dsign = hi ? (A)1 : (A)-1;
        wgt *= (d == gdim) ? dsign : f;
      }
    }
    if (ok) val += wgt * ld<A>(data + offset);
  }
  return val;
}

// ---- gradient towards the array, shared by dk_nd.cu and dk_global.cu
//
// Lanes = 32 channels; the warps of a cluster of kNdCluster blocks split the batch.  A sample touches 2^D cells, the same
// for every channel: a warp adds its weights times dy into accumulators of its own, [cell][lane] in shared memory (no bank
// conflict, no atomics).  The warps' sums meet in the block's first accumulator, the blocks' in the first block's through
// distributed shared memory, in a fixed order.  One thread per (channel, cell) walking the whole batch instead, as before,
// is a serial chain of dependent loads: 271 us against 5.1 us at C = 256, 4 x 4 cells, 288 samples.
constexpr int kNdCluster = 8;
constexpr int kNdAccBytes = 96 * 1024;  // accumulators of a block; larger banks take fewer warps

// warps per block (0: not even one warp's accumulators fit)
template <typename A>
inline int nd_acc_warps(int prod, int batch) {
  const size_t one = (size_t)prod * 32 * sizeof(A);
  int warps = 8;
  while (warps > 1 && warps * kNdCluster > 2 * batch) warps >>= 1;
  while (warps > 1 && warps * one > (size_t)kNdAccBytes) warps >>= 1;
  return warps * one > (size_t)kNdAccBytes ? 0 : warps;
}

// acc: [warps][prod][32], zeroed here; the caller's block is one of a cluster of kNdCluster blocks, ranked `rank`.
// Whole clusters must call it.
template <typename T, typename A, bool LDG>
__device__ void nd_accumulate_bank(A* acc, const T* __restrict__ dy, const T* __restrict__ coord, T* __restrict__ ddata, int rank,
                                   int c0, int B, int C, int D, int prod, const NdShape& sh) {
  namespace cg = cooperative_groups;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  A* mine = acc + (size_t)warp * prod * 32;
  for (int i = lane; i < prod * 32; i += 32) mine[i] = (A)0;
  const int c = c0 + lane;
  const bool ok_c = c < C;
  for (int b = rank * warps + warp; b < B; b += kNdCluster * warps) {
    NdPoint<A> pt;
    nd_point<T, A, LDG>(coord + (size_t)b * D, D, sh, pt);
    if (!pt.valid) continue;
    const A g = !ok_c ? (A)0 : LDG ? ld<A>(dy + (size_t)b * C + c) : static_cast<A>(dy[(size_t)b * C + c]);
    for (unsigned i = 0; i < (1u << D); ++i) {
      int offset = 0;
      A wgt = (A)1;
      bool ok = true;
#pragma unroll
      for (int d = 0; d < kMaxNdDims; ++d) {
        if (d < D) {
          const int hi = (i >> d) & 1, pos = pt.low[d] + hi;
          ok = ok && pos >= 0 && pos <= sh.s[d] - 1;
          offset = offset * sh.s[d] + pos;
          wgt *= hi ? pt.frac[d] : (A)1 - pt.frac[d];
        }
      }
      if (ok && wgt != (A)0) mine[offset * 32 + lane] += wgt * g;
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < prod * 32; i += blockDim.x) {
    A s = acc[i];
    for (int w = 1; w < warps; ++w) s += acc[(size_t)w * prod * 32 + i];
    acc[i] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  // every block of the cluster finishes a share of the (channel, cell) pairs
  for (int i = rank * blockDim.x + threadIdx.x; i < prod * 32; i += kNdCluster * blockDim.x) {
    const int j = i / prod, cell = i - j * prod;
    if (c0 + j < C) {
      A s = (A)0;
#pragma unroll
      for (int r = 0; r < kNdCluster; ++r) s += cluster.map_shared_rank(acc, r)[cell * 32 + j];
      st<T, A>(ddata + (size_t)(c0 + j) * prod + cell, s);
    }
  }
  cluster.sync();  // no block leaves while another reads its shared memory
}

template <typename K, typename... Args>
inline int launch_nd_clusters(K kernel, unsigned clusters, int threads, size_t smem, cudaStream_t s, Args... args) {
  const int rc = enable_smem(kernel, smem);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(clusters * kNdCluster);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = kNdCluster, attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  if (e != cudaSuccess) {
    set_last_cuda_error(e);
    return DK_ERR_CUDA;
  }
  return check_launch();
}

}  // namespace dk
