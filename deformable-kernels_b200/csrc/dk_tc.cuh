// tcgen05 (fifth-generation tensor cores, TMEM) helpers of the channel-per-lane kernels in dk_local_tc.cu.
//
// All of it is one block on one SM (cta_group::1).  The block allocates all 512 columns of TMEM; the launches ask for more
// than half of an SM's shared memory, so that two blocks never compete for them.
#pragma once

#include "dk_ring.cuh"

namespace dk {
namespace tc {

using ring::smem_u32;

// ---- TMEM allocation (one whole warp)
__device__ __forceinline__ void tmem_alloc_all(unsigned smem_slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_slot) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_free_all(unsigned addr) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(addr) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// all tcgen05.mma of this thread so far -> one arrival on `bar`
__device__ __forceinline__ void commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
// one lane of a converged warp.  The tcgen05 instructions take their operands from uniform registers: the code around them
// stays warp-uniform and only the instruction itself is under this predicate (inside an `if (lane == 0)` branch every
// operand goes through a slow move first: some 400 cycles per mma).
__device__ __forceinline__ bool elect_one() {
  unsigned ok;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(ok));
  return ok != 0;
}

// ---- descriptors
// fp16 operands, fp32 (or fp16) accumulator, M x N; tA / tB: the operand is MN-major
__host__ __device__ constexpr unsigned idesc_f16(int m, int n, bool tA, bool tB, bool f32 = true) {
  return ((unsigned)f32 << 4) | ((unsigned)tA << 15) | ((unsigned)tB << 16) | ((unsigned)(n >> 3) << 17) | ((unsigned)(m >> 4) << 24);
}
// shared-memory operand without swizzle: core matrices of 8 rows x 16 bytes, 128 contiguous bytes each; K-major: `lead` =
// bytes between core matrices along K, `stride` = along M / N
__device__ __forceinline__ uint64_t sdesc(unsigned addr, unsigned lead, unsigned stride) {
  return (uint64_t)((addr >> 4) & 0x3fff) | ((uint64_t)((lead >> 4) & 0x3fff) << 16) | ((uint64_t)((stride >> 4) & 0x3fff) << 32) |
         (1ull << 46);
}

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_ts(unsigned d, unsigned a, uint64_t b, unsigned idesc, bool acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "r"((unsigned)acc)
      : "memory");
}
// D[tmem] = D * 2^-SHIFT + A[tmem] * B[smem]
template <int SHIFT>
__device__ __forceinline__ void mma_ts_scaled(unsigned d, unsigned a, uint64_t b, unsigned idesc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.eq.u32 p, 0, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p, %4;\n}\n" ::"r"(d), "r"(a), "l"(b), "r"(idesc), "n"(SHIFT)
      : "memory");
}

// ---- TMEM <-> registers: lane l of a warp owns TMEM lane 32 (warp % 4) + l, one register per column
__device__ __forceinline__ void st8(unsigned a, const unsigned (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// 24 columns of fp32 values
__device__ __forceinline__ void ld24(unsigned (&r)[24], unsigned a) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(a));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23])
               : "r"(a + 16));
}
// 24 columns that hold one fp16 value each, two adjacent columns per register
__device__ __forceinline__ void ld24(unsigned (&r)[12], unsigned a) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.pack::16b.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(a));
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.pack::16b.b32 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11])
               : "r"(a + 16));
}
// waits for all TMEM loads of this thread; the registers named here cannot be read before it
__device__ __forceinline__ void wait_ld(unsigned (&r)[12]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11])
               :
               : "memory");
}
__device__ __forceinline__ void wait_ld(unsigned (&r)[24]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23])
               :
               : "memory");
}

// ---- register shares of the roles.  The shares of all warps must add up to no more than what the launch allocated
// (threads x compiled registers): the launchers check that before the first run.
template <int N> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(N)); }

// ---- packed fp32 pairs (pair, unpair, fma2: dk_common.cuh)
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// ---- bounded wait that also ends when another warp of the block gave up
__device__ __forceinline__ bool wait_bar(unsigned bar, unsigned parity, volatile int* abort_flag) {
  if (ring::mbar_try_wait(bar, parity)) return true;
  for (unsigned i = 0; i < ring::kMaxPolls; ++i) {
    if (ring::mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  *abort_flag = 1;
  return false;
}

}  // namespace tc
}  // namespace dk
