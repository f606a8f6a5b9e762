// Blackwell (sm_100a) primitives for the tensor-core contractions: mbarriers
// with bounded waits, TMA tiled loads, tcgen05 MMA / TMEM, written as inline
// PTX.  Bit layouts of the UMMA descriptors follow the PTX ISA (tcgen05
// "Matrix descriptors" and "Instruction descriptor" for kind::f16).
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace m2 {
namespace tc {

// Every wait gives up after this many polls and reports the failure; a
// correct schedule never comes near it (each poll may also suspend briefly).
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Wait for the phase with the given parity to complete; false after `limit`
// polls.
__device__ __forceinline__ bool mbar_wait_n(uint64_t* bar, uint32_t parity, uint32_t limit) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t i = 0; i < limit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) { return mbar_wait_n(bar, parity, WAIT_LIMIT); }

// 2-D tiled TMA load (no multicast) into shared memory, completing on `bar`.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------- TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols));
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem desc] * B[smem desc]^T, kind::f16 (BF16 in, FP32 acc).
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}

// Arrive on `bar` once all previously issued tcgen05.mma of this thread complete.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// 32 lanes x 16 columns of 32-bit values (one row per lane).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 bytes to a 32-byte aligned address: whole L2 sectors per lane.
__device__ __forceinline__ void st_global_32(void* p, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// One row's 16 NC values as BF16 hi and lo, whole 32-byte sectors per store;
// returns the sum of the lo parts' squares.
template <int NC>
__device__ __forceinline__ float store_split(const float* v, __nv_bfloat16* hi, __nv_bfloat16* lo) {
  float lsq = 0.0f;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    uint32_t hh[8], ll[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float f0 = v[c * 16 + 2 * e], f1 = v[c * 16 + 2 * e + 1];
      const __nv_bfloat162 h = __floats2bfloat162_rn(f0, f1);
      const __nv_bfloat162 l = __floats2bfloat162_rn(f0 - __low2float(h), f1 - __high2float(h));
      hh[e] = reinterpret_cast<const uint32_t&>(h);
      ll[e] = reinterpret_cast<const uint32_t&>(l);
      lsq = fmaf(__low2float(l), __low2float(l), lsq);
      lsq = fmaf(__high2float(l), __high2float(l), lsq);
    }
    st_global_32(hi + c * 16, hh);
    st_global_32(lo + c * 16, ll);
  }
  return lsq;
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 B,
// 8-row core groups 1024 B apart (SBO), sm_100 descriptor version 1.
__device__ __forceinline__ uint64_t sdesc_kmajor_sw128(const void* smem) {
  const uint64_t addr = smem_u32(smem);
  uint64_t d = 0;
  d |= (addr & 0x3FFFFull) >> 4;          // [0,14)  start address >> 4
  d |= (uint64_t)(16 >> 4) << 16;         // [16,30) LBO (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;       // [32,46) SBO = 1024 B
  d |= (uint64_t)1 << 46;                 // [46,48) version = 1
  d |= (uint64_t)2 << 61;                 // [61,64) SWIZZLE_128B
  return d;
}

// Shared-memory matrix descriptor: MN-major, 128-byte swizzle.  Each 128 B
// row holds 64 consecutive M (or N) elements at one k; 8 k rows form a
// 1024 B swizzle atom.  lbo_bytes: distance between 64-element M groups;
// sbo_bytes: distance between 8-row k groups.
__device__ __forceinline__ uint64_t sdesc_mnmajor_sw128(const void* smem, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  const uint64_t addr = smem_u32(smem);
  uint64_t d = 0;
  d |= (addr & 0x3FFFFull) >> 4;                          // [0,14)  start address >> 4
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;      // [16,30) LBO
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;      // [32,46) SBO
  d |= (uint64_t)1 << 46;                                 // [46,48) version = 1
  d |= (uint64_t)2 << 61;                                 // [61,64) SWIZZLE_128B
  return d;
}

// Instruction descriptor for kind::f16: BF16 x BF16 -> FP32, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4)                        // D format F32
         | (1u << 7)                      // A format BF16
         | (1u << 10)                     // B format BF16
         | ((uint32_t)(N >> 3) << 17)     // N >> 3
         | ((uint32_t)(M >> 4) << 24);    // M >> 4
}
// The same with A read MN-major (transposed A).
__host__ __device__ constexpr uint32_t idesc_bf16_f32_amn(int M, int N) { return idesc_bf16_f32(M, N) | (1u << 15); }

}  // namespace tc
}  // namespace m2
