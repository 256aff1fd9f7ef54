// Blackwell (sm_103a) tensor-core primitives for the BF16 kernels, written as inline PTX: tensor-memory allocation,
// tcgen05.mma (kind::f16, BF16 operands, FP32 accumulators in TMEM), tcgen05.commit to an mbarrier, tcgen05.ld,
// bulk (TMA) copies, and bounded mbarrier waits.
//
// Operand layout in shared memory: the canonical K-major, non-swizzled layout. An R x K operand (R = rows of A or of
// B^T) is stored as 8 x 8 "core matrices" (8 rows x 16 bytes): element (r, k) sits at byte
//   (r / 8) * SBO + (k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2,      SBO = K * 16
// i.e. the K-chunks of one 8-row group are adjacent (LBO = 128 bytes) and the row groups follow each other.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <cuda_bf16.h>

namespace ffno {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// byte offset of element (r, k) in a canonical K-major tile with K columns
__device__ __forceinline__ uint32_t kmajor_offset(int r, int k, int K) {
  return (uint32_t)((r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor, K-major, no swizzle (version bits 46..48 = 0b001)
__device__ __forceinline__ uint64_t kmajor_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

// instruction descriptor of tcgen05.mma kind::f16: D (F32) [M x N] += A (BF16, K-major) * B (BF16, K-major, or
// MN-major with b_mn)
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, bool b_mn = false) {
  return (1u << 4)                       // D format: F32
         | (1u << 7)                     // A format: BF16
         | (1u << 10)                    // B format: BF16
         | ((b_mn ? 1u : 0u) << 16)      // B major-ness: 0 K-major, 1 MN-major
         | ((uint32_t)(N >> 3) << 17)    // N / 8
         | ((uint32_t)(M >> 4) << 24);   // M / 16
}

// the same with either operand MN-major (A: bit 15, B: bit 16)
__host__ __device__ constexpr uint32_t idesc_bf16_ab(int M, int N, bool a_mn, bool b_mn) {
  return idesc_bf16(M, N, b_mn) | ((a_mn ? 1u : 0u) << 15);
}

// byte offset of element (n, k) of an N x K operand stored MN-major (n contiguous): 8 (k) x 16-byte core matrices,
// n-groups adjacent (SBO = 128 bytes), k-groups N * 16 bytes apart (LBO)
__device__ __forceinline__ uint32_t mnmajor_offset(int n, int k, int N) {
  return (uint32_t)((k >> 3) * (N * 16) + (n >> 3) * 128 + (k & 7) * 16 + (n & 7) * 2);
}

// shared-memory matrix descriptor of an MN-major operand (no swizzle): LBO = K-group stride, SBO = MN-group stride
__device__ __forceinline__ uint64_t mnmajor_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  return kmajor_desc(saddr, lbo_bytes, sbo_bytes);
}

// ---------------------------------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_init_fence() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Wait for the phase with this parity to complete, at most `limit` polls. Returns false if it ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t limit = (1u << 26)) {
  for (uint32_t i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// Wait for the phase with this parity, giving up after about `ns` nanoseconds of the global timer.
__device__ __forceinline__ bool mbar_wait_for(uint64_t* bar, uint32_t parity, uint64_t ns) {
  uint64_t t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (uint32_t i = 0;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 63u) {
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      if (t - t0 > ns) return false;
    }
  }
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// 16 bytes of shared memory by an explicit shared load: through a pointer that was rounded up as an integer the compiler
// emits generic loads, which queue behind the global accesses of other warps. Conversion warps, generic -> this, 2.4 M
// voxels, C = 64: gate backward 728 -> 686 us, fusion second half 855 -> 738, MLP forward with a residual 565 -> 512.
__device__ __forceinline__ float4 lds4(const void* p) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(smem_u32(p))
               : "memory");   // neither above the mbarrier wait of its stage nor below the arrival that releases it
  return v;
}

// Plain arrival (count 1) of this thread on bar.
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// ---------------------------------------------------------------------------------------------------- bulk copy
// 1-D bulk copy global -> shared completing on an mbarrier (cp.async.bulk, the TMA engine's untiled form). Both
// addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Tiled 4-D TMA load of one box of the tensor map into shared memory, completing on an mbarrier. The innermost
// coordinate c0 times the element size must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

// Tiled 2-D TMA load (box at innermost coordinate c0, row c1), completing on an mbarrier. c0 times the element size
// must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (the library does not link the driver directly);
// null if the driver does not provide it.
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
  }();
  return fn;
}

// ---------------------------------------------------------------------------------------------------- fences
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------------------------------------------- TMEM
// Allocate ncols (power of two >= 32) tensor-memory columns; one full warp calls it; the base address lands in *dst.
__device__ __forceinline__ void tmem_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_free(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---------------------------------------------------------------------------------------------------- MMA
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(tmem_d),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same with the A operand in tensor memory (lane i = row i; K packed two BF16 per 32-bit column, the lower k in
// the low half) at tmem_a.
__device__ __forceinline__ void mma_bf16_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive on bar when every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// D [128 x N] += A [128 x K] * B [N x K]^T for canonical K-major tiles at a_base / b_base (shared addresses), K a
// multiple of 16. Issued by one thread.
__device__ __forceinline__ void gemm_128xN(uint32_t tmem_d, uint32_t a_base, uint32_t b_base, int K, int N,
                                           bool accumulate) {
  const uint32_t idesc = idesc_bf16(128, N);
  for (int k = 0; k < K; k += 16) {
    const uint64_t ad = kmajor_desc(a_base + (uint32_t)(k / 8) * 128u, 128u, (uint32_t)K * 16u);
    const uint64_t bd = kmajor_desc(b_base + (uint32_t)(k / 8) * 128u, 128u, (uint32_t)K * 16u);
    mma_bf16(tmem_d, ad, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
  }
}

// D [128 x N] (+)= A [128 x K] (K-major) * B [N x K] with B stored MN-major (n contiguous, mnmajor_offset with N).
__device__ __forceinline__ void gemm_128xN_bmn(uint32_t tmem_d, uint32_t a_base, uint32_t b_base, int K, int N,
                                               bool accumulate) {
  const uint32_t idesc = idesc_bf16(128, N, true);
  for (int k = 0; k < K; k += 16) {
    const uint64_t ad = kmajor_desc(a_base + (uint32_t)(k / 8) * 128u, 128u, (uint32_t)K * 16u);
    const uint64_t bd = mnmajor_desc(b_base + (uint32_t)(k / 8) * (uint32_t)N * 16u, (uint32_t)N * 16u, 128u);
    mma_bf16(tmem_d, ad, bd, idesc, (accumulate || k > 0) ? 1u : 0u);
  }
}

// ---------------------------------------------------------------------------------------------------- TMEM -> regs
// 16 consecutive FP32 columns of this thread's lane (32x32b shape: warp w reads lanes 32w .. 32w+31).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// Store 16 consecutive FP32 columns of this thread's lane (the 32x32b shape of tmem_ld16) and wait for the store.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const float (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])), "r"(__float_as_uint(v[3])),
      "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])), "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])),
      "r"(__float_as_uint(v[8])), "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
      "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])), "r"(__float_as_uint(v[15]))
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Raw 32-bit forms without the wait (several loads or stores in flight, then one tmem_wait_ld / tmem_wait_st).
__device__ __forceinline__ void tmem_ld16u(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st8u(uint32_t taddr, const uint32_t (&v)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
               "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st16u(uint32_t taddr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
          taddr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %2, %1;" : "=r"(r) : "f"(a), "f"(b));
  return r;
}

__device__ __forceinline__ float bf16_round(float a) { return __bfloat162float(__float2bfloat16_rn(a)); }

// Split-BF16 pair of two values: hi = bf16(a), lo = bf16(a - hi), packed as (a, b) pairs. Two paired conversions:
// the rounded hi values are read back out of the packed word with integer shifts.
__device__ __forceinline__ void split_pack(float a, float b, uint32_t& hi, uint32_t& lo) {
  hi = pack_bf16(a, b);
  const float ah = __uint_as_float(hi << 16), bh = __uint_as_float(hi & 0xffff0000u);
  lo = pack_bf16(a - ah, b - bh);
}

// D [128 x N] = A B^T with split-BF16 operands (A = Ah + Al, B = Bh + Bl): Ah Bh + Ah Bl + Al Bh, FP32 accumulation.
// Relative error about 2^-16, against 2^-8 for one BF16 product. Issued by one thread.
__device__ __forceinline__ void gemm3_128xN(uint32_t tmem_d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi,
                                            uint32_t b_lo, int K, int N) {
  gemm_128xN(tmem_d, a_hi, b_hi, K, N, false);
  gemm_128xN(tmem_d, a_hi, b_lo, K, N, true);
  gemm_128xN(tmem_d, a_lo, b_hi, K, N, true);
}

// Prefetch bytes of global memory into L2 (bulk, no shared-memory destination).
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// 32 contiguous bytes (8 floats) per thread in one request, p 32-byte aligned: when every thread of a warp reads its
// own row (one voxel's channels), the warp asks for 32 sectors per request instead of 32 half sectors twice
// Volatile with a clobber: to the compiler a plain asm is a function of the pointer, free to move above the wait that makes
// the data valid (griddepcontrol.wait above all) and, issued ahead of a wait for MMAs, to sink to its use.
__device__ __forceinline__ void ld8(const float* p, float* o) {
  asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]), "=f"(o[6]), "=f"(o[7])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void st8(float* p, const float* v) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

}  // namespace tc
}  // namespace ffno
