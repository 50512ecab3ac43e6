// Blackwell (sm_100a) device primitives used by the tcgen05 kernels: mbarrier, TMA (no multicast),
// tensor-memory allocation, UMMA descriptors / issue / commit, tensor-memory loads and stores.
// Every wait is bounded: after the limit the waiter records an error code and the kernel drains.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "f32x2.cuh"

namespace sm100 {

using namespace mlstm;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier ---------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_inval(uint64_t* bar) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {   // (shared-memory address)
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool aborted(uint32_t abort) {
  uint32_t a;
  asm volatile("ld.volatile.shared::cta.u32 %0, [%1];" : "=r"(a) : "r"(abort) : "memory");
  return a != 0;
}
// Bounded wait.  Returns false if the phase did not complete within some `limit` polls, or if another role of the same
// CTA has already given up.  Two words are involved: `abort` is the CTA's own flag in shared memory (set on expiry,
// polled by every other wait of the CTA so that all roles fall through to the common exit; nullptr = never abort
// early, used where the CTA must wait for copies still in flight), `status` is the device-wide word the host reads:
// it keeps the code of the FIRST wait that ran out and is never consulted by a kernel, so one expired wait does not
// make later launches give up.
// A kernel has up to 31 waits.  Only their first polls are inlined, everything else is one function: with the limit, the sleep
// and the flags at every wait the intra-chunk kernels, whose warps go through their code once or a few times, took 3 to 7 %
// longer, waiting for instructions (8 heads, 4096 tokens 128/256: forward 19.6 -> 19.0 us, backward 41.3 -> 38.6).
constexpr uint32_t kWaitLimit = 20u * 1000u * 1000u;
__device__ __forceinline__ bool mbar_poll_on(uint32_t bar, uint32_t parity, uint32_t abort, int* status, int code, uint32_t limit) {
#pragma unroll 1
  for (uint32_t it = 0; it < limit; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    __nanosleep(32);
    if (abort != 0 && (it & 1023) == 0 && aborted(abort)) return false;
  }
  if (abort != 0) asm volatile("st.volatile.shared::cta.u32 [%0], %1;" :: "r"(abort), "r"(1u) : "memory");
  if (status != nullptr) atomicCAS(status, 0, code);
  return false;
}
static __device__ __noinline__ bool mbar_wait_long(uint32_t bar, uint32_t parity, uint32_t abort, int* status, int code,
                                                   uint32_t limit) {
  return mbar_poll_on(bar, parity, abort, status, code, limit);
}
// IN_LINE: without the call, for a role that has its registers full (the call is never made in a run that goes well, but what
// lives across it is kept where the call leaves it alone: with the call the state warps of the 128-column recurrences spilled 20 to
// 56 bytes).
template <bool IN_LINE = false>
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* abort, int* status, int code,
                                          uint32_t limit = kWaitLimit) {
  const uint32_t b = smem_u32(bar);
#pragma unroll 1
  for (int it = 0; it < 64; ++it)
    if (mbar_try_wait(b, parity)) return true;
  const uint32_t a = abort != nullptr ? smem_u32(abort) : 0u;
  return IN_LINE ? mbar_poll_on(b, parity, a, status, code, limit) : mbar_wait_long(b, parity, a, status, code, limit);
}

// Where a whole warp waits, every lane polls for itself, and a wait that runs out may do so in some lanes only: others still
// see the phase complete.  A lane that left alone would leave its warp waiting without a bound in the next warp-wide operation
// (elect, __syncwarp, shuffle, tensor-memory access).  So no lane leaves: one whose wait has run out goes on to the end of
// its role with the others, or meets them in what warp-wide operations are left; it arrives nowhere, which ends the other
// roles' waits, and what it computes is never looked at.  (A vote after each wait would let the warp leave at once; it
// measured 3-5 % of the recurrence's time and 1-2 % of the intra-chunk kernels'.)

// True in one lane of a fully active warp.  Preferred to `lane == 0` for the threads that issue copies and MMAs: the compiler
// then knows that one thread runs and keeps descriptors and coordinates in uniform registers (a TMA issue takes 15 cycles
// instead of 45).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}

// one arrival per warp, after what its lanes did before; none once a wait of the arriving lane has run out
__device__ __forceinline__ void warp_arrive(uint64_t* bar, bool ok) {
  __syncwarp();
  if (elect_one() && ok) mbar_arrive(bar);
}

// ---- proxies and fences -------------------------------------------------------------------------
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- TMA (tiled, no multicast) --------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// x = innermost coordinate (elements), y = row inside the slab, z = slab.  Rows or slabs outside the tensor are
// filled with zeros (the box may hang over the end of a slab: a ragged last chunk).
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// store of (x, row y inside slab z); elements of the box outside the tensor are not written
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}
// Untiled bulk copy global -> shared (both addresses 16-byte aligned, size a multiple of 16 bytes); completes on `bar`.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               :: "r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// ---- tensor memory ------------------------------------------------------------------------------
// Must be executed by one full warp.  ncols: power of two in [32, 512].
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ---- UMMA descriptors ---------------------------------------------------------------------------
// Shared-memory matrix descriptor, 128-byte swizzle (layout type 2), descriptor version 1.
//   K-major operand  : rows of 64 bf16 (128 B); 8-row groups 1024 B apart (SBO); LBO unused.
//   MN-major operand : 64-element (128 B) runs along M/N; K rows 128 B apart inside an 8-row group,
//                      groups SBO bytes apart; the next 64-wide M/N block LBO bytes away.
// In two words, for issuing threads that go from operand to operand by adding (bytes >> 4) to the low one: a single
// thread issues all products of a CTA, and putting a descriptor together anew for each costs it more than the issue.
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t smem_addr, uint32_t lbo_bytes) { return ((smem_addr & 0x3FFFFu) >> 4) | (lbo_bytes >> 4) << 16; }
constexpr uint32_t umma_desc_hi(uint32_t sbo_bytes) { return (sbo_bytes >> 4) | 1u << 14 | 2u << 29; }
__device__ __forceinline__ uint64_t umma_desc(uint32_t lo, uint32_t hi) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(lo), "r"(hi));
  return d;
}
// Instruction descriptor, kind::f16, 16-bit x 16-bit -> f32.  a_mn / b_mn: 1 = MN-major operand.
// f16 = false: both operands bf16 (format code 1); f16 = true: both operands IEEE half (format code 0).
__host__ __device__ constexpr uint32_t umma_idesc_16(bool f16, int M, int N, int a_mn, int b_mn) {
  return (1u << 4)                      // D format f32
         | ((f16 ? 0u : 1u) << 7)       // A format
         | ((f16 ? 0u : 1u) << 10)      // B format
         | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16)
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]; issued by ONE thread.
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accum)
      : "memory");
}
// Arrive on an mbarrier once all tcgen05 operations issued so far by this thread have completed.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

// ---- tensor memory <-> registers (warp collective; the warp touches lanes 32*(warp%4) .. +31) ----
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// Four 8 x 8 tiles of 16-bit elements out of shared memory, transposed: lane l gives the address of row l % 8 of tile l / 8 and
// gets elements (2 (l % 4), l / 4) and (2 (l % 4) + 1, l / 4) of each.
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// 16 lanes x 32 columns: lane l of the warp holds columns 4 i + l % 4 of lanes l / 4 (r[2 i]) and l / 4 + 8 (r[2 i + 1])
__device__ __forceinline__ void tmem_st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Wait for the outstanding tensor-memory loads; the registers of the load are operands of the wait so that the
// compiler cannot schedule a use of them ahead of it (needed when other work sits between the load and the wait).
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :: "memory");
}
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
// Two 16-bit elements in one 32-bit word (low half first), bf16 or IEEE half.
template <bool F16> struct Pair16 {
  static __device__ __forceinline__ uint32_t pack(float lo, float hi) { return F16 ? pack_f16(lo, hi) : pack_bf16(lo, hi); }
  static __device__ __forceinline__ void unpack(uint32_t w, float& lo, float& hi) {
    if (F16) {
      const __half2 h2 = *reinterpret_cast<const __half2*>(&w);
      lo = __low2float(h2); hi = __high2float(h2);
    } else {   // bf16 -> f32 is a 16-bit shift
      lo = __uint_as_float(w << 16); hi = __uint_as_float(w & 0xffff0000u);
    }
  }
};

// two 16-bit elements as a pair of floats, and back
template <bool F16> __device__ __forceinline__ uint64_t unpack2(uint32_t w) {
  float lo, hi;
  Pair16<F16>::unpack(w, lo, hi);
  return f2(lo, hi);
}
template <bool F16> __device__ __forceinline__ uint32_t pack2(uint64_t v) {
  float lo, hi;
  unf2(v, lo, hi);
  return Pair16<F16>::pack(lo, hi);
}

}  // namespace sm100

// ---- host side: tensor-map construction through the runtime's driver entry point ------------------
namespace sm100_host {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 16-bit tensor [slabs x rows x cols] (cols contiguous, slabs rows * cols elements apart); box = box_cols x box_rows x 1;
// 128-byte swizzle (box_cols * 2 bytes must be 128).  Out-of-range rows read as zero.
inline bool make_map_3d(CUtensorMap* map, const void* base, uint64_t slabs, uint64_t rows, uint64_t cols,
                             uint32_t box_rows, uint32_t box_cols, bool f16 = false) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  cuuint64_t dims[3] = {cols, rows, slabs};
  cuuint64_t strides[2] = {cols * 2, rows * cols * 2};
  cuuint32_t box[3] = {box_cols, box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace sm100_host
