// Shared device helpers for the tccg_b200 kernels (sm_100a only).
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>

#ifndef TCCG_DEVICE_WAIT_NS
// Upper bound of every spin-wait in the kernels (mbarrier waits): after this
// many nanoseconds of %globaltimer the wait gives up, records an error code in
// the plan's status word and the kernel winds down instead of hanging.
#define TCCG_DEVICE_WAIT_NS 4000000000ull
#endif

namespace tccg {

// Grouped launches: index of the last segment whose first CTA/tile begin[i]
// is <= t, in the ascending array begin[0..n) (begin[0] == 0). The array is
// compact (8 bytes per segment), so the search stays in L1 after the first
// CTAs of an SM touched it.
__device__ __forceinline__ int find_segment(const int64_t* __restrict__ begin, int n, int64_t t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(begin + mid) <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---- mbarrier -------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for the phase with the given parity to complete. Returns false
// when limit_ns elapsed first (the caller records an error).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity,
                                          uint64_t limit_ns = TCCG_DEVICE_WAIT_NS) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 63u) == 0 && globaltimer_ns() - t0 > limit_ns) return false;
  }
}

// ---- TMA ------------------------------------------------------------------
__device__ __forceinline__ void tma_prefetch_desc(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// 2-D tiled bulk tensor load into this CTA's shared memory, completing on `bar`.
// c0 is the innermost coordinate (elements); it must be a multiple of 16 bytes.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* tmap, int32_t c0,
                                            int32_t c1, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(c0), "r"(c1), "r"(smem_u32(bar))
      : "memory");
}

// 2-D tiled bulk tensor store from this CTA's shared memory (bulk-group
// completion); elements outside the tensor are not written. c0 as for loads.
__device__ __forceinline__ void tma_store_2d(const void* tmap, const void* smem_src, int32_t c0,
                                             int32_t c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(tmap)),
               "r"(smem_u32(smem_src)), "r"(c0), "r"(c1)
               : "memory");
}
// 1-D bulk copy global -> shared, completing on `bar`; both addresses 16-byte
// aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_load_1d(void* smem_dst, const void* gsrc, uint32_t bytes,
                                             uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
// 1-D bulk copy shared -> global (bulk-group completion); both addresses
// 16-byte aligned, bytes a multiple of 16
__device__ __forceinline__ void bulk_store_1d(void* gdst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(
                   reinterpret_cast<uint64_t>(gdst)),
               "r"(smem_u32(smem_src)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// every committed bulk copy of this thread has completed (its writes done)
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// the shared-memory source of every committed bulk store has been read
__device__ __forceinline__ void bulk_wait_read_all() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// orders this thread's generic shared-memory writes before later async-proxy
// (TMA) reads of them
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// First error code wins; the host reads it after the launch.
__device__ __forceinline__ void record_error(int32_t* status, int32_t code) {
  if (status) atomicCAS(status, 0, code);
}

// ---- programmatic dependent launch ------------------------------------------
// A kernel launched with the programmatic-stream-serialization attribute may
// start while the kernel before it on the stream is still running. It calls
// grid_dep_wait() before reading anything that kernel writes: the wait returns
// once that grid has completed and its writes are visible (at once for an
// ordinary launch). grid_dep_launch() lets the next kernel's CTAs start as
// soon as every CTA of this grid has issued it.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// ---- tcgen05 ---------------------------------------------------------------
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Whole-warp TMEM allocation; the base address is written to *slot (smem).
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(slot)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

// D[tmem] (+)= A[smem desc] * B[smem desc]^T, kind::f16 (bf16 inputs, f32 accumulate).
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                           uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem desc]^T, kind::f16: A's M = 128 rows in TMEM
// lanes, two bf16 of K per 32-bit column (the lower k in the low half).
__device__ __forceinline__ void tc_mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc,
                                              uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrive on `bar` once all previously issued tcgen05 operations of this thread completed.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns per warp (lane i <- TMEM lane base+i).
__device__ __forceinline__ void tmem_ld_32x32b_x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
}

// 32 lanes x 16 consecutive 32-bit columns per warp.
__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 32 lanes x 16 consecutive 32-bit columns per warp (lane i -> TMEM lane base+i).
__device__ __forceinline__ void tmem_st_32x32b_x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
      "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

__device__ __forceinline__ void tmem_st_wait() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major operand tile stored with the
// 128-byte swizzle (rows of 128 B, 8-row atoms of 1024 B): start address,
// LBO = 16 B (unused for swizzled K-major), SBO = 1024 B, version 1,
// layout type 2 (SWIZZLE_128B).
__device__ __forceinline__ uint64_t umma_desc_k128(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// The same for the 64-byte swizzle (rows of 64 B, 8-row atoms of 512 B):
// SBO = 512 B, layout type 4 (SWIZZLE_64B).
__device__ __forceinline__ uint64_t umma_desc_k64(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}

// Instruction descriptor of kind::f16 with BF16 A/B, FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4)                          // D format: F32
         | (1u << 7)                        // A format: BF16
         | (1u << 10)                       // B format: BF16
         | ((uint32_t)(N >> 3) << 17)       // N / 8
         | ((uint32_t)(M >> 4) << 24);      // M / 16
}

// ---- packed FP32 pairs -------------------------------------------------------
// Two FP32 values in one 64-bit register pair: x = low, y = high word.
// fma_x2 is fma.rn.f32x2: both lanes rounded as fmaf rounds one, in one
// instruction.
__device__ __forceinline__ uint64_t f32x2(float x, float y) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  return v;
}
__device__ __forceinline__ float f32x2_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f32x2_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t f32x2_swap(uint64_t v) { return f32x2(f32x2_hi(v), f32x2_lo(v)); }
__device__ __forceinline__ uint64_t fma_x2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// ---- split-BF16x3 representation ---------------------------------------------
// hi = bf16_rn(x), lo = bf16_rn(x - hi) for two values, each pair converted
// by one packed instruction (cvt.rn.bf16x2.f32): the same values as
// converting every element alone, at half the conversion instructions (the
// scalar conversion runs on the SM's narrow conversion pipe and bounded the
// operand conversion). hi / lo hold x0 in the low and x1 in the high half.
__device__ __forceinline__ void split_bf16x2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x0 - __low2float(h), x1 - __high2float(h));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// ---- three-way split of FP32 ---------------------------------------------------
// x = hi + mid + lo exactly: hi = bf16_rn(x), mid = bf16_rn(x - hi), lo =
// x - hi - mid (|x - hi| <= 2^-8 |x| and |x - hi - mid| <= 2^-17 |x|, so at
// most 7 of x's 24 significant bits are left for lo). Exact for every (scaled)
// x that f32_split_exact() accepts.
__device__ __forceinline__ void split3_bf16x2(float x0, float x1, uint32_t& hi, uint32_t& mid,
                                              uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
  const float r0 = x0 - __low2float(h), r1 = x1 - __high2float(h);
  const __nv_bfloat162 m = __floats2bfloat162_rn(r0, r1);
  const __nv_bfloat162 l = __floats2bfloat162_rn(r0 - __low2float(m), r1 - __high2float(m));
  hi = *reinterpret_cast<const uint32_t*>(&h);
  mid = *reinterpret_cast<const uint32_t*>(&m);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Magnitude range of one operand, kept by the packing pass as two words that
// shrink by atomicMin from 0xffffffff: w[0] = ~(largest |x|'s bits), w[1] =
// (smallest nonzero |x|'s bits) - 1. NaN and infinity count as the largest.
struct AbsRange {
  uint32_t not_max = 0xffffffffu, min_less1 = 0xffffffffu;
  __device__ __forceinline__ void add(float x) {
    const uint32_t b = __float_as_uint(x) & 0x7fffffffu;
    not_max = min(not_max, ~b);
    min_less1 = min(min_less1, b - 1u);  // zero wraps to 0xffffffff
  }
  // one warp's values into w (all lanes take part); the words are read first,
  // so that few warps need an atomic
  __device__ __forceinline__ void flush(uint32_t* w) {
    const uint32_t a = __reduce_min_sync(0xffffffffu, not_max);
    const uint32_t b = __reduce_min_sync(0xffffffffu, min_less1);
    if ((threadIdx.x & 31) == 0) {
      if (a < *reinterpret_cast<volatile uint32_t*>(w)) atomicMin(w, a);
      if (b < *reinterpret_cast<volatile uint32_t*>(w + 1)) atomicMin(w + 1, b);
    }
  }
};

// A contraction over K terms of operands with the range words w[0..1] and
// w[2..3] (null: not such a contraction), each multiplied by 2^shift before its
// split. With F32_SPLIT_SHIFT (2^-149, FP32's smallest step, becomes 2^-126) the
// parts of every value, subnormals too, are normal bf16 numbers or zero, so the
// split of any finite value is exact; products, scaled by 2^46, leave FP32's
// range only below 2^-172, where FP32 multiply-adds round them off as well.
// Only large values are left outside.
constexpr int F32_SPLIT_SHIFT = 23;
struct SplitRange {
  const uint32_t* w;
  int32_t K, shift;
};

// Whether its FP32 products may run as products of three-way splits: every
// value finite and, scaled, below 2^127 (the split's rounding cannot overflow),
// and no sum of scaled products near overflow: |a| |b| K below 2^78 at
// F32_SPLIT_SHIFT. With a smaller shift also: nonzero values at least 2^-100 (every
// part of the split is a normal bf16 or exact) and nonzero products at least
// 2^-100 (the dropped and the smallest kept terms stay clear of FP32's
// subnormals).
__device__ __forceinline__ bool f32_split_exact(const SplitRange& s) {
  const uint4 r = *reinterpret_cast<const uint4*>(s.w);
  const int ea = (int)(~r.x >> 23), eb = (int)(~r.z >> 23);  // biased exponents
  if (ea + s.shift >= 254 || eb + s.shift >= 254) return false;
  if (r.y == 0xffffffffu || r.w == 0xffffffffu) return true;  // an operand of zeros
  const int logk = 32 - __clz(s.K);
  if (ea - 127 + eb - 127 + 2 * s.shift + 2 + logk >= 126) return false;
  if (s.shift >= F32_SPLIT_SHIFT) return true;
  const int ma = (int)((r.y + 1u) >> 23) - 127, mb = (int)((r.w + 1u) >> 23) - 127;
  return ma >= -100 && mb >= -100 && ma + mb >= -100;
}

// ---- cp.async (SIMT kernels) ------------------------------------------------
__device__ __forceinline__ void cp_async_16(void* smem_dst, const void* gsrc) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(smem_dst)), "l"(gsrc)
               : "memory");
}
// element-wise asynchronous copy (4 or 8 bytes), for gathers through offset tables
template <int BYTES>
__device__ __forceinline__ void cp_async_elem(void* smem_dst, const void* gsrc) {
  static_assert(BYTES == 4 || BYTES == 8, "cp.async.ca copies 4, 8 or 16 bytes");
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_u32(smem_dst)), "l"(gsrc),
               "n"(BYTES)
               : "memory");
}
// the same where `in` holds, else zeros (a copy of no source bytes: nothing is
// read); without a branch
template <int BYTES>
__device__ __forceinline__ void cp_async_elem_or_zero(void* smem_dst, const void* gsrc, bool in) {
  static_assert(BYTES == 4 || BYTES == 8, "cp.async.ca copies 4, 8 or 16 bytes");
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(smem_dst)),
               "l"(gsrc), "n"(BYTES), "r"(in ? BYTES : 0)
               : "memory");
}
// the same where `in` holds, without a branch (a divergent branch per copy
// costs about 100 cycles)
__device__ __forceinline__ void cp_async_4_if(void* smem_dst, const void* gsrc, bool in) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
      "@q cp.async.ca.shared.global [%0], [%1], 4;\n\t}" ::"r"(smem_u32(smem_dst)),
      "l"(gsrc), "r"((uint32_t)in)
      : "memory");
}
__device__ __forceinline__ void cp_async_16_if(void* smem_dst, const void* gsrc, bool in) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
      "@q cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(smem_u32(smem_dst)),
      "l"(gsrc), "r"((uint32_t)in)
      : "memory");
}
// Arrive on `bar` once all of this thread's earlier cp.async copies landed
// (the barrier's expected count includes this arrival).
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t* bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void named_barrier_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}

}  // namespace tccg
