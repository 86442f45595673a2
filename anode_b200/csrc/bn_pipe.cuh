// What the warp-specialised kernels share: barriers in shared memory with bounded waits, bulk copies, tensor memory as a store
// for tiles, arithmetic on pairs of floats.  (bn_ring.cuh, bn_band.cuh)
#pragma once
#include "bn_device.cuh"
#include "../../include/anode_routines_gpu.h"

namespace anode_b200 {

constexpr uint32_t kBackoffNs = 100;

// ---- mbarrier / bulk-copy primitives --------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned long long *bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long *bar)
{
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long *bar, uint32_t bytes)
{
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned long long *bar, uint32_t parity)
{
  uint32_t ok;
  // the last operand lets the hardware keep the thread suspended (up to that many nanoseconds)
  // until the phase completes, instead of returning early to a polling loop
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(100000u) : "memory");
  return ok != 0;
}
// Bounded wait.  Returns false (after raising the abort flag) when the barrier did not flip in time
// or when another role already gave up.  The bound is three times `limit`, the caller's one (FusedArgs::wait_cycles, by reference: read
// from the parameters where it is compared; as a word of Ctl it cost [256,64,112,112] 0.6 %): a barrier hangs on the waits
// for words and records (twice the limit, and once), which should run out first and say in the status word what was missing.
template <typename Ctl>
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, uint32_t parity, Ctl *ctl, uint32_t *status, uint32_t bit, const long long &limit)
{
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t it = 0;
  for (;;) {
    if (mbar_try(bar, parity)) return true;
    // back off: a spinning waiter takes issue slots from the warps that do the work
    __nanosleep(kBackoffNs);
    if ((++it & 15u) == 0u) {
      if (ctl->abort) return false;
      if (clock64() - t0 > 3 * limit) {
        atomicOr(status, bit);
        ctl->abort = 1;
        return false;
      }
    }
  }
}
// Every lane gets the same answer.  The common case, a phase that is already complete (or completes while the
// hardware holds the warp), is one instruction for the whole warp; only a wait that outlasts that is handed to
// one lane, which polls with the time limit.
template <typename Ctl>
__device__ __forceinline__ bool warp_wait(unsigned long long *bar, uint32_t parity, Ctl *ctl, uint32_t *status, uint32_t bit, const long long &limit)
{
  if (__all_sync(0xffffffffu, mbar_try(bar, parity))) return true;
  uint32_t ok = 1;
  if ((threadIdx.x & 31) == 0) ok = mbar_wait(bar, parity, ctl, status, bit, limit) ? 1u : 0u;
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
// Which of its two buffers of tagged words a launch uses, for the whole warp; `warps` of them ask in every block.  The last of the grid
// to have asked turns the word for the next launch: all of this one have their answer then.  (Asked ahead of the first barrier and
// counted when a block left, that was a load, a fence and an atomic's way to L2 and back on every launch's critical path.)
__device__ __forceinline__ uint32_t buffer_of_launch(uint32_t *counter, uint32_t *word, uint32_t warps)
{
  uint32_t p = 0;
  if ((threadIdx.x & 31) == 0) {
    p = ld_acquire_gpu(word) & 1u;
    uint32_t before;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(before) : "l"(counter) : "memory");
    if (before + 1 == warps * gridDim.x) { *counter = 0; *word = p ^ 1u; }
  }
  return __shfl_sync(0xffffffffu, p, 0);
}
// global -> shared bulk copy, completion counted on `bar`; bytes and both addresses are multiples of 16
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, unsigned long long *bar, uint64_t policy)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(policy) : "memory");
}
// global -> L2; bytes and address are multiples of 16
__device__ __forceinline__ void bulk_prefetch(const void *src, uint32_t bytes)
{
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// ---- tensor memory: 512 columns of 128 lanes; a warp reaches the 32 lanes of its place in its group of four ----------
constexpr uint32_t kTmemCols = 512;
__device__ __forceinline__ void tmem_alloc(uint32_t *dst)
{
  // never waits: the launch takes the SM's whole shared memory, so that no other block holds columns (launch_ring)
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "n"(kTmemCols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base)
{
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "n"(kTmemCols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// ---- 64-bit words in global memory that other blocks poll
__device__ __forceinline__ unsigned long long ld_relaxed_gpu_u64(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_gpu_u64(unsigned long long *p, unsigned long long v)
{
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// ---- pairs of floats: one instruction for two, each rounded as its scalar form
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi)); return r; }
__device__ __forceinline__ f32x2 pair(float v) { return pair(v, v); }
__device__ __forceinline__ float2 split(f32x2 v) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v)); return r; }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) { f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r; }
__device__ __forceinline__ f32x2 slopes(f32x2 y, float slope)      // act'(y)
{
  const float2 t = split(y);
  return pair(t.x > 0.0f ? 1.0f : slope, t.y > 0.0f ? 1.0f : slope);
}
struct Quad { f32x2 a, b; };     // a 16-byte vector
__device__ __forceinline__ Quad quad(float v) { const f32x2 p = pair(v); return Quad{p, p}; }
__device__ __forceinline__ float4 floats(const Quad &q) { const float2 a = split(q.a), b = split(q.b); return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ Quad lds_quad(uint32_t saddr)
{
  Quad r;
  asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "r"(saddr) : "memory");
  return r;
}
__device__ __forceinline__ Quad ldg_quad(const float *p)
{
  Quad r;
  asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(r.a), "=l"(r.b) : "l"(p) : "memory");
  return r;
}
__device__ __forceinline__ void stg_quad(float *p, const Quad &q) { asm volatile("st.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(q.a), "l"(q.b) : "memory"); }
__device__ __forceinline__ void stg_stream(float *p, const Quad &q) { asm volatile("st.global.cs.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(q.a), "l"(q.b) : "memory"); }

// ---- tensor memory, a vector per thread and four columns (the whole warp)
#define ANODE_T16 "{t0, t1, t2, t3, t4, t5, t6, t7, t8, t9, t10, t11, t12, t13, t14, t15}"
__device__ __forceinline__ void tmem_st(uint32_t at, const Quad &a)
{
  asm volatile("{\n\t.reg .b32 t<4>;\n\tmov.b64 {t0, t1}, %1;\n\tmov.b64 {t2, t3}, %2;\n\t"
               "tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {t0, t1, t2, t3};\n\t}" ::"r"(at), "l"(a.a), "l"(a.b) : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t at, const Quad &a, const Quad &b)
{
  asm volatile("{\n\t.reg .b32 t<8>;\n\tmov.b64 {t0, t1}, %1;\n\tmov.b64 {t2, t3}, %2;\n\tmov.b64 {t4, t5}, %3;\n\tmov.b64 {t6, t7}, %4;\n\t"
               "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {t0, t1, t2, t3, t4, t5, t6, t7};\n\t}"
               ::"r"(at), "l"(a.a), "l"(a.b), "l"(b.a), "l"(b.b) : "memory");
}
__device__ __forceinline__ void tmem_st(uint32_t at, const Quad &a, const Quad &b, const Quad &c, const Quad &d)
{
  asm volatile("{\n\t.reg .b32 t<16>;\n\tmov.b64 {t0, t1}, %1;\n\tmov.b64 {t2, t3}, %2;\n\tmov.b64 {t4, t5}, %3;\n\tmov.b64 {t6, t7}, %4;\n\t"
               "mov.b64 {t8, t9}, %5;\n\tmov.b64 {t10, t11}, %6;\n\tmov.b64 {t12, t13}, %7;\n\tmov.b64 {t14, t15}, %8;\n\t"
               "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], " ANODE_T16 ";\n\t}"
               ::"r"(at), "l"(a.a), "l"(a.b), "l"(b.a), "l"(b.b), "l"(c.a), "l"(c.b), "l"(d.a), "l"(d.b) : "memory");
}
// (the wait stands in the same statement as the load, so that nothing can use a register before it has arrived)
__device__ __forceinline__ void tmem_ld(uint32_t at, Quad &a)
{
  asm volatile("{\n\t.reg .b32 t<4>;\n\ttcgen05.ld.sync.aligned.32x32b.x4.b32 {t0, t1, t2, t3}, [%2];\n\ttcgen05.wait::ld.sync.aligned;\n\t"
               "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\t}" : "=l"(a.a), "=l"(a.b) : "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t at, Quad &a, Quad &b)
{
  asm volatile("{\n\t.reg .b32 t<8>;\n\ttcgen05.ld.sync.aligned.32x32b.x8.b32 {t0, t1, t2, t3, t4, t5, t6, t7}, [%4];\n\ttcgen05.wait::ld.sync.aligned;\n\t"
               "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\tmov.b64 %2, {t4, t5};\n\tmov.b64 %3, {t6, t7};\n\t}"
               : "=l"(a.a), "=l"(a.b), "=l"(b.a), "=l"(b.b) : "r"(at) : "memory");
}
__device__ __forceinline__ void tmem_ld(uint32_t at, Quad &a, Quad &b, Quad &c, Quad &d)
{
  asm volatile("{\n\t.reg .b32 t<16>;\n\ttcgen05.ld.sync.aligned.32x32b.x16.b32 " ANODE_T16 ", [%8];\n\ttcgen05.wait::ld.sync.aligned;\n\t"
               "mov.b64 %0, {t0, t1};\n\tmov.b64 %1, {t2, t3};\n\tmov.b64 %2, {t4, t5};\n\tmov.b64 %3, {t6, t7};\n\t"
               "mov.b64 %4, {t8, t9};\n\tmov.b64 %5, {t10, t11};\n\tmov.b64 %6, {t12, t13};\n\tmov.b64 %7, {t14, t15};\n\t}"
               : "=l"(a.a), "=l"(a.b), "=l"(b.a), "=l"(b.b), "=l"(c.a), "=l"(c.b), "=l"(d.a), "=l"(d.b) : "r"(at) : "memory");
}
#undef ANODE_T16

__device__ __forceinline__ float median3(float a, float b, float c) { return fmaxf(fminf(a, b), fminf(fmaxf(a, b), c)); }

}  // namespace anode_b200
