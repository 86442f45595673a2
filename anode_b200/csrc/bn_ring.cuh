// Warp-specialised version of the fused batch-norm pipeline for the 128-bit paths.
//
// Same algorithm as bn_fused.cuh (reduce a tile, complete its unit, apply the tile a bounded
// number of steps later), but no consumer thread ever waits on global memory:
//
//   producer warp    walks the block's schedule and streams tiles into a ring of shared-memory
//                    slots with bulk asynchronous copies (cp.async.bulk + mbarrier), tagged
//                    with L2 eviction hints: "keep" for the reduce visit, "drop" for the
//                    apply visit.  The ring keeps HBM requests in flight while everything
//                    else happens.  Each slot carries a description of its visit.
//   consumer warps   (8 or 16) read slots with 128-bit shared loads, accumulate / normalise, write
//                    results with 128-bit streaming stores, and hand partials to the delivery
//                    warp through a shared-memory mailbox.  Every warp works on its
//                    own share of a tile and never synchronises with the other warps.  Of most
//                    tiles the reduce visit leaves what it read in TENSOR MEMORY (256 KB per SM,
//                    37 MB on the device), from where the apply visit takes it: no second trip
//                    through L2 and no slot.
//   delivery warp    merges the consumer warps' partials of a tile and stores them as ONE tagged
//                    8-byte word per tile in the workspace (no counter, no fence, no atomic).
//   coefficient warp polls, for each upcoming apply visit, the partial words of the visit's
//                    channel until none is zero, merges them in a fixed order in double
//                    precision (every block obtains bit-identical coefficients; with several
//                    GPUs the owner block exchanges per-GPU records with the peers here) and
//                    stages the visit's coefficients and description in a second mailbox.
//                    (In the three-launch form of the synchronized calls the reduce launch still counts
//                    partials per unit and the apply launch reads prepared coefficients.)
//
// What bounds it: the first visits' loads and the stores where all of a window stays in tensor memory, and on the way there
// the instructions of the consumers and the merge of a channel's partials.  Forward / backward in us, with every second visit
// from L2, with tensor memory, with descriptions and pairs on top, with the shorter merge on top: [256,64,112,112] 301 / 495,
// 370 / 595, 281 / 436, 276 / 420; [2048,256,56,56] 2555 / 4362, 2446 / 4371, 2197 / 3763, 2134 / 3347;
// [4,32,128,128,128] 454 / 737, 389 / 634, 372 / 621, 350 / 598.  (Tensor memory alone was no gain: its stores and loads
// came on top of 23 / 55 instructions per element, where 10 / 16 are arithmetic.)
//
// Every wait is bounded: a wait that runs out sets a status bit, raises the block's abort flag
// and all three roles drain and leave.
// This header has no include guard on purpose: it is included once per consumer-warp count, with
// ANODE_RING_NS naming the namespace of the instantiation and ANODE_RING_CONSUMERS the number of
// consumer threads (the forward pass runs best with 8 consumer warps, the backward pass with 16).
#include "bn_fused.cuh"
#include "bn_pipe.cuh"

#if !defined(ANODE_RING_NS) || !defined(ANODE_RING_CONSUMERS)
#error "define ANODE_RING_NS and ANODE_RING_CONSUMERS before including bn_ring.cuh"
#endif

namespace anode_b200 {
namespace ANODE_RING_NS {

constexpr uint32_t kConsumers = ANODE_RING_CONSUMERS;   // consumer threads (a power of two, 256..1024)
constexpr uint32_t kRingThreads = kConsumers + 96;   // + producer, delivery and coefficient warps

struct RingCtl {
  unsigned long long full[kMaxSlots], empty[kMaxSlots];
  unsigned long long res_full[kResQ], res_empty[kResQ];
  unsigned long long coef_full[kCoefQ], coef_empty[kCoefQ];
  volatile uint32_t abort;
  uint32_t parity;       // which of the two tagged-partial buffers this launch uses
  uint32_t tmem;         // base address of the block's tensor memory (g.keep_slots > 0)
};
static_assert(sizeof(RingCtl) <= kRingCtlBytes, "RingCtl outgrew the room reserved for it");

// ---- tensor memory as a store for tiles ---------------------------------------------------------
// The SM's 256 KB of tensor memory hold what the reduce visits of `keep_slots` out of every keep_period tiles have read
// (forward: x; backward: x - mean and dz), so that their apply visits need neither L2 nor a slot of the ring.  A warp
// reaches the 32 lanes of its place in its group of four warps; the groups divide the 512 columns among them.
// Every instruction here is the whole warp's.
// ---- the block's schedule --------------------------------------------------------------------
// The visits of a block: steps s = 0, 1, ...; at step s first REDUCE its tile number s (if any is left), then APPLY number
// s - look (if s >= look).  Tile number n of the block is tile b + n*G.  Every role walks this same sequence by itself.
struct Sched {
  uint32_t my_tiles, look, b, G;
  uint32_t steps, reduces, applies;       // steps, reduce visits, apply visits
  __device__ __forceinline__ void init(const FusedArgs &a)
  {
    b = blockIdx.x; G = gridDim.x;
    my_tiles = (b < a.plan.total_tiles) ? (a.plan.total_tiles - b + G - 1) / G : 0;
    look = (a.mode == MODE_FUSED) ? a.plan.lookahead_steps : 0;
    steps = my_tiles + look;
    reduces = a.mode != MODE_APPLY ? my_tiles : 0; applies = a.mode != MODE_STATS ? my_tiles : 0;
  }
  __device__ __forceinline__ bool reduce_at(uint32_t s) const { return s < reduces; }
  __device__ __forceinline__ bool apply_at(uint32_t s) const { return s >= look && s - look < applies; }
};

// dynamic shared memory accessors
__device__ __forceinline__ float *slot_x(unsigned char *sm, const RingGeom &g, uint32_t slot) { return reinterpret_cast<float *>(sm + g.off_slots + (size_t)slot * g.slot_stride); }
// a slot holds kPlanes tensors side by side: x, then dy (backward), then the residual (forward) / saved output (backward)
template <int DIR, bool EXTRA> constexpr uint32_t kPlanes = (DIR == 1 ? 2u : 1u) + (EXTRA ? 1u : 0u);
// an apply visit from tensor memory needs a slot only for the residual
template <int DIR, bool EXTRA> constexpr bool kSlotAlways = DIR == 0 && EXTRA;
// behind the planes: the visit (reduce visits only) and, in the backward pass, (mean, scale, beta) of its channel
template <int DIR, bool EXTRA> __device__ __forceinline__ float4 *slot_side(unsigned char *sm, const RingGeom &g, uint32_t slot)
{
  return reinterpret_cast<float4 *>(slot_x(sm, g, slot) + kPlanes<DIR, EXTRA> * g.slot_floats);
}
__device__ __forceinline__ float4 *res_box(unsigned char *sm, const RingGeom &g, uint32_t q) { return reinterpret_cast<float4 *>(sm + g.off_res) + (size_t)q * g.res_stride; }
// a mailbox entry of the coefficient warp: (mean, scale, beta, cB), (cC, -, -, -), the visit
__device__ __forceinline__ float4 *coef_box(unsigned char *sm, const RingGeom &g, uint32_t q) { return reinterpret_cast<float4 *>(sm + g.off_coef) + q * kCoefBox; }

// ======================================================================================
// consumer side
// ======================================================================================
// What bounds the consumers is the instructions they issue: a visit is three or four vectors per thread in the backward
// pass, so whatever is done once per visit weighs as much as the arithmetic.  Hence the visit's range comes ready-made from
// the service warps (one 16-byte word), arithmetic is two floats per instruction, and places are found by adding up.
// Instructions per element, [256,16,112,112]: forward 23, backward 55 when every warp walked the schedule by itself.
constexpr uint32_t kCWarps = kConsumers / 32;
constexpr uint32_t kVecStride = kConsumers * 16;     // bytes between consecutive vectors of one thread

// Shift of the sums: the median of three elements.  A single one is no shift to rely on: the first of an image is the corner
// that a zero-padded convolution makes, and far from the mean it costs the variance its digits.  Relative error of the
// variance with the first element of each row at 100 standard deviations, that element and the median as the shift:
// [64,12,55,55] 7.7e-5 and 9e-8, [64,8,56,56] 2.7e-5 and 9e-8.  Aligned rows take the elements from the warp's first
// vector, ragged ones from the tile's beginning, middle and end.  (Aligned rows with the latter, the residual epilogue's
// forward pass on [256,256,56,56]: 522 -> 560 us, although each warp does less; with the former 526.  A mean of the warp's
// first vectors: 542 - 570.)

// Backward pass of the residual epilogue: dres = dz leaves during the reduce visit and the apply visit reads it back
// (from L2) in the place of dy and the saved output, unless there is no dres or it is x itself (FusedArgs::dres_early).
// The read is a bulk copy, hence the fence between the two proxies before the slot is given back.
__device__ __forceinline__ void fence_global_to_bulk() { asm volatile("fence.proxy.async.global;" ::: "memory"); }

// A visit, as the service warps describe it to the consumers (16 bytes): its vectors, its place in tensor memory + 1 (0:
// none), the float offset of its first element (below 2^32, check_dims), floats per row, rows.
// The service warps work 32 of them out at a time, one per lane: one after another they took the producer a microsecond
// each, more than its copies, and bounded tiles of less than 32 KB.
__device__ __forceinline__ uint4 describe(const TileRange &tr, bool ragged, const Keep &keep)
{
  const uint32_t nvec = (ragged ? ragged_pitch(tr.len) : tr.len / 4) * tr.rows;
  return make_uint4(nvec | (keep.kept ? keep.slot + 1u : 0u) << 16, (uint32_t)tr.base, tr.len, tr.rows);
}
__device__ __forceinline__ uint4 shfl4(const uint4 &v, uint32_t lane)
{
  return make_uint4(__shfl_sync(0xffffffffu, v.x, lane), __shfl_sync(0xffffffffu, v.y, lane), __shfl_sync(0xffffffffu, v.z, lane),
                    __shfl_sync(0xffffffffu, v.w, lane));
}

// The visit as one thread sees it: its vectors are tid, tid + kConsumers, ... of the tile's rows laid back to back (`cnt` of
// them; the warp's lane with the most has `steps`), kept in tensor memory from column `tm` on.
template <bool KEEP>
struct Mine {
  uint32_t tid, cnt, steps, tm;
  __device__ __forceinline__ Mine(const RingGeom &g, const RingCtl *ctl, const uint4 &d)
  {
    tid = threadIdx.x; tm = 0;
    const uint32_t nvec = d.x & 0xffffu;
    if constexpr (KEEP) {
      const uint32_t warp = tid >> 5;
      uint32_t dealt, column;
      keep_place(g, (d.x >> 16) - 1, warp, kCWarps, dealt, column);
      tid = dealt * 32 + (tid & 31);
      tm = ctl->tmem + ((warp & 3u) << 21) + (warp >> 2) * (kTmemCols * 4 / kCWarps) + column;
    }
    cnt = (nvec + kConsumers - 1 - tid) / kConsumers;
    steps = (nvec + kConsumers - 1 - (tid & ~31u)) / kConsumers;
  }
};

// Places of a thread's vectors in global memory: a step is an add and a compare, without a division or a 64-bit product.
// (Ragged rows: `at` is the row's first float plus 4 * col, whose last two bits say how far into a vector the row starts.)
struct Walk {
  uint32_t at, col;
  __device__ __forceinline__ Walk(const FusedArgs &a, const RingGeom &g, uint32_t base, uint32_t tid)
  {
    const uint32_t r = __umulhi(tid, g.walk_mul);
    col = tid - r * g.walk_per; at = base + r * (a.plan.C * a.plan.dim0) + 4 * col;
  }
  __device__ __forceinline__ void advance(const RingGeom &g)
  {
    at += g.walk_step; col += g.walk_col;
    if (col >= g.walk_per) { col -= g.walk_per; at += g.walk_wrap; }
  }
  __device__ __forceinline__ uint32_t vector() const { return at & ~3u; }                         // ragged rows: the vector
  __device__ __forceinline__ int first() const { return (int)(4 * col) - (int)(at & 3u); }        // and its first float's place in the row
};

template <int DIR, bool EXTRA, bool RAGGED, bool KEEP>
__device__ __forceinline__ void visit_reduce(const FusedArgs &a, const RingGeom &g, unsigned char *sm, RingCtl *ctl,
                                             const uint4 &d, uint32_t slot, float4 *res)
{
  const uint32_t lane = threadIdx.x & 31;
  const Mine<KEEP> mine(g, ctl, d);
  const uint32_t cnt = mine.cnt, steps = mine.steps;
  const float *xs = slot_x(sm, g, slot);
  uint32_t ax = smem_u32(xs) + mine.tid * 16, tm = mine.tm;
  const int len = (int)d.z;
  float4 out;
  if constexpr (DIR == 0) {
    // shifted sums (see bn_fused.cuh); one shift per warp makes them plain sums over lanes
    float K = 0.f;
    uint32_t n = 0;
    f32x2 sa = 0, sb = 0, qa = 0, qb = 0;
    if constexpr (!RAGGED) {
      if (steps) { const float4 v0 = floats(lds_quad(ax - lane * 16)); K = median3(v0.x, v0.y, v0.z); }
      const f32x2 nK = pair(-K);
      auto take = [&](const Quad &v) {
        const f32x2 da = add2(v.a, nK), db = add2(v.b, nK);
        sa = add2(sa, da); qa = fma2(da, da, qa); sb = add2(sb, db); qb = fma2(db, db, qb);
      };
      uint32_t i = 0;
      for (; i + 4 <= steps; i += 4, ax += 4 * kVecStride, tm += 16) {
        // (the lanes differ in their last vector only; a missing one is K)
        const Quad v0 = lds_quad(ax), v1 = lds_quad(ax + kVecStride), v2 = lds_quad(ax + 2 * kVecStride);
        Quad v3 = quad(K);
        if (i + 3 < cnt) v3 = lds_quad(ax + 3 * kVecStride);
        if constexpr (KEEP) { __syncwarp(); tmem_st(tm, v0, v1, v2, v3); }
        take(v0); take(v1); take(v2); take(v3);
      }
      for (; i < steps; ++i, ax += kVecStride, tm += 4) {
        Quad v0 = quad(K);
        if (i < cnt) v0 = lds_quad(ax);
        if constexpr (KEEP) { __syncwarp(); tmem_st(tm, v0); }
        take(v0);
      }
      // the warp's vectors: whole steps, and what the last one has
      if (steps) { const uint32_t left = (d.x & 0xffffu) - (mine.tid & ~31u) - (steps - 1) * kConsumers; n = 128 * (steps - 1) + 4 * (left < 32 ? left : 32); }
    } else {
      const uint32_t per_row = ragged_pitch(d.z), first = d.y, rs = a.plan.C * a.plan.dim0, rm = d.w / 2, rl = d.w - 1;
      K = median3(xs[(first & 3u) + d.z / 6], xs[4 * per_row * rm + ((first + rm * rs) & 3u) + d.z / 2],
                  xs[4 * per_row * rl + ((first + rl * rs) & 3u) + d.z - 1 - d.z / 6]);
      const f32x2 nK = pair(-K);
      Walk w(a, g, first, mine.tid);
      auto take = [&](const Quad &v, bool live) {
        const int i0 = live ? w.first() : len;
        Quad e{add2(v.a, nK), add2(v.b, nK)};
        if (ragged_whole(i0, len)) {
          n += 4;
        } else {      // foreign floats at a row's ends count nothing
          const float4 t = floats(e);
          auto own = [&](float f, int k) { const bool in = (uint32_t)(i0 + k) < (uint32_t)len; n += in; return in ? f : 0.f; };
          e.a = pair(own(t.x, 0), own(t.y, 1)); e.b = pair(own(t.z, 2), own(t.w, 3));
        }
        sa = add2(sa, e.a); qa = fma2(e.a, e.a, qa); sb = add2(sb, e.b); qb = fma2(e.b, e.b, qb);
        w.advance(g);
      };
      uint32_t i = 0;
      for (; i + 4 <= steps; i += 4, ax += 4 * kVecStride, tm += 16) {
        const Quad v0 = lds_quad(ax), v1 = lds_quad(ax + kVecStride), v2 = lds_quad(ax + 2 * kVecStride);
        Quad v3 = quad(K);
        if (i + 3 < cnt) v3 = lds_quad(ax + 3 * kVecStride);
        if constexpr (KEEP) { __syncwarp(); tmem_st(tm, v0, v1, v2, v3); }
        take(v0, true); take(v1, true); take(v2, true); take(v3, i + 3 < cnt);
      }
      for (; i < steps; ++i, ax += kVecStride, tm += 4) {
        Quad v = quad(K);
        if (i < cnt) v = lds_quad(ax);
        if constexpr (KEEP) { __syncwarp(); tmem_st(tm, v); }
        take(v, i < cnt);
      }
      n = __reduce_add_sync(0xffffffffu, n);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&ctl->empty[slot]);
    const float2 st = split(add2(sa, sb)), qt = split(add2(qa, qb));
    const float s = warp_sum(st.x + st.y), q = warp_sum(qt.x + qt.y);
    out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n) {
      out.x = (float)n;
      const float inv = __fdividef(1.0f, out.x);
      out.y = fmaf(s, inv, K);
      out.z = fmaxf(q - s * s * inv, 0.f);
    }
  } else {
    uint32_t ad = ax + g.slot_floats * 4;
    const float4 cf = slot_side<1, EXTRA>(sm, g, slot)[1];
    const f32x2 nmean = pair(-cf.x), scale = pair(cf.y), beta = pair(cf.z);
    const float slope = a.neg_slope;      // activation: t * (t > 0 ? 1 : slope)
    float *dres = EXTRA && a.dres_early ? a.dres : nullptr;
    Walk w(a, g, d.y, mine.tid);          // (unused in the ordinary aligned form)
    f32x2 s1a = 0, s1b = 0, s2a = 0, s2b = 0;
    // two vectors at a time; a missing one is (mean, 0), which adds nothing
    auto load = [&](bool live, Quad &x, Quad &gy, Quad &y) {
      x = quad(cf.x); gy = quad(0.f); y = gy;
      if (live) {
        x = lds_quad(ax); gy = lds_quad(ad);
        if constexpr (EXTRA) y = lds_quad(ad + g.slot_floats * 4);
      }
      ax += kVecStride; ad += kVecStride;
    };
    auto work = [&](const Quad &x, const Quad &gy, Quad y, Quad &e, Quad &z) {
      e.a = add2(x.a, nmean); e.b = add2(x.b, nmean);
      // residual epilogue: the saved output carries the mask
      if constexpr (!EXTRA) { y.a = fma2(e.a, scale, beta); y.b = fma2(e.b, scale, beta); }
      // dz = dy * (float)(y > 0)  (routines_gpu/flat_map.cu:191-192)
      z.a = mul2(gy.a, slopes(y.a, slope)); z.b = mul2(gy.b, slopes(y.b, slope));
    };
    auto sum = [&](bool live, Quad e, Quad z) {
      if constexpr (!RAGGED) {
        if constexpr (EXTRA) { if (dres && live) stg_quad(dres + w.at, z); }
      } else {
        const int i0 = live ? w.first() : len;
        if (ragged_whole(i0, len)) {
          if constexpr (EXTRA) { if (dres) stg_quad(dres + w.vector(), z); }
        } else {      // (foreign floats may be anything, an infinity or a NaN too)
          const float4 t = floats(z), u = floats(e);
          auto in = [&](int k) { return (uint32_t)(i0 + k) < (uint32_t)len; };
          if constexpr (EXTRA) {
            if (dres) {
              float *p = dres + w.vector();
              if (in(0)) p[0] = t.x;
              if (in(1)) p[1] = t.y;
              if (in(2)) p[2] = t.z;
              if (in(3)) p[3] = t.w;
            }
          }
          z.a = pair(in(0) ? t.x : 0.f, in(1) ? t.y : 0.f); z.b = pair(in(2) ? t.z : 0.f, in(3) ? t.w : 0.f);
          e.a = pair(in(0) ? u.x : 0.f, in(1) ? u.y : 0.f); e.b = pair(in(2) ? u.z : 0.f, in(3) ? u.w : 0.f);
        }
      }
      s1a = add2(s1a, z.a); s2a = fma2(z.a, e.a, s2a); s1b = add2(s1b, z.b); s2b = fma2(z.b, e.b, s2b);
      if constexpr (EXTRA || RAGGED) w.advance(g);
    };
    for (uint32_t i = 0; i < steps; i += 2, tm += 16) {
      const bool l0 = i < cnt, l1 = i + 1 < cnt;
      Quad x0, g0, y0, x1, g1, y1, e0, z0, e1, z1;
      load(l0, x0, g0, y0); load(l1, x1, g1, y1);
      work(x0, g0, y0, e0, z0); work(x1, g1, y1, e1, z1);
      if constexpr (KEEP) {
        __syncwarp();
        if (i + 1 < steps) tmem_st(tm, e0, z0, e1, z1); else tmem_st(tm, e0, z0);
      }
      sum(l0, e0, z0); sum(l1, e1, z1);
    }
    if constexpr (EXTRA) { if (dres) fence_global_to_bulk(); }
    __syncwarp();
    if (lane == 0) mbar_arrive(&ctl->empty[slot]);
    const float2 u = split(add2(s1a, s1b)), v = split(add2(s2a, s2b));
    out = make_float4(warp_sum(u.x + u.y), warp_sum(v.x + v.y), 0.f, 0.f);
  }
  if (lane == 0) res[threadIdx.x >> 5] = out;
}

template <int DIR, bool EXTRA, bool RAGGED, bool KEEP, bool ADDS>
__device__ __forceinline__ void visit_apply(const FusedArgs &a, const RingGeom &g, unsigned char *sm, RingCtl *ctl,
                                            const uint4 &d, uint32_t slot, const float4 *coef, uint32_t coef_q)
{
  const uint32_t lane = threadIdx.x & 31;
  const Mine<KEEP> mine(g, ctl, d);
  const uint32_t cnt = mine.cnt, steps = mine.steps;
  const float slope = a.neg_slope;      // activation: t * (t > 0 ? 1 : slope)
  const bool early = EXTRA && DIR == 1 && a.dres_early;      // plane 1 holds dz (see fence_global_to_bulk)
  float *dres = EXTRA && DIR == 1 && !early ? a.dres : nullptr;
  const float4 c0 = coef[0];
  const f32x2 nmean = pair(-c0.x), scale = pair(c0.y), beta = pair(c0.z), cB = pair(c0.w), cC = pair(coef[1].x);
  const int len = (int)d.z;
  uint32_t ax = smem_u32(slot_x(sm, g, slot)) + mine.tid * 16, tm = mine.tm;
  uint32_t ad = ax + g.slot_floats * 4;
  Walk w(a, g, d.y, mine.tid);
  // one vector: activation(bn(x)) or the input gradient.  x: the input (KEEP and backward: x - mean); gy: dy or dz;
  // e: residual or saved output; old: what an accumulating write adds to (aligned rows)
  auto one = [&](const Quad &x, const Quad &gy, const Quad &e, const Quad &old) {
    Quad o, z;
    const Quad u = KEEP && DIR == 1 ? x : Quad{add2(x.a, nmean), add2(x.b, nmean)};
    if constexpr (DIR == 0) {
      o.a = fma2(u.a, scale, beta); o.b = fma2(u.b, scale, beta);
      if constexpr (EXTRA) { o.a = add2(o.a, e.a); o.b = add2(o.b, e.b); }
      o.a = mul2(o.a, slopes(o.a, slope)); o.b = mul2(o.b, slopes(o.b, slope));
    } else {
      z = gy;
      if (!KEEP && !early) {
        const Quad y = EXTRA ? e : Quad{fma2(u.a, scale, beta), fma2(u.b, scale, beta)};
        z.a = mul2(gy.a, slopes(y.a, slope)); z.b = mul2(gy.b, slopes(y.b, slope));
      }
      o.a = fma2(scale, z.a, fma2(cB, u.a, cC)); o.b = fma2(scale, z.b, fma2(cB, u.b, cC));
    }
    float *p = a.out + (RAGGED ? w.vector() : w.at);
    const int i0 = RAGGED ? w.first() : 0;
    if (!RAGGED || ragged_whole(i0, len)) {
      if constexpr (ADDS) {
        const Quad was = RAGGED ? ldg_quad(p) : old;
        o.a = add2(was.a, o.a); o.b = add2(was.b, o.b);
      }
      stg_stream(p, o);
      if constexpr (EXTRA && DIR == 1) { if (dres) stg_stream(dres + (p - a.out), z); }
    } else {
      const float4 t = floats(o), s = floats(z);
      auto put = [&](int k, float f, float r) {
        if ((uint32_t)(i0 + k) < (uint32_t)len) {
          p[k] = ADDS ? p[k] + f : f;
          if constexpr (EXTRA && DIR == 1) { if (dres) dres[(p - a.out) + k] = r; }
        }
      };
      put(0, t.x, s.x); put(1, t.y, s.y); put(2, t.z, s.z); put(3, t.w, s.w);
    }
    w.advance(g);
  };
  // Accumulating writes: the next vectors' old values are on their way while one is worked on, and the producer has brought the tile to
  // L2.  (Loaded from HBM one after the other: [256,64,112,112] 768 us and, so, 545, [300,64,56,56] 222 and 164, [64,95,55,55] 88 and 72.)
  Walk far = w;
  auto olds = [&](bool live) {
    Quad q = quad(0.f);
    if constexpr (!RAGGED && ADDS) {
      if (live) q = ldg_quad(a.out + far.at);
      far.advance(g);
    }
    return q;
  };
  if constexpr (KEEP) {
    tmem_wait_st();      // what this warp stored in the reduce visits
    uint32_t i = 0;
    if constexpr (DIR == 0) {
      auto put = [&](const Quad &x, uint32_t j) {
        if (j >= cnt) return;
        Quad e = x;
        if constexpr (EXTRA) { e = lds_quad(ad); ad += kVecStride; }
        one(x, x, e, x);
      };
      if constexpr (!RAGGED) {
        // (ragged rows: [64,95,55,55] residual 60 -> 76 us with four at a time)
        for (; i + 4 <= steps; i += 4, tm += 16) {
          Quad x0, x1, x2, x3;
          tmem_ld(tm, x0, x1, x2, x3);
          put(x0, i); put(x1, i + 1); put(x2, i + 2); put(x3, i + 3);
          __syncwarp();
        }
      }
      if constexpr (!RAGGED) {
        if (i + 2 <= steps) {
          Quad x0, x1;
          tmem_ld(tm, x0, x1);
          put(x0, i); put(x1, i + 1);
          __syncwarp();
          i += 2; tm += 8;
        }
      }
      for (; i < steps; ++i, tm += 4) {
        Quad x0;
        tmem_ld(tm, x0);
        put(x0, i);
        __syncwarp();
      }
    } else {
      Quad o0 = olds(0 < cnt), o1 = olds(1 < cnt);
      if constexpr (!RAGGED) {
        for (; i + 2 <= steps; i += 2, tm += 16) {
          Quad d0, z0, d1, z1;
          tmem_ld(tm, d0, z0, d1, z1);
          const Quad n0 = olds(i + 2 < cnt), n1 = olds(i + 3 < cnt);
          one(d0, z0, d0, o0);
          if (i + 1 < cnt) one(d1, z1, d1, o1);
          o0 = n0; o1 = n1;
          __syncwarp();
        }
      }
      for (; i < steps; ++i, tm += 8) {      // (one at most, or all of a ragged visit)
        Quad d0, z0;
        tmem_ld(tm, d0, z0);
        if (i < cnt) one(d0, z0, d0, o0);
        __syncwarp();
      }
    }
  } else {
    Quad o0 = olds(0 < cnt), o1 = olds(1 < cnt);
    for (uint32_t i = 0; i < cnt; ++i, ax += kVecStride, ad += kVecStride) {
      const Quad x = lds_quad(ax);
      Quad gy = x, e = x;
      if constexpr (DIR == 1) gy = lds_quad(ad);
      if constexpr (EXTRA) { if (!early) e = lds_quad(DIR == 1 ? ad + g.slot_floats * 4 : ad); }
      const Quad n1 = olds(i + 2 < cnt);
      one(x, gy, e, o0);
      o0 = o1; o1 = n1;
    }
  }
  __syncwarp();
  if (lane == 0) { if (!KEEP || kSlotAlways<DIR, EXTRA>) mbar_arrive(&ctl->empty[slot]); mbar_arrive(&ctl->coef_empty[coef_q]); }
}

// ======================================================================================
// delivery warp: unit completion
// ======================================================================================
// (count, mean, M2) in double precision and Chan's pairwise update; used to merge a unit's
// partials in ONE pass over them, so that every partial is loaded exactly once and all loads
// of a batch are in flight together (the merge sits on the critical path of the pipeline).
struct Moments64 { double n, mean, m2; };
__device__ __forceinline__ Moments64 merge64(Moments64 a, Moments64 b)
{
  const double n = a.n + b.n;
  if (n <= 0.0) return Moments64{0.0, 0.0, 0.0};
  const double f = b.n / n, d = b.mean - a.mean;
  return Moments64{n, a.mean + d * f, a.m2 + b.m2 + d * d * a.n * f};
}
constexpr int kFinRegs = 16;     // partials a lane holds in registers (regime R: 512 tiles per unit)

// Regime R: one channel, up to thousands of partials.  The merge sits on the critical path of the
// pipeline, so all of a lane's loads are issued together (one round trip) and both passes of the
// two-pass merge (weighted mean, then M2 about it) run from registers.  Units with more than
// 32*kFinRegs tiles take further rounds and fold each round in with Chan's update.
template <int DIR>
__device__ __forceinline__ void warp_finish_unit_R(const FusedArgs &a, uint32_t u)
{
  const Plan &P = a.plan;
  const uint32_t lane = threadIdx.x & 31, T = P.tiles_per_unit;
  const float4 *part = ws_f4(a, P.off_part) + (size_t)u * T;
  Moments64 tot{0.0, 0.0, 0.0};
  double s1 = 0.0, s2 = 0.0;
  for (uint32_t k0 = 0; k0 < T; k0 += 32u * kFinRegs) {
    float rx[kFinRegs], ry[kFinRegs], rz[kFinRegs];
#pragma unroll
    for (int i = 0; i < kFinRegs; ++i) {
      const uint32_t k = k0 + lane + 32u * i;
      const float4 p = (k < T) ? __ldcg(part + k) : make_float4(0.f, 0.f, 0.f, 0.f);
      rx[i] = p.x; ry[i] = p.y; rz[i] = p.z;
    }
    if constexpr (DIR == 0) {
      double sn = 0.0, sm = 0.0;
#pragma unroll
      for (int i = 0; i < kFinRegs; ++i) { sn += (double)rx[i]; sm = fma((double)rx[i], (double)ry[i], sm); }
      sn = warp_sum_all(sn); sm = warp_sum_all(sm);
      const double mean = sn > 0.0 ? sm / sn : 0.0;
      double sq = 0.0;
#pragma unroll
      for (int i = 0; i < kFinRegs; ++i) { const double d = (double)ry[i] - mean; sq += (double)rz[i] + (double)rx[i] * d * d; }
      sq = warp_sum_all(sq);
      tot = merge64(tot, Moments64{sn, mean, sq});
    } else {
#pragma unroll
      for (int i = 0; i < kFinRegs; ++i) { s1 += (double)rx[i]; s2 += (double)ry[i]; }
    }
  }
  if constexpr (DIR == 0) {
    if (lane == 0) finish_channel_fwd(a, u, tot.n, tot.mean, tot.m2);
  } else {
    s1 = warp_sum_all(s1); s2 = warp_sum_all(s2);
    if (lane == 0) finish_channel_bwd(a, u, s1, s2);
  }
}

// ======================================================================================
// fused mode, regime R: every block merges the partials of the units it applies itself
// ======================================================================================
// Instead of counting deliveries and electing a finisher, a delivery is a single 8-byte store of a
// tagged partial -- forward (mean, M2), backward (sum dz, sum dz*(x-mean)), lowest mantissa bit of
// the second value forced to one so the word is never all zero -- and whoever needs a unit polls
// the unit's partial words until none is zero, then merges them in a fixed order in double
// precision.  All blocks compute bit-identical coefficients; no atomics, fences or extra round
// trips sit between the last delivery and the first apply.  The element count of a partial
// follows from the tile geometry.  Two buffers are used alternately, launch by launch (parity
// word in the workspace header): a delivery also zeroes its word in the other buffer.
__device__ __forceinline__ unsigned long long *tag_buf(const FusedArgs &a, uint32_t parity)
{
  return reinterpret_cast<unsigned long long *>(a.ws + a.plan.off_tag) + (size_t)parity * a.plan.total_tiles * a.plan.cb;
}
__device__ __forceinline__ unsigned long long ld_relaxed_sys_u64(const unsigned long long *p)
{
  unsigned long long v;
  asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_sys_u64(unsigned long long *p, unsigned long long v)
{
  asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Partial words per lane per round of pull_merge_unit.  Rounds are short, so that most words are merged while the last ones
// are still on their way: [2048,256,56,56] backward with 2 / 3 / 4 / 5 / 8 words 3504 / 3441 / 3493 / 3554 / 3567 us,
// [256,64,112,112] forward 284 / 275 / 273 / 270 / 313.  (One word per block and unit instead of one per tile makes the merge
// shorter still, but all blocks then poll a few lines while all blocks write them: 4026 us, and 3673 with the words 32 bytes
// apart.)
constexpr int kPullRegsFwd = 4, kPullRegsBwd = 3;

// Whole warp.  Returns false when the wait ran out (abort raised).  On success c0 / c1 hold the
// unit's coefficients in every lane; `owner` makes lane 0 write the per-channel outputs.
// The merge runs in every block for every unit, on the way from the last delivery to the first apply: sums about one shift
// in a single pass, no double precision division (inv_local and inv_total: reciprocals of this GPU's and of all GPUs' elements
// per channel).  With two passes and three divisions a merge took 2800 cycles after its last word had come, in the forward
// pass a third of the kernel's time.
template <int DIR>
__device__ __forceinline__ bool pull_merge_unit(const FusedArgs &a, RingCtl *ctl, uint32_t *status,
                                                uint32_t u, bool owner, const float4 &in, double inv_local, double inv_total, float4 &c0, float4 &c1)
{
  constexpr int kPullRegs = DIR == 0 ? kPullRegsFwd : kPullRegsBwd;
  const Plan &P = a.plan;
  const uint32_t lane = threadIdx.x & 31, T = P.tiles_per_unit;
  const unsigned long long *buf = tag_buf(a, ctl->parity) + (size_t)u * T;
  const float gm = in.x, bt = in.y;      // gamma, beta; backward: mean, 1 / std
  Moments64 tot{0.0, 0.0, 0.0};
  double s1 = 0.0, s2 = 0.0, K = 0.0;      // forward: sums about K, the mean of the first partial
  const long long t0 = clock64();
  // With several GPUs only the unit's owner block needs the local merge (it ships the result to
  // every rank); all other blocks go straight to the exchanged records.
  const bool local = (a.world <= 1) || owner;
  for (uint32_t k0 = 0; local && k0 < T; k0 += 32u * kPullRegs) {
    unsigned long long r[kPullRegs];
    uint32_t nk[kPullRegs];
    if constexpr (DIR == 0) {
#pragma unroll
      for (int i = 0; i < kPullRegs; ++i) {
        const uint32_t k = k0 + lane + 32u * i;
        uint32_t sb = k, piece = 0;
        if (P.pieces != 1) { sb = k / P.pieces; piece = k - sb * P.pieces; }
        const uint32_t n0 = sb * P.rows_per_tile, col0 = piece * P.piece_len;
        const uint32_t rows = (P.N - n0 < P.rows_per_tile) ? (P.N - n0) : P.rows_per_tile;
        const uint32_t len = (P.dim0 - col0 < P.piece_len) ? (P.dim0 - col0) : P.piece_len;
        nk[i] = k < T ? rows * len : 0u;
      }
    }
    for (;;) {
      bool all = true;
#pragma unroll
      for (int i = 0; i < kPullRegs; ++i) {
        const uint32_t k = k0 + lane + 32u * i;
        r[i] = (k < T) ? ld_relaxed_gpu_u64(buf + k) : 1ull;
        all = all && (r[i] != 0ull);
      }
      if (__all_sync(0xffffffffu, all)) break;
      __nanosleep(100);
      uint32_t stop = 0;
      if (lane == 0) {
        if (ctl->abort) stop = 1;
        else if (clock64() - t0 > 2 * a.wait_cycles) { atomicOr(status, ANODE_ST_WAIT_STATS); ctl->abort = 1; stop = 1; }
      }
      if (__shfl_sync(0xffffffffu, stop, 0)) return false;
    }
    if constexpr (DIR == 0) {
      if (k0 == 0) K = (double)__shfl_sync(0xffffffffu, __uint_as_float((uint32_t)r[0]), 0);
#pragma unroll
      for (int i = 0; i < kPullRegs; ++i) {
        if (nk[i]) {
          const double n = (double)nk[i], d = (double)__uint_as_float((uint32_t)r[i]) - K;
          s1 = fma(n, d, s1); s2 += fma(n * d, d, (double)__uint_as_float((uint32_t)(r[i] >> 32)));
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < kPullRegs; ++i) {
        const uint32_t k = k0 + lane + 32u * i;
        if (k < T) {
          s1 += (double)__uint_as_float((uint32_t)(r[i] & 0xffffffffull));
          s2 += (double)__uint_as_float((uint32_t)(r[i] >> 32));
        }
      }
    }
  }
  if (local) {
    s1 = warp_sum_all(s1); s2 = warp_sum_all(s2);
    if constexpr (DIR == 0) {
      const double m = s1 * inv_local;
      tot = Moments64{(double)a.plan.dim0 * (double)a.plan.N, K + m, not_below_zero(s2 - s1 * m)};
    }
  }
  if (a.world > 1) {
    // ---- exchange between GPUs.  A record is three 8-byte words (value in the low half, the
    // call's epoch in the high half): every word validates itself, so plain peer stores suffice
    // and nothing is ever zeroed; consecutive calls alternate between two buffers.
    const uint32_t par = a.epoch & 1u;
    const size_t slot = (((size_t)par * a.world) * a.xchg_channels + u) * 4;      // + src * xchg_channels * 4
    const size_t src_stride = (size_t)a.xchg_channels * 4;
    if (owner && lane < a.world) {
      // word 0 of a forward record is the element count as an exact integer (a float would round counts above 2^24)
      const uint32_t w0 = DIR == 0 ? (uint32_t)tot.n : __float_as_uint((float)s1);
      const uint32_t w1 = __float_as_uint(DIR == 0 ? (float)tot.mean : (float)s2);
      const uint32_t w2 = __float_as_uint(DIR == 0 ? (float)tot.m2 : 0.f);
      unsigned long long *dst = a.xchg[lane] + slot + a.rank * src_stride;       // this rank's slot in peer `lane`
      const unsigned long long e = (unsigned long long)a.epoch << 32;
      st_relaxed_sys_u64(dst + 0, e | w0);
      st_relaxed_sys_u64(dst + 1, e | w1);
      st_relaxed_sys_u64(dst + 2, e | w2);
    }
    // lane r collects rank r's record from this GPU's own buffer
    const unsigned long long *mine = a.xchg[a.rank] + slot + (lane < a.world ? lane : 0) * src_stride;
    unsigned long long v0 = 0, v1 = 0, v2 = 0;
    for (;;) {
      bool ok = true;
      if (lane < a.world) {
        v0 = ld_relaxed_sys_u64(mine + 0); v1 = ld_relaxed_sys_u64(mine + 1); v2 = ld_relaxed_sys_u64(mine + 2);
        ok = (uint32_t)(v0 >> 32) == a.epoch && (uint32_t)(v1 >> 32) == a.epoch && (uint32_t)(v2 >> 32) == a.epoch;
      }
      if (__all_sync(0xffffffffu, ok)) break;
      __nanosleep(200);
      uint32_t stop = 0;
      if (lane == 0) {
        if (ctl->abort) stop = 1;
        else if (clock64() - t0 > a.wait_cycles) { atomicOr(status, ANODE_ST_WAIT_PEER); ctl->abort = 1; stop = 1; }
      }
      if (__shfl_sync(0xffffffffu, stop, 0)) return false;
    }
    // merge in rank order (lane = rank; the shuffle tree is the same on every GPU, so all ranks
    // obtain bit-identical statistics)
    const bool live = lane < a.world;
    const double f0 = live ? (DIR == 0 ? (double)(uint32_t)v0 : (double)__uint_as_float((uint32_t)v0)) : 0.0;
    const double f1 = live ? (double)__uint_as_float((uint32_t)v1) : 0.0;
    const double f2 = live ? (double)__uint_as_float((uint32_t)v2) : 0.0;
    if constexpr (DIR == 0) {
      const double sn = warp_sum_all(f0), sm = warp_sum_all(f0 * f1);
      const double mean = sm / sn;
      const double d = f1 - mean;
      const double sq = warp_sum_all(live ? f2 + f0 * d * d : 0.0);
      tot = Moments64{sn, mean, sq};
    } else {
      s1 = warp_sum_all(f0); s2 = warp_sum_all(f1);
    }
  }
  if constexpr (DIR == 0) {
    const float mf = (float)tot.mean;
    const float vf = (float)(tot.m2 * inv_total + (double)a.epsilon);     // biased, epsilon folded in (batch_norm.cu:160)
    c0 = make_float4(mf, gm * inv_std(vf), bt, 0.f);
    c1 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (owner && lane == 0) {
      a.mean[u] = mf; a.var[u] = vf;
      if (a.run_mean) { const float o = a.run_mean[u]; a.run_mean[u] = o + a.avg_rate * (mf - o); }
      if (a.run_var) { const float o = a.run_var[u]; a.run_var[u] = o + a.avg_rate * (vf - o); }
    }
  } else {
    const float r = in.w;
    const double rs2 = (double)r * s2;                       // sum(dz * xhat)
    const double A = (double)gm * (double)r;
    c0 = make_float4(in.z, gm * r, bt, 0.f);
    c1 = make_float4((float)(-A * (double)r * rs2 * inv_total), (float)(-A * s1 * inv_total), 0.f, 0.f);
    if (owner && lane == 0) {
      if (a.dbeta) a.dbeta[u] = (float)s1;
      if (a.dgamma) a.dgamma[u] = (float)rs2;
    }
  }
  return true;
}

// ======================================================================================
// the kernel
// ======================================================================================
// Whole-row tiles only (one channel per unit): short-row shapes are served by the cluster kernel
// (bn_segres.cu) and the plain kernel.
// EXTRA: residual epilogue; RAGGED: rows that are not a multiple of four floats; TMEM: some tiles may stay in tensor memory
// (ring_keeps); ADDS: the output is added to.
template <int DIR, bool EXTRA, bool RAGGED, bool TMEM = true, bool ADDS = false>
__global__ void __launch_bounds__(kRingThreads, 1) bn_ring_kernel(const FusedArgs a, const RingGeom g)
{
  extern __shared__ __align__(128) unsigned char sm[];
  RingCtl *ctl = reinterpret_cast<RingCtl *>(sm);
  const Plan &P = a.plan;
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t *status = a.status;
  uint32_t *done = ws_u32(a, P.off_done);

  if (tid == kConsumers) {      // (warp 0 allocates meanwhile)
    for (uint32_t i = 0; i < g.slots; ++i) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], kCWarps); }
    for (uint32_t i = 0; i < kResQ; ++i) { mbar_init(&ctl->res_full[i], kCWarps); mbar_init(&ctl->res_empty[i], 1); }
    for (uint32_t i = 0; i < kCoefQ; ++i) { mbar_init(&ctl->coef_full[i], 1); mbar_init(&ctl->coef_empty[i], kCWarps); }
    ctl->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (TMEM && g.keep_slots && warp == 0) { __syncwarp(); tmem_alloc(&ctl->tmem); tmem_fence_before(); }
  __syncthreads();
  if (TMEM && g.keep_slots) tmem_fence_after();

  Sched sc; sc.init(a);
  // the two warps that use the tagged words each see to it that ctl->parity is there for them (in shared memory: a register more and
  // the backward pass was slower, 390 -> 426 us on [256,64,112,112])
  auto buffer = [&] {
    if (a.mode != MODE_FUSED) return;
    const uint32_t p = buffer_of_launch(ws_u32(a, g.hdr), ws_u32(a, g.hdr + 4), 2);
    if (lane == 0) ctl->parity = p;
    __syncwarp();
  };

  if (warp < kConsumers / 32) {
    // ------------------------------------------------------------------ consumers
    uint32_t slot = g.slots - 1, par = 1;     // ring position, stepped without divisions
    uint32_t qres = 0, rpar = 1, qcoef = 0, cpar = 0;      // mailbox positions
    for (uint32_t s = 0; s < sc.steps; ++s) {
      if (sc.reduce_at(s)) {
        if (++slot == g.slots) { slot = 0; par ^= 1u; }
        // the partial mailbox entry must have been emptied by the delivery warp (first pass: free)
        bool ok = warp_wait(&ctl->res_empty[qres], rpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles);
        ok = ok && warp_wait(&ctl->full[slot], par, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles);
        if (!ok) break;                                 // warps are independent: no barrier to honour
        const uint4 d = *reinterpret_cast<const uint4 *>(slot_side<DIR, EXTRA>(sm, g, slot));
        float4 *res = res_box(sm, g, qres);
        if (TMEM && d.x >> 16) visit_reduce<DIR, EXTRA, RAGGED, true>(a, g, sm, ctl, d, slot, res);
        else visit_reduce<DIR, EXTRA, RAGGED, false>(a, g, sm, ctl, d, slot, res);
        if (lane == 0) mbar_arrive(&ctl->res_full[qres]);
        if (++qres == kResQ) { qres = 0; rpar ^= 1u; }
      }
      if (sc.apply_at(s)) {
        if (!warp_wait(&ctl->coef_full[qcoef], cpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
        const float4 *coef = coef_box(sm, g, qcoef);
        const uint4 d = *reinterpret_cast<const uint4 *>(coef + 2);
        const bool kept = TMEM && (d.x >> 16) != 0;
        if (!kept || kSlotAlways<DIR, EXTRA>) {
          if (++slot == g.slots) { slot = 0; par ^= 1u; }
          if (!warp_wait(&ctl->full[slot], par, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
        }
        if (TMEM && kept) visit_apply<DIR, EXTRA, RAGGED, true, ADDS>(a, g, sm, ctl, d, slot, coef, qcoef);
        else visit_apply<DIR, EXTRA, RAGGED, false, ADDS>(a, g, sm, ctl, d, slot, coef, qcoef);
        if (++qcoef == kCoefQ) { qcoef = 0; cpar ^= 1u; }
      }
    }
  } else if (warp == kConsumers / 32) {
    // ------------------------------------------------------------------ producer
    // where the window between the two visits exceeds what L2 keeps, only the fraction that fits is marked "keep"
    const uint64_t keep = g.keep_frac < 1.0f ? policy_keep_fraction(g.keep_frac) : policy_keep(), drop = policy_drop();
    const uint32_t rs = P.C * P.dim0;                  // float offsets are below 2^32 (check_dims)
    const uint32_t row0 = lane / g.copies, off0 = (lane - row0 * g.copies) * kRingCopyBytes;      // the lane's copy of a tile
    uint32_t k = 0;
    uint32_t slot = g.slots - 1, par = 1;
    bool ok = true;
    // lane l: the visits of tiles n + l, n a multiple of 32; and, backward, (mean, gamma / std, beta) of the tile's channel
    uint4 red = make_uint4(0, 0, 0, 0), app = red;
    float4 side = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t v = 0; ok && v < 2 * sc.steps; ++v) {
      const uint32_t s = v >> 1, kind = v & 1u;
      if (kind == 0 ? !sc.reduce_at(s) : !sc.apply_at(s)) continue;
      if (kind == 1 && !kSlotAlways<DIR, EXTRA> && g.keep_slots == g.keep_period && !ADDS) continue;      // all from tensor memory
      const uint32_t n = kind == 0 ? s : s - sc.look;
      float4 raw = make_float4(0.f, 1.f, 1.f, 0.f);
      const bool fresh = (n & 31u) == 0u;
      if (fresh) {
        uint4 d = make_uint4(0, 0, 0, 0);
        if (n + lane < sc.my_tiles) {
          const TileRange tr = tile_range(P, sc.b + (n + lane) * sc.G);
          d = describe(tr, RAGGED, keep_at(g, n + lane));
          if (DIR == 1 && kind == 0) {
            raw.x = a.mean_in[tr.c0]; raw.y = a.var_in[tr.c0];
            if (a.gamma) raw.z = a.gamma[tr.c0];
            if (a.gamma && a.beta) raw.w = a.beta[tr.c0];
          }
        }
        if (kind == 0) red = d; else app = d;
      }
      const uint4 d = shfl4(kind == 0 ? red : app, n & 31u);
      const bool kept = (d.x >> 16) != 0;
      if (ADDS && kind == 1) {
        // what the apply visit adds to is brought to L2 some steps ahead of the consumers (of a ragged row what lies between two 16-byte boundaries)
        const uint32_t whole = rs * P.N & ~3u;
        for (uint32_t r = row0; r < d.w; r += 32) {
          const uint32_t first = d.y + r * rs, from = RAGGED ? (first + 3) & ~3u : first, to = RAGGED ? (first + d.z) & ~3u : first + d.z;
          const uint32_t at = from + off0 / 4;
          if (at < to && to <= whole) bulk_prefetch(a.out + at, (to - at < kRingCopyBytes / 4 ? to - at : kRingCopyBytes / 4) * 4);
        }
      }
      if (kind == 1 && kept && !kSlotAlways<DIR, EXTRA>) continue;
      ++k;
      if (++slot == g.slots) { slot = 0; par ^= 1u; }
      // (one lane polls here: a producer that reacts sooner was measured slower where the window between the two
      // visits exceeds what L2 keeps, and hardly faster elsewhere)
      uint32_t okw = 1;
      if (lane == 0) okw = mbar_wait(&ctl->empty[slot], par ^ 1u, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles) ? 1u : 0u;
      if constexpr (DIR == 1 && EXTRA) {
        // the dz this visit reads back was stored by visit kr (counting those that use a slot), which must have been
        // given back: implied by the wait above unless fewer than `slots` visits lie in between
        if (kind == 1 && lane == 0 && okw && a.dres_early) {
          const uint32_t before = n > sc.look ? n - sc.look : 0u;
          const uint32_t kr = n + before - kept_before(g, before);
          if (k - 1 - kr < g.slots)
            okw = mbar_wait(&ctl->empty[kr % g.slots], (kr / g.slots) & 1u, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles) ? 1u : 0u;
        }
      }
      ok = __shfl_sync(0xffffffffu, okw, 0) != 0;     // one lane decides for the warp
      if (!ok) { --k; break; }
      float *xs = slot_x(sm, g, slot);
      const uint32_t base = d.y, len = d.z, rows = d.w;
      const uint64_t pol = (kind == 0 && a.mode == MODE_FUSED && !kept) ? keep : drop;
      // the visit's tensors: x; dy, or the dz that the reduce visit stored; residual or saved output where it is needed
      const float *p1 = nullptr, *p2 = nullptr;
      uint64_t pol1 = pol;
      if constexpr (DIR == 1) {
        p1 = a.dy;
        if constexpr (EXTRA) {
          if (!a.dres_early) p2 = a.ymask;
          else if (kind == 0) { p2 = a.ymask; pol1 = drop; }      // dy and the saved output are not read again
          else p1 = a.dres;
        }
      } else if constexpr (EXTRA) {
        if (kind == 1) p1 = a.res;
      }
      const bool p0 = !kSlotAlways<DIR, EXTRA> || kind == 0 || !kept;
      const uint32_t planes = (p0 ? 1u : 0u) + (p1 ? 1u : 0u) + (p2 ? 1u : 0u);
      auto fetch = [&](float *dst, uint32_t src, uint32_t bytes) {
        if (p0) bulk_g2s(dst, a.x + src, bytes, &ctl->full[slot], pol);
        if (p1) bulk_g2s(dst + g.slot_floats, p1 + src, bytes, &ctl->full[slot], pol1);
        if (p2) bulk_g2s(dst + 2 * g.slot_floats, p2 + src, bytes, &ctl->full[slot], pol1);
      };
      // the copies go out first; the visit's description and the arrival that completes the barrier's count follow
      if constexpr (!RAGGED) {
        // a long row is fetched as several bulk copies (one per lane), so that many are in flight
        const uint32_t row_bytes = len * 4u;
        if (lane == 0) mbar_expect_tx(&ctl->full[slot], row_bytes * rows * planes);
        __syncwarp();
        if (off0 < row_bytes) {
          const uint32_t nb = row_bytes - off0 < kRingCopyBytes ? row_bytes - off0 : kRingCopyBytes;
          for (uint32_t r = row0; r < rows; r += 32) fetch(xs + r * len + off0 / 4, base + r * rs + off0 / 4, nb);
        }
      } else {
        // from the boundary below each row's start to the one above its end, but never past the tensor's own end:
        // the last floats of a tensor whose size is no multiple of four are stored by three lanes instead
        const uint32_t per_row = ragged_pitch(len), total = rs * P.N, whole = total & ~3u;
        auto span = [&](uint32_t r, uint32_t &start) {      // bytes of row r, and the float it is fetched from
          const uint32_t first = base + r * rs;
          start = first & ~3u;
          return ((first + len >= whole ? whole : (first + len + 3) & ~3u) - start) * 4u;
        };
        uint32_t bytes = 0;
        for (uint32_t r = lane; r < rows; r += 32) { uint32_t start; bytes += span(r, start); }
        bytes = __reduce_add_sync(0xffffffffu, bytes) * planes;
        const uint32_t last = base + (rows - 1) * rs, tail = total & 3u;
        if (last + len > whole && lane < tail) {
          const uint32_t src = whole + lane;
          float *dst = xs + 4 * per_row * (rows - 1) + (src - (last & ~3u));
          if (p0) *dst = __ldcg(a.x + src);
          if (p1) dst[g.slot_floats] = __ldcg(p1 + src);
          if (p2) dst[2 * g.slot_floats] = __ldcg(p2 + src);
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // (before a later copy into this slot)
        }
        if (lane == 0) mbar_expect_tx(&ctl->full[slot], bytes);
        __syncwarp();
        for (uint32_t r = lane; r < rows; r += 32) {
          uint32_t start;
          const uint32_t nb = span(r, start);
          if (nb) fetch(xs + 4 * per_row * r, start, nb);
        }
      }
      if (kind == 0) {
        float4 *box = slot_side<DIR, EXTRA>(sm, g, slot);
        if constexpr (DIR == 1) {
          // coefficients of the visit's ReLU mask
          if (fresh) side = make_float4(raw.x, raw.z * inv_std(raw.y), raw.w, 0.f);
          if (lane == (n & 31u)) box[1] = side;
        }
        if (lane == (n & 31u)) *reinterpret_cast<uint4 *>(box) = d;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->full[slot]);
    }
    // wait (bounded) for every copy that was issued: after an abort, of this warp or, now or later, of another, nobody else may
    if (lane == 0) {
      const uint32_t first = k > g.slots ? k - g.slots : 0;
      for (uint32_t kk = first; kk < k; ++kk) {
        const long long t0 = clock64();
        while (!mbar_try(&ctl->full[kk % g.slots], (kk / g.slots) & 1u) && clock64() - t0 < kDrainCycles) {}
      }
    }
  } else if (warp == kConsumers / 32 + 1) {
    // ------------------------------------------------------------------ delivery warp
    // Reduce visit j of this block is tile b + j*G.  The consumer warps' partials of a tile are merged in a fixed order.
    uint32_t q = 0, qpar = 0, tile = sc.b;
    buffer();
    for (uint32_t j = 0; j < sc.reduces; ++j) {
      if (!warp_wait(&ctl->res_full[q], qpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
      float4 v = lane < kCWarps ? res_box(sm, g, q)[lane] : make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (DIR == 0) {
        Moments m{v.x, v.y, v.z};
#pragma unroll
        for (int o = (int)kCWarps / 2; o > 0; o >>= 1) {
          Moments c;
          c.n = __shfl_down_sync(0xffffffffu, m.n, o, kCWarps);
          c.mean = __shfl_down_sync(0xffffffffu, m.mean, o, kCWarps);
          c.m2 = __shfl_down_sync(0xffffffffu, m.m2, o, kCWarps);
          m = merge(m, c);
        }
        v = make_float4(m.n, m.mean, m.m2, 0.f);
      } else {
#pragma unroll
        for (int o = (int)kCWarps / 2; o > 0; o >>= 1) {
          v.x += __shfl_down_sync(0xffffffffu, v.x, o, kCWarps);
          v.y += __shfl_down_sync(0xffffffffu, v.y, o, kCWarps);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->res_empty[q]);
      if (++q == kResQ) { q = 0; qpar ^= 1u; }
      if (a.mode == MODE_FUSED) {
        // one tagged 8-byte word per tile; nothing else to do for a delivery
        if (lane == 0) {
          const float lo = DIR == 0 ? v.y : v.x, hi = DIR == 0 ? v.z : v.y;
          st_relaxed_gpu_u64(tag_buf(a, ctl->parity) + tile, pack_rec(lo, __uint_as_float(__float_as_uint(hi) | 1u)));
          tag_buf(a, ctl->parity ^ 1u)[tile] = 0ull;
        }
        tile += sc.G;
        continue;
      }
      const uint32_t unit = tile / P.tiles_per_unit;
      uint32_t last = 0;
      if (lane == 0) {
        __stcg(ws_f4(a, P.off_part) + tile, v);
        // release: the partial stored above is visible before the count; acquire: whoever sees the
        // full count also sees every partial counted before
        uint32_t old;
        asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(done + unit) : "memory");
        last = (old + 1 == P.tiles_per_unit) ? 1u : 0u;
      }
      if (__shfl_sync(0xffffffffu, last, 0)) {
        warp_finish_unit_R<DIR>(a, unit);
        if (lane == 0) done[unit] = 0;
      }
      tile += sc.G;
    }
  } else {
    // ------------------------------------------------------------------ coefficient warp
    // Apply visit j of this block is tile b + j*G (one channel per unit).
    const double inv_local = 1.0 / ((double)P.dim0 * (double)P.N), inv_total = 1.0 / a.count_total;
    uint32_t q = 0, qpar = 1;
    // fused mode: each unit's partials are merged here (see pull_merge_unit), and consecutive visits of the same unit reuse
    // the result.  Apply pass of the three-launch form: the coefficients were prepared by the exchange / merge kernel.
    uint32_t have = 0xffffffffu;
    float4 c0 = make_float4(0.f, 0.f, 0.f, 0.f), c1 = c0;
    // lane l: the visits of tiles n + l, n a multiple of 32, their channels and these channels' parameters
    uint4 visit = make_uint4(0, 0, 0, 0);
    uint32_t unit = 0;
    float4 in = c0;
    buffer();
    for (uint32_t n = 0; n < sc.applies; ++n) {
      const uint32_t at = n & 31u;
      if (at == 0 && n + lane < sc.my_tiles) {
        const TileRange tr = tile_range(P, sc.b + (n + lane) * sc.G);
        visit = describe(tr, RAGGED, keep_at(g, n + lane)); unit = tr.unit;
        if (a.mode == MODE_FUSED) {
          in.x = a.gamma ? a.gamma[unit] : 1.0f;
          in.y = (a.gamma && a.beta) ? a.beta[unit] : 0.0f;
          if constexpr (DIR == 1) { in.z = a.mean_in[unit]; in.w = inv_std(a.var_in[unit]); }
        }
      }
      if (!warp_wait(&ctl->coef_empty[q], qpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
      const uint32_t u = __shfl_sync(0xffffffffu, unit, at);
      if (u != have) {
        if (a.mode == MODE_FUSED) {
          const float4 v = make_float4(__shfl_sync(0xffffffffu, in.x, at), __shfl_sync(0xffffffffu, in.y, at),
                                       __shfl_sync(0xffffffffu, in.z, at), __shfl_sync(0xffffffffu, in.w, at));
          // the block that owns the unit's first tile also writes the per-channel outputs
          if (!pull_merge_unit<DIR>(a, ctl, status, u, sc.b + n * sc.G == u * P.tiles_per_unit, v, inv_local, inv_total, c0, c1)) break;
        } else {
          const float4 *coef = ws_f4(a, P.off_coef) + 2 * (size_t)u;
          c0 = __ldcg(coef); c1 = __ldcg(coef + 1);
        }
        have = u;
      }
      float4 *box = coef_box(sm, g, q);
      if (lane == at) *reinterpret_cast<uint4 *>(box + 2) = visit;
      if (lane == 0) { box[0] = make_float4(c0.x, c0.y, c0.z, c1.x); box[1] = make_float4(c1.y, 0.f, 0.f, 0.f); }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->coef_full[q]);
      if (++q == kCoefQ) { q = 0; qpar ^= 1u; }
    }
  }

  // ---- leave
  if (TMEM && g.keep_slots) {
    if (warp < kCWarps) { __syncwarp(); tmem_wait_st(); }
    tmem_fence_before();
  }
  __syncthreads();
  if (TMEM && g.keep_slots && warp == 0) { tmem_fence_after(); tmem_free(ctl->tmem); }
  if (ctl->abort && tid == 0) atomicOr(status, ANODE_ST_ABORTED);
}

}  // namespace ANODE_RING_NS
}  // namespace anode_b200
