// Fused batch-norm (+activation, +residual) for large layers of short rows, e.g. [1024, 2048, 7, 7]: what the streaming kernel
// (bn_stream.cu) hands over, because it reads every tensor twice and leaves SMs idle between its clusters' steps.
//
// One persistent block per SM walks tiles of bands (bn_band.cuh) in unit-major order, as the tiled kernel (bn_ring.cuh) does with
// tiles of rows: at step s it reduces its tile number s and applies number s - look.  Every tile stays on chip in between, in
// tensor memory (256 KB per SM: look + 1 tiles of 62 KB), so each tensor crosses HBM once.
//   producer warp     streams tiles into a ring of slots: one tensor copy (cp.async.bulk.tensor) per box, hundreds of runs of a
//                     few hundred bytes in one instruction, where a bulk copy per run would be the producer's bound
//   consumer warps    (8) a thread keeps its column's vectors of a tile, at most 16 per tensor, sums them up (two floats per
//                     instruction) and leaves them in tensor memory (forward: x; backward: x - mean and dz); later reads them
//                     back, applies the coefficients and stores
//   delivery warp     folds the threads' sums of a tile to channels and stores one pair of doubles per channel and tile, forward
//                     (sum x, sum x^2), backward (sum dz, sum dz*(x-mean)), as two words that are never zero; no counter, fence or atomic
//   coefficient warp  polls the words of the unit that is applied next until none is zero and merges them in a fixed order
//                     (bit-identical in every block); the block of a unit's first tile writes its results
// Precision: at most 16 samples of a column are added up in f32, about a shift; everything beyond that is in double precision, as in the
// streaming kernel, whose f32 sums are longer.  Relative error against float64 (2-norm over the channels, geometric mean over nine shapes and three
// distributions), streaming kernel and this one: mean 4.6e-8 and 3.9e-8, variance 2.89e-8 and 2.86e-8, dgamma 2.2e-7 and 2.0e-7, dbeta
// 1.6e-7 and 1.2e-7.  (With f32 words and f32 sums of four columns: 5.8e-8, 3.13e-8, 2.2e-7, 1.7e-7.)
// Two buffers of words alternate launch by launch: a delivery zeroes its word of the other one.  Every wait is bounded; one that
// runs out sets a status bit and the block drains and leaves.  The launch is cooperative and takes the SM's whole shared memory,
// so that no other block holds columns of tensor memory or waits for them.
//
// What bounds it: HBM, and some 10 us in which the schedule fills and drains.  Streaming kernel and this one, us from launch to launch of the
// same call over buffers beyond L2, forward / backward: [1024,2048,7,7] 179 / 298 and 151 / 204 (0.83 / 0.92 of the copy bandwidth), residual
// epilogue 246 / 427 and 216 / 347 (0.87 / 0.90); [256,1024,14,14] 102 / 148 and 82 / 106, residual 137 / 211 and 110 / 167.  On the way there, in an
// older form: sixteen consumer warps (96 registers) 150 / 218 in the place of 143 / 203; all vectors of the threads' sums added up one by one 156 / 238.
#include <cuda.h>      // types only: the one function is looked up at run time

#include "bn_band.cuh"
#include "bn_host.h"
#include "bn_pipe.cuh"

namespace anode_b200 {

struct BandCtl {
  unsigned long long full[kBandMaxSlots], empty[kBandMaxSlots];
  unsigned long long res_full[kBandQ], res_empty[kBandQ], coef_full[kBandQ], coef_empty[kBandQ];
  volatile uint32_t abort;
  uint32_t parity, tmem;
};
static_assert(sizeof(BandCtl) <= kBandCtlBytes, "BandCtl outgrew the room reserved for it");

// x; dy; the residual (forward) or the saved output (backward): two-dimensional, [samples][C * dim0] floats
struct BandMaps { CUtensorMap x, dy, e; };

__device__ __forceinline__ void tensor_g2s(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, unsigned long long *bar, uint64_t policy)
{
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy) : "memory");
}

// The tiles b, b + G, ... of a block, one after another: unit and number within the unit.
struct BandWalk {
  uint32_t unit, k, dq, dr, tiles;
  __device__ __forceinline__ BandWalk(const BandGeom &g, uint32_t first, uint32_t G) : tiles(g.tiles)
  {
    unit = first / tiles; k = first - unit * tiles;
    dq = G / tiles; dr = G - dq * tiles;
  }
  __device__ __forceinline__ void next()
  {
    unit += dq; k += dr;
    if (k >= tiles) { k -= tiles; ++unit; }
  }
};

// What the consumer threads leave of a tile: [thread] its sums for its first channel, [group][channel] those of the vector that begins in
// the channel before.
struct BandSums {
  double2 *first, *second;
  __device__ __forceinline__ BandSums(unsigned char *sm, const BandGeom &g, uint32_t q)
  {
    unsigned char *at = sm + g.off_res + q * g.res_bytes;
    first = reinterpret_cast<double2 *>(at); second = reinterpret_cast<double2 *>(at + g.off_second);
  }
};

// A channel's pair of doubles for a tile: two 8-byte words that are never all zero bits ("not delivered"): a zero has its sign set.
struct BandWord { unsigned long long lo, hi; };
static_assert(sizeof(BandWord) == kBandWordBytes, "the geometry's room for a word");
__device__ __forceinline__ unsigned long long band_bits(double v)
{
  const long long b = __double_as_longlong(v);
  return b ? (unsigned long long)b : 1ull << 63;
}
__device__ __forceinline__ void st_word(BandWord *p, double lo, double hi)
{
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(band_bits(lo)), "l"(band_bits(hi)) : "memory");
}
__device__ __forceinline__ BandWord ld_word(const BandWord *p)
{
  BandWord w;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.lo), "=l"(w.hi) : "l"(p) : "memory");
  return w;
}

// ADDS: the output is added to
template <int DIR, bool EXTRA, bool ADDS>
__global__ void __launch_bounds__(kBandThreads, 1) bn_band_kernel(const FusedArgs a, const BandGeom g, const __grid_constant__ BandMaps maps)
{
  extern __shared__ __align__(128) unsigned char sm[];
  BandCtl *ctl = reinterpret_cast<BandCtl *>(sm);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t *status = a.status;
  constexpr uint32_t kKept = DIR == 0 ? 1u : 2u;                    // tensors kept in tensor memory
  constexpr uint32_t kPlanes = DIR == 0 ? 1u : EXTRA ? 3u : 2u;     // tensors of a reduce visit
  constexpr bool kSlotToo = DIR == 0 && EXTRA;                      // apply visits fetch the residual

  // Backward passes ask for the launch's buffer here and turn the word when they leave, as the tiled kernel did: asked for by the warps that
  // use it (buffer_of_launch) forward passes are 1.5 us faster, [1024,2048,7,7] 150.9 and 149.4, backward ones no faster by themselves and
  // slower behind a forward pass, [4096,512,7,7] both 391 and 396 - 399 (and with the atomic elsewhere in the launch 400 - 408).
  constexpr bool kAsk = DIR == 0;
  uint32_t *counter = reinterpret_cast<uint32_t *>(a.ws + g.hdr);
  if (tid == (kAsk ? kBandWarps * 32 : 0)) {      // (warp 0 allocates meanwhile)
    for (uint32_t i = 0; i < g.slots; ++i) { mbar_init(&ctl->full[i], 1); mbar_init(&ctl->empty[i], kBandWarps); }
    for (uint32_t i = 0; i < kBandQ; ++i) {
      mbar_init(&ctl->res_full[i], kBandWarps); mbar_init(&ctl->res_empty[i], 1);
      mbar_init(&ctl->coef_full[i], 1); mbar_init(&ctl->coef_empty[i], kBandWarps);
    }
    ctl->abort = 0;
    if (!kAsk) ctl->parity = counter[1] & 1u;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 0) { __syncwarp(); tmem_alloc(&ctl->tmem); tmem_fence_before(); }
  __syncthreads();
  tmem_fence_after();

  const uint32_t dim0 = a.plan.dim0, C = a.plan.C, N = a.plan.N, rs = C * dim0;
  const uint32_t b = blockIdx.x, G = gridDim.x;
  const uint32_t mine = b < g.total ? (g.total - b + G - 1) / G : 0, steps = mine ? mine + g.look : 0;

  // for the two warps that use the tagged words
  auto buffer = [&] {
    if constexpr (kAsk) {
      const uint32_t p = buffer_of_launch(counter, counter + 1, 2);
      if (lane == 0) ctl->parity = p;
      __syncwarp();
    }
  };

  if (warp < kBandWarps) {
    // ------------------------------------------------------------------ consumers
    const uint32_t grp0 = tid / g.L4;
    const bool live = grp0 < g.groups;
    const uint32_t grp = live ? grp0 : 0, v = live ? tid - grp0 * g.L4 : 0;
    const uint32_t chA = 4 * v / dim0, eB = (chA + 1) * dim0 - 4 * v, chB = eB < 4 ? chA + 1 : chA;
    const uint32_t pitch = g.box4 * 16, box = v / g.box4;
    const uint32_t off_s = box * g.box_bytes + grp * pitch + (v - box * g.box4) * 16, step_s = g.groups * pitch;
    const uint32_t off_g = grp * rs + 4 * v, step_g = g.groups * rs;
    const float slope = a.neg_slope;
    const uint32_t tm0 = ctl->tmem + ((warp & 3u) << 21) + (warp >> 2) * (kTmemCols * 4 / kBandWarps), tm_step = g.vpt * 4 * kKept;
    // a value per channel, for the thread's four floats
    const bool b1 = eB > 1, b2 = eB > 2, b3 = eB > 3;
    auto spread = [&](float A, float B) { return Quad{pair(A, b1 ? A : B), pair(b2 ? A : B, b3 ? A : B)}; };
    // the thread's sums for its two channels: its columns' own sums are in f32, 16 samples at most, everything beyond them is in double
    // precision, as in the streaming kernel.  Forward: of x and x^2 about zero, from n samples' sums about K
    auto fold = [&](const BandSums &part, uint32_t n, const Quad &K, const f32x2 &sa, const f32x2 &sb, const f32x2 &qa, const f32x2 &qb) {
      const float2 s0 = split(sa), s1 = split(sb), q0 = split(qa), q1 = split(qb), k0 = split(K.a), k1 = split(K.b);
      double S[4] = {s0.x, s0.y, s1.x, s1.y}, Q[4] = {q0.x, q0.y, q1.x, q1.y};
      if (DIR == 0) {
        const double k[4] = {k0.x, k0.y, k1.x, k1.y}, cnt = n;
#pragma unroll
        for (int e = 0; e < 4; ++e) { Q[e] = fma(k[e], fma(cnt, k[e], 2.0 * S[e]), Q[e]); S[e] = fma(cnt, k[e], S[e]); }
      }
      part.first[tid] = make_double2((S[0] + (b1 ? S[1] : 0.0)) + ((b2 ? S[2] : 0.0) + (b3 ? S[3] : 0.0)),
                                     (Q[0] + (b1 ? Q[1] : 0.0)) + ((b2 ? Q[2] : 0.0) + (b3 ? Q[3] : 0.0)));
      if (!b3 && live)
        part.second[grp * g.cb + chB] = make_double2((b1 ? 0.0 : S[1]) + ((b2 ? 0.0 : S[2]) + S[3]), (b1 ? 0.0 : Q[1]) + ((b2 ? 0.0 : Q[2]) + Q[3]));
    };
    // One tile.  FULL: it has all its rows, so no vector is missing (what threads without a column read and add up is not used).
    auto reduce = [&](auto full, uint32_t rows, uint32_t slot, uint32_t tm, const BandSums &part) {
      constexpr bool FULL = decltype(full)::value;
      const uint32_t slot_off = g.off_slots + slot * g.slot_stride;
      uint32_t ax = smem_u32(sm) + slot_off + off_s;
      if constexpr (DIR == 0) {
        Quad K = quad(0.f), nK = K;      // shift of the sums: per column the mean of its first four samples (or its first one)
        f32x2 sa = 0, sb = 0, qa = 0, qb = 0;
        const uint32_t n = FULL ? g.vpt : grp < rows ? min(g.vpt, (rows - grp - 1) / g.groups + 1) : 0u;
        auto there = [&](uint32_t i) { return FULL || i < n; };
        auto load = [&](Quad &x, uint32_t i) { if (there(i)) x = lds_quad(ax); ax += step_s; };      // (a missing vector is the shift)
        auto shift = [&](const Quad &sum, float inv) {
          auto of = [&](const f32x2 &s) { const float2 t = split(s); return pair(fabsf(t.x) < 1e36f ? t.x * inv : 0.f, fabsf(t.y) < 1e36f ? t.y * inv : 0.f); };
          K.a = of(sum.a); K.b = of(sum.b);      // (an infinity or a NaN is no shift, the sums show it)
          nK.a = mul2(K.a, pair(-1.f, -1.f)); nK.b = mul2(K.b, pair(-1.f, -1.f));
        };
        // (four samples' sums by themselves first, so that the thread's are rounded once per four of them)
        auto take = [&](const Quad &x0, const Quad &x1, const Quad &x2, const Quad &x3) {
          const f32x2 a0 = add2(x0.a, nK.a), a1 = add2(x1.a, nK.a), a2 = add2(x2.a, nK.a), a3 = add2(x3.a, nK.a);
          const f32x2 c0 = add2(x0.b, nK.b), c1 = add2(x1.b, nK.b), c2 = add2(x2.b, nK.b), c3 = add2(x3.b, nK.b);
          sa = add2(sa, add2(add2(a0, a1), add2(a2, a3))); sb = add2(sb, add2(add2(c0, c1), add2(c2, c3)));
          qa = add2(qa, fma2(a3, a3, fma2(a2, a2, fma2(a1, a1, mul2(a0, a0))))); qb = add2(qb, fma2(c3, c3, fma2(c2, c2, fma2(c1, c1, mul2(c0, c0)))));
        };
        auto take1 = [&](const Quad &x) {
          const f32x2 da = add2(x.a, nK.a), db = add2(x.b, nK.b);
          sa = add2(sa, da); qa = fma2(da, da, qa); sb = add2(sb, db); qb = fma2(db, db, qb);
        };
        uint32_t i = 0;
        for (; i + 4 <= g.vpt; i += 4, tm += 16) {
          Quad x0 = K, x1 = K, x2 = K, x3 = K;
          load(x0, i); load(x1, i + 1); load(x2, i + 2); load(x3, i + 3);
          if (i == 0) {
            shift(Quad{add2(add2(x0.a, x1.a), add2(x2.a, x3.a)), add2(add2(x0.b, x1.b), add2(x2.b, x3.b))}, FULL ? 0.25f : __fdividef(1.f, (float)max(min(n, 4u), 1u)));      // (a thread may have none)
            if constexpr (!FULL) { if (!there(0)) x0 = K; if (!there(1)) x1 = K; if (!there(2)) x2 = K; if (!there(3)) x3 = K; }
          }
          if constexpr (!FULL) __syncwarp();
          tmem_st(tm, x0, x1, x2, x3);
          take(x0, x1, x2, x3);
        }
        for (; i < g.vpt; ++i, tm += 4) {
          Quad x0 = K;
          load(x0, i);
          if (i == 0) shift(x0, 1.f);
          if constexpr (!FULL) __syncwarp();
          tmem_st(tm, x0);
          take1(x0);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->empty[slot]);
        fold(part, n, K, sa, sb, qa, qb);
      } else {
        const float4 *side = reinterpret_cast<const float4 *>(sm + g.off_side) + slot * kBandChannels;
        const float4 pA = side[chA], pB = side[chB];
        const Quad mean = spread(pA.x, pB.x), nmean = spread(-pA.x, -pB.x), scale = spread(pA.y, pB.y), beta = spread(pA.z, pB.z);
        f32x2 s1a = 0, s1b = 0, s2a = 0, s2b = 0;
        [[maybe_unused]] uint32_t r = grp;
        // a missing vector is (mean, 0), which adds nothing
        auto load = [&](Quad &x, Quad &gy, Quad &y) {
          y = quad(0.f);
          if constexpr (!FULL) { x = mean; gy = quad(0.f); }
          if (FULL || r < rows) {
            x = lds_quad(ax); gy = lds_quad(ax + g.plane_bytes);
            if constexpr (EXTRA) y = lds_quad(ax + 2 * g.plane_bytes);
          }
          ax += step_s;
          if constexpr (!FULL) r += g.groups;
        };
        auto work = [&](const Quad &x, const Quad &gy, Quad y, Quad &e, Quad &z) {
          e.a = add2(x.a, nmean.a); e.b = add2(x.b, nmean.b);
          if constexpr (!EXTRA) { y.a = fma2(e.a, scale.a, beta.a); y.b = fma2(e.b, scale.b, beta.b); }
          // dz = dy * act'(y)  (routines_gpu/flat_map.cu:191-192)
          z.a = mul2(gy.a, slopes(y.a, slope)); z.b = mul2(gy.b, slopes(y.b, slope));
          s1a = add2(s1a, z.a); s2a = fma2(z.a, e.a, s2a); s1b = add2(s1b, z.b); s2b = fma2(z.b, e.b, s2b);
        };
        uint32_t i = 0;
        for (; i + 2 <= g.vpt; i += 2, tm += 16) {
          Quad x0, g0, y0, x1, g1, y1, e0, z0, e1, z1;
          load(x0, g0, y0); load(x1, g1, y1);
          work(x0, g0, y0, e0, z0); work(x1, g1, y1, e1, z1);
          if constexpr (!FULL) __syncwarp();
          tmem_st(tm, e0, z0, e1, z1);
        }
        if (i < g.vpt) {
          Quad x0, g0, y0, e0, z0;
          load(x0, g0, y0);
          work(x0, g0, y0, e0, z0);
          if constexpr (!FULL) __syncwarp();
          tmem_st(tm, e0, z0);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->empty[slot]);
        fold(part, 0, mean, s1a, s1b, s2a, s2b);
      }
    };
    // alive: the thread has a column of this unit; base: the tile's first float, from which a thread's places are below 4 GB
    auto apply = [&](auto full, uint32_t rows, bool alive, size_t base, uint32_t slot, uint32_t tm, const float4 *coef) {
      constexpr bool FULL = decltype(full)::value;
      const float4 pA = coef[2 * chA], pB = coef[2 * chB];
      const Quad scale = spread(pA.y, pB.y);
      unsigned char *out = reinterpret_cast<unsigned char *>(a.out + base);
      uint32_t at = 4 * off_g, r = grp;
      tmem_wait_st();      // what this warp stored in the reduce visits
      auto next = [&] { at += 4 * step_g; if constexpr (!FULL) r += g.groups; };
      auto there = [&] { return alive && (FULL || r < rows); };
      if constexpr (DIR == 0) {
        uint32_t ae = smem_u32(sm) + g.off_slots + slot * g.slot_stride + off_s;
        const Quad nmean = spread(-pA.x, -pB.x), beta = spread(pA.z, pB.z);
        auto one = [&](const Quad &x) {
          Quad o;
          o.a = fma2(add2(x.a, nmean.a), scale.a, beta.a); o.b = fma2(add2(x.b, nmean.b), scale.b, beta.b);
          if constexpr (EXTRA) { const Quad e = lds_quad(ae); o.a = add2(o.a, e.a); o.b = add2(o.b, e.b); ae += step_s; }
          o.a = mul2(o.a, slopes(o.a, slope)); o.b = mul2(o.b, slopes(o.b, slope));
          if (there()) stg_stream(reinterpret_cast<float *>(out + at), o);
          next();
        };
        uint32_t i = 0;
        for (; i + 4 <= g.vpt; i += 4, tm += 16) {
          Quad x0, x1, x2, x3;
          tmem_ld(tm, x0, x1, x2, x3);
          one(x0); one(x1); one(x2); one(x3);
          __syncwarp();
        }
        for (; i < g.vpt; ++i, tm += 4) {
          Quad x0;
          tmem_ld(tm, x0);
          one(x0);
          __syncwarp();
        }
      } else {
        const Quad cB = spread(pA.w, pB.w), cC = spread(coef[2 * chA + 1].x, coef[2 * chB + 1].x);
        [[maybe_unused]] unsigned char *dres = EXTRA && a.dres ? reinterpret_cast<unsigned char *>(a.dres + base) : nullptr;
        // Accumulating writes: the next four vectors' old values are on their way while two are worked on, and the producer has brought the
        // tile to L2 ([256,1024,14,14]: one after the other from HBM 283 us, with both two ahead 202, four ahead 185).
        uint32_t far = at, rf = r;
        auto olds = [&](uint32_t i) {
          Quad q = quad(0.f);
          if constexpr (ADDS) {
            if (i < g.vpt && alive && (FULL || rf < rows)) q = ldg_quad(reinterpret_cast<const float *>(out + far));
            far += 4 * step_g; rf += g.groups;
          }
          return q;
        };
        auto one = [&](const Quad &e, const Quad &z, [[maybe_unused]] const Quad &old) {
          Quad o;
          o.a = fma2(scale.a, z.a, fma2(cB.a, e.a, cC.a)); o.b = fma2(scale.b, z.b, fma2(cB.b, e.b, cC.b));
          if (there()) {
            float *p = reinterpret_cast<float *>(out + at);
            if constexpr (ADDS) { o.a = add2(old.a, o.a); o.b = add2(old.b, o.b); }
            stg_stream(p, o);
            if constexpr (EXTRA) { if (dres) stg_stream(reinterpret_cast<float *>(dres + at), z); }
          }
          next();
        };
        uint32_t i = 0;
        if constexpr (ADDS) {
          Quad o0 = olds(0), o1 = olds(1), o2 = olds(2), o3 = olds(3);
          for (; i + 2 <= g.vpt; i += 2, tm += 16) {
            Quad e0, z0, e1, z1;
            tmem_ld(tm, e0, z0, e1, z1);
            const Quad n0 = olds(i + 4), n1 = olds(i + 5);
            one(e0, z0, o0); one(e1, z1, o1);
            o0 = o2; o1 = o3; o2 = n0; o3 = n1;
            __syncwarp();
          }
          if (i < g.vpt) {
            Quad e0, z0;
            tmem_ld(tm, e0, z0);
            one(e0, z0, o0);
          }
        } else {
          for (; i + 2 <= g.vpt; i += 2, tm += 16) {
            Quad e0, z0, e1, z1;
            tmem_ld(tm, e0, z0, e1, z1);
            one(e0, z0, e0); one(e1, z1, e1);
            __syncwarp();
          }
          if (i < g.vpt) {
            Quad e0, z0;
            tmem_ld(tm, e0, z0);
            one(e0, z0, e0);
          }
        }
      }
      __syncwarp();
    };
    BandWalk red(g, b, G), app(g, b, G);
    uint32_t slot = g.slots - 1, par = 1, qres = 0, rpar = 1, qcoef = 0, cpar = 0;
    uint32_t red_place = 0, app_place = 0;
    for (uint32_t s = 0; s < steps; ++s) {
      if (s < mine) {
        if (++slot == g.slots) { slot = 0; par ^= 1u; }
        bool ok = warp_wait(&ctl->res_empty[qres], rpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles);
        ok = ok && warp_wait(&ctl->full[slot], par, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles);
        if (!ok) break;
        const BandSums part(sm, g, qres);
        const uint32_t rows = N - red.k * g.rows, tm = tm0 + red_place * tm_step;
        if (rows >= g.rows) reduce(std::true_type{}, g.rows, slot, tm, part);
        else reduce(std::false_type{}, rows, slot, tm, part);
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->res_full[qres]);
        if (++qres == kBandQ) { qres = 0; rpar ^= 1u; }
        if (++red_place > g.look) red_place = 0;
        red.next();
      }
      if (s >= g.look) {
        if (!warp_wait(&ctl->coef_full[qcoef], cpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
        if constexpr (kSlotToo) {
          if (++slot == g.slots) { slot = 0; par ^= 1u; }
          if (!warp_wait(&ctl->full[slot], par, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
        }
        const uint32_t n0 = app.k * g.rows, c0 = app.unit * g.cb, rows = N - n0, tm = tm0 + app_place * tm_step;
        const bool alive = live && 4 * v < (C - c0) * dim0;
        const size_t base = (size_t)n0 * rs + (size_t)c0 * dim0;
        const float4 *coef = reinterpret_cast<const float4 *>(sm + g.off_coef) + qcoef * 2 * kBandChannels;
        if (rows >= g.rows) apply(std::true_type{}, g.rows, alive, base, slot, tm, coef);
        else apply(std::false_type{}, rows, alive, base, slot, tm, coef);
        if (lane == 0) { if (kSlotToo) mbar_arrive(&ctl->empty[slot]); mbar_arrive(&ctl->coef_empty[qcoef]); }
        if (++qcoef == kBandQ) { qcoef = 0; cpar ^= 1u; }
        if (++app_place > g.look) app_place = 0;
        app.next();
      }
    }
  } else if (warp == kBandWarps) {
    // ------------------------------------------------------------------ producer
    const uint64_t pol = g.whole ? policy_drop() : policy_normal();
    BandWalk red(g, b, G), app(g, b, G);
    uint32_t slot = g.slots - 1, par = 1, k = 0;
    bool ok = true;
    // backward: lane l has the parameters of the next tile's channel number l
    float4 raw = make_float4(0.f, 1.f, 1.f, 0.f);
    auto params = [&](uint32_t unit) {
      const uint32_t c = unit * g.cb + lane;
      if (DIR == 1 && lane < g.cb && c < C) {
        raw.x = a.mean_in[c]; raw.y = a.var_in[c];
        raw.z = a.gamma ? a.gamma[c] : 1.0f; raw.w = a.gamma && a.beta ? a.beta[c] : 0.f;
      }
    };
    if (mine) params(red.unit);
    for (uint32_t t = 0; ok && t < 2 * steps; ++t) {
      const uint32_t s = t >> 1, kind = t & 1u;
      if (kind == 0 ? s >= mine : !kSlotToo || s < g.look) continue;
      BandWalk &w = kind == 0 ? red : app;
      ++k;
      if (++slot == g.slots) { slot = 0; par ^= 1u; }
      uint32_t okw = 1;
      if (lane == 0) okw = mbar_wait(&ctl->empty[slot], par ^ 1u, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles) ? 1u : 0u;
      ok = __shfl_sync(0xffffffffu, okw, 0) != 0;
      if (!ok) { --k; break; }
      const uint32_t planes = kind == 0 ? kPlanes : 1u;
      if (lane == 0) mbar_expect_tx(&ctl->full[slot], planes * g.boxes * g.rows * g.box4 * 16);
      __syncwarp();
      if (lane < planes * g.boxes) {
        const uint32_t plane = lane / g.boxes, j = lane - plane * g.boxes;
        const CUtensorMap *map = kind == 1 || plane == 2 ? &maps.e : plane == 1 ? &maps.dy : &maps.x;
        tensor_g2s(smem_u32(sm + g.off_slots + (size_t)slot * g.slot_stride) + plane * g.plane_bytes + j * g.box_bytes, map,
                   w.unit * g.cb * dim0 + j * g.box4 * 4, w.k * g.rows, &ctl->full[slot], pol);
      }
      if (ADDS && kind == 0) {
        // what the apply visit adds to, on its way to L2
        const uint32_t n0 = w.k * g.rows, c0 = w.unit * g.cb, run = (C - c0 < g.cb ? C - c0 : g.cb) * dim0 * 4;
        for (uint32_t r = lane; r < g.rows && n0 + r < N; r += 32) bulk_prefetch(a.out + (size_t)(n0 + r) * rs + (size_t)c0 * dim0, run);
      }
      if (kind == 0 && DIR == 1) {
        float4 *side = reinterpret_cast<float4 *>(sm + g.off_side) + slot * kBandChannels;
        if (lane < g.cb) side[lane] = make_float4(raw.x, raw.z * inv_std(raw.y), raw.w, 0.f);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->full[slot]);
      w.next();
      if (kind == 0 && DIR == 1 && s + 1 < mine) params(w.unit);
    }
    // wait (bounded) for every copy that was issued: after an abort, of this warp or, now or later, of another, nobody else may
    if (lane == 0) {
      const uint32_t first = k > g.slots ? k - g.slots : 0;
      for (uint32_t kk = first; kk < k; ++kk) {
        const long long t0 = clock64();
        while (!mbar_try(&ctl->full[kk % g.slots], (kk / g.slots) & 1u) && clock64() - t0 < kDrainCycles) {}
      }
    }
  } else if (warp == kBandWarps + 1) {
    // ------------------------------------------------------------------ delivery warp
    const uint32_t lp = 1u << g.lane_shift, ci = lane >> g.lane_shift, sub = lane & (lp - 1u);
    const uint32_t v0 = ci * dim0 / 4, v1 = (ci * dim0 + dim0 - 1) / 4;      // the channel's first and last vector
    BandWord *buf = reinterpret_cast<BandWord *>(a.ws + g.tag);
    const size_t other = (size_t)g.total * g.cb;
    buffer();
    BandWord *now = buf + (ctl->parity ? other : 0), *then = buf + (ctl->parity ? 0 : other);
    BandWalk w(g, b, G);
    uint32_t q = 0, qpar = 0;
    size_t at = (size_t)b * g.cb + ci;
    for (uint32_t j = 0; j < mine; ++j) {
      const bool has = ci < g.cb && w.unit * g.cb + ci < C;
      if (!warp_wait(&ctl->res_full[q], qpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
      const BandSums part(sm, g, q);
      double t1 = 0.0, t2 = 0.0;
      // four of the lane's vectors at a time, their sums added in pairs: the loads are under way together (one vector after another:
      // 2.5 us a tile, the kernel's bound)
      uint32_t vi = v0 + sub, gi = has && vi <= v1 ? 0 : g.groups;
      while (gi < g.groups) {
        double2 p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          p[u] = make_double2(0.0, 0.0);
          if (gi < g.groups) {
            // (a vector that begins in the channel before holds this one's sums behind those)
            p[u] = 4 * vi >= ci * dim0 ? part.first[gi * g.L4 + vi] : part.second[gi * g.cb + ci];
            vi += lp;
            if (vi > v1) { vi = v0 + sub; ++gi; }
          }
        }
        t1 += (p[0].x + p[1].x) + (p[2].x + p[3].x); t2 += (p[0].y + p[1].y) + (p[2].y + p[3].y);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->res_empty[q]);
      if (++q == kBandQ) { q = 0; qpar ^= 1u; }
      for (uint32_t o = lp >> 1; o > 0; o >>= 1) { t1 += __shfl_xor_sync(0xffffffffu, t1, o); t2 += __shfl_xor_sync(0xffffffffu, t2, o); }
      if (has && sub == 0) {
        st_word(now + at, t1, t2);
        then[at] = BandWord{0ull, 0ull};
      }
      at += (size_t)G * g.cb;
      w.next();
    }
  } else {
    // ------------------------------------------------------------------ coefficient warp
    const uint32_t lp = 1u << g.lane_shift, ci = lane >> g.lane_shift, sub = lane & (lp - 1u);
    buffer();
    const BandWord *buf = reinterpret_cast<const BandWord *>(a.ws + g.tag) + (ctl->parity ? (size_t)g.total * g.cb : 0);
    BandWalk w(g, b, G);
    uint32_t q = 0, qpar = 1;
    float gm = 1.f, bt = 0.f, mean = 0.f, var = 1.f;
    auto params = [&](uint32_t unit) {
      const uint32_t c = unit * g.cb + ci;
      if (ci < g.cb && c < C) {
        gm = a.gamma ? a.gamma[c] : 1.0f; bt = a.gamma && a.beta ? a.beta[c] : 0.f;
        if (DIR == 1) { mean = a.mean_in[c]; var = a.var_in[c]; }
      }
    };
    if (mine) params(w.unit);
    bool ok = true;
    for (uint32_t n = 0; ok && n < mine; ++n) {
      const uint32_t c = w.unit * g.cb + ci;
      const bool has = ci < g.cb && c < C;
      const BandWord *words = buf + (size_t)w.unit * g.tiles * g.cb + ci;
      double s1 = 0.0, s2 = 0.0;
      const long long t0 = clock64();
      // The unit's words, P per lane at a time: all of them under way together, and added up in pairs.  The merge is the longest chain of a
      // step of many words, and every P beyond what a lane has costs instructions: always eight, and by their number, us backward,
      // [4096,1024,7,7], 412 words, 449 and 421, [128,2048,7,7], 64 words, 32.6 and 31.3.
      auto pull = [&](auto count) {
        constexpr uint32_t P = decltype(count)::value;
        for (uint32_t k0 = 0; k0 < g.tiles; k0 += P * lp) {
          BandWord r[P];
#pragma unroll
          for (uint32_t i = 0; i < P; ++i) r[i].lo = r[i].hi = has && k0 + sub + i * lp < g.tiles ? 0ull : 1ull << 63;
          for (;;) {
            bool all = true;
#pragma unroll
            for (uint32_t i = 0; i < P; ++i) {
              if (r[i].lo == 0ull || r[i].hi == 0ull) r[i] = ld_word(words + (size_t)(k0 + sub + i * lp) * g.cb);      // (one that has come is not asked for again)
              all = all && r[i].lo != 0ull && r[i].hi != 0ull;
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
          double lo[P], hi[P];
#pragma unroll
          for (uint32_t i = 0; i < P; ++i) { lo[i] = __longlong_as_double((long long)r[i].lo); hi[i] = __longlong_as_double((long long)r[i].hi); }
#pragma unroll
          for (uint32_t h = P / 2; h > 0; h /= 2)
#pragma unroll
            for (uint32_t i = 0; i < h; ++i) { lo[i] += lo[i + h]; hi[i] += hi[i + h]; }
          s1 += lo[0]; s2 += hi[0];
        }
        return true;
      };
      ok = g.tiles > 8 * lp ? pull(std::integral_constant<uint32_t, 16>{}) : g.tiles > 4 * lp ? pull(std::integral_constant<uint32_t, 8>{}) : pull(std::integral_constant<uint32_t, 4>{});
      if (!ok) break;
      for (uint32_t o = lp >> 1; o > 0; o >>= 1) { s1 += __shfl_xor_sync(0xffffffffu, s1, o); s2 += __shfl_xor_sync(0xffffffffu, s2, o); }
      if (!warp_wait(&ctl->coef_empty[q], qpar, ctl, status, ANODE_ST_WAIT_STATS, a.wait_cycles)) break;
      float4 *coef = reinterpret_cast<float4 *>(sm + g.off_coef) + q * 2 * kBandChannels + 2 * ci;
      const bool owner = w.k == 0;
      if (has && sub == 0) {
        if (DIR == 0) {
          const double m = s1 * g.inv_count;
          const float mf = (float)m;
          const float vf = (float)(not_below_zero(s2 - s1 * m) * g.inv_count + (double)a.epsilon);      // biased, epsilon folded in (batch_norm.cu:160)
          coef[0] = make_float4(mf, gm * inv_std(vf), bt, 0.f);
          if (owner) {
            a.mean[c] = mf; a.var[c] = vf;
            if (a.run_mean) { const float o = a.run_mean[c]; a.run_mean[c] = o + a.avg_rate * (mf - o); }
            if (a.run_var) { const float o = a.run_var[c]; a.run_var[c] = o + a.avg_rate * (vf - o); }
          }
        } else {
          const float rstd = inv_std(var);
          const double rs2 = (double)rstd * s2;                  // sum(dz * xhat)
          const double A = (double)gm * (double)rstd;
          coef[0] = make_float4(mean, gm * rstd, bt, (float)(-A * (double)rstd * rs2 * g.inv_count));
          coef[1] = make_float4((float)(-A * s1 * g.inv_count), 0.f, 0.f, 0.f);
          if (owner) {
            if (a.dbeta) a.dbeta[c] = (float)s1;
            if (a.dgamma) a.dgamma[c] = (float)rs2;
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&ctl->coef_full[q]);
      if (++q == kBandQ) { q = 0; qpar ^= 1u; }
      w.next();
      if (n + 1 < mine) params(w.unit);
    }
  }

  // ---- leave
  if (warp < kBandWarps) { __syncwarp(); tmem_wait_st(); }
  tmem_fence_before();
  __syncthreads();
  if (warp == 0) { tmem_fence_after(); tmem_free(ctl->tmem); }
  if (ctl->abort) {
    if (tid == 0) atomicOr(status, ANODE_ST_ABORTED);
    return;
  }
  if (!kAsk && tid == 0) {
    __threadfence();
    if (atomicAdd(counter, 1u) + 1 == gridDim.x) { counter[1] = ctl->parity ^ 1u; counter[0] = 0; }
  }
}

// ---- host side -------------------------------------------------------------------------------

typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiled encode_tiled()
{
  static const EncodeTiled f = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult r;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &r) != cudaSuccess || r != cudaDriverEntryPointSuccess) {
      (void)cudaGetLastError();
      p = nullptr;
    }
    return (EncodeTiled)p;
  }();
  return f;
}

static bool tensor_map(CUtensorMap &m, const float *p, uint32_t width, uint32_t N, uint32_t box, uint32_t rows)
{
  const cuuint64_t dims[2] = {width, N}, strides[1] = {4ull * width};
  const cuuint32_t boxes[2] = {box, rows}, one[2] = {1, 1};
  return encode_tiled()(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(p), dims, strides, boxes, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Where the streaming kernel hands a layer over: rows below those that the tiled kernel takes (tiled_takes), from so many elements
// on.  Below, the fill and the drain of the schedule, some 10 us, outweigh the second walk it saves.  Streaming kernel and this
// one, us:
//   forward    15.0 M [3699,203,20] 37.4 and 29.9, [548,596,46] 40.6 and 30.3, 16.1 M [320,1024,7,7] 32.1 and 30.6, 16.8 M [512,128,16,16] 34.2
//              and 30.8, 25.7 M [256,2048,7,7] 57.5 and 41.1
//   backward   8.0 M [80,2048,7,7] 24.1 and 24.0, [160,1024,7,7] 30.5 and 24.7, 9.7 M [200,400,11,11] 39.2 and 27.2, 12.8 M [128,2048,7,7]
//              45.4 and 32.6
//   residual   9.9 M [1508,71,92] 29.6 and 27.6, 10.0 M [200,1024,7,7] 29.4 and 28.8, 12.8 M [256,256,14,14] 34.8 and 27.5; backward 8.0 M
//              [80,2048,7,7] 34.1 and 32.9, [160,1024,7,7] 40.8 and 33.2
constexpr uint32_t kBandLongRow = 320, kBandWaveRow = 40;
// Forward passes of rows of 40 floats and more that the streaming kernel has in one wave of resident blocks (stream_one_wave) stay with it longer:
//   forward    [320,400,11,11] 15.5 M 23.4 and 27.9, [400,400,11,11] 19.4 M 33.1 and 32.9, [200,2048,7,7] 20.1 M 36.8 and 40.2,
//              [224,2048,7,7] 22.5 M 45.1 and 38.8, but [512,2048,4,4] 16.8 M 29.6 and 26.9, [512,1000,6,6] 18.4 M 31.7 and 31.0
//   residual   [96,2048,7,7] 9.6 M 24.1 and 27.1, [112,2048,7,7] 11.2 M 27.3 and 29.9, [256,400,11,11] 12.4 M 29.3 and 30.0,
//              [128,2048,7,7] 12.8 M 27.7 and 26.8
constexpr uint64_t kBandLeast[2][2] = {{15000000, 9000000}, {8000000, 8000000}};      // [direction][residual]
constexpr uint64_t kBandLeastWave[2] = {21000000, 12500000};      // forward, [residual]

bool band_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, BandGeom &g)
{
  const uint64_t elements = (uint64_t)dim0 * C * N;
  if (elements < kBandLeast[dir][extra] || dim0 >= kBandLongRow) return false;
  if (dir == 0 && elements < kBandLeastWave[extra] && dim0 >= kBandWaveRow && stream_one_wave(dim0, C, N, dir, extra)) return false;
  return band_geom(dim0, C, N, dir, extra, sm_count(), g);
}

// Lines that two units share are read by two blocks, one after the other.  Ordinary backward passes over tensors beyond L2 load them with the
// normal priority in the place of the one to be evicted first.  Us so and with the latter, backward, on two devices: [1024,2048,7,7] 202 and 206,
// [2048,1024,7,7] 205 and 210, [4096,1024,7,7] 418 and 436, [3000,512,7,7] 159 and 165, [2000,500,9,9] 172 and 177, [400,1024,14,14] 161 - 165 and
// 161; but [128,2048,7,7] 33 and 36 the other way round, runs of whole lines [2000,2048,4,4] 134 and 136.  It is not the traffic, every byte comes from
// HBM once either way ([1024,2048,7,7]: 822.4 and 822.9 MB for 822.1 of x and dy); why it gains is not known.
constexpr uint64_t kBandShared = 192ull << 20;      // bytes of x and dy
int launch_band(FusedArgs &a, const BandGeom &g, int dir, cudaStream_t stream)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  if (!encode_tiled()) return ANODE_E_LAUNCH;
  BandMaps m;
  const uint32_t width = a.plan.C * a.plan.dim0;
  if (!tensor_map(m.x, a.x, width, a.plan.N, g.box4 * 4, g.rows)) return ANODE_E_LAUNCH;
  m.dy = m.x; m.e = m.x;
  if (dir == 1 && !tensor_map(m.dy, a.dy, width, a.plan.N, g.box4 * 4, g.rows)) return ANODE_E_LAUNCH;
  if (extra && !tensor_map(m.e, dir == 0 ? a.res : a.ymask, width, a.plan.N, g.box4 * 4, g.rows)) return ANODE_E_LAUNCH;
  const void *k = dir == 0 ? (extra ? (const void *)bn_band_kernel<0, true, false> : (const void *)bn_band_kernel<0, false, false>)
                  : a.accumulate ? (extra ? (const void *)bn_band_kernel<1, true, true> : (const void *)bn_band_kernel<1, false, true>)
                                 : (extra ? (const void *)bn_band_kernel<1, true, false> : (const void *)bn_band_kernel<1, false, false>);
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, bool> ready;
  {
    int dev = 0;
    (void)cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(k, dev);
    auto it = ready.find(key);
    if (it == ready.end()) {
      const bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBandSmem) == cudaSuccess;
      if (!ok) (void)cudaGetLastError();
      it = ready.emplace(key, ok).first;
    }
    if (!it->second) return ANODE_E_LAUNCH;
  }
  BandGeom gg = g;
  gg.whole = dir == 0 || extra || (uint64_t)width * a.plan.N * 8 < kBandShared || g.L4 % 8 == 0;
  void *params[] = {(void *)&a, (void *)&gg, (void *)&m};
  if (cudaLaunchCooperativeKernel(k, dim3(g.grid), dim3(kBandThreads), params, kBandSmem, stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return ANODE_E_LAUNCH;
  }
  return ANODE_OK;
}

}  // namespace anode_b200
