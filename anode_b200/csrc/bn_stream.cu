// Fused batch-norm (+activation, +residual) for large layers of short rows, e.g. [1024, 2048, 7, 7]: a channel's data is
// thousands of short runs far apart, too many to hold on chip.
//
// A unit is a block of cb channels, i.e. per sample one contiguous, 16-byte aligned run of cb*dim0 floats.  A
// thread-block CLUSTER owns one unit and splits its samples; a thread keeps one float4 column of the run and walks down
// the samples twice:
//   1. statistics: kBatch 128-bit loads in flight per thread, shifted sums (or the backward sums) per column in registers,
//      folded over the block's threads in a fixed order in double precision;
//   2. each block pushes its channel sums into every block of the cluster (remote shared memory), one cluster barrier;
//   3. every block merges them in rank order (bit-identical coefficients) and walks its samples again, last batch first:
//      that one is still in registers, the others come from L2.  The cluster size keeps what all resident blocks have
//      between their two walks within reach of L2 (kStreamWindow).
//
// (The largest of these layers are walked once, by bn_band.cu, where the call has a workspace.)
//
// Rows without an aligned run (C*dim0 or every run of a few channels no multiple of four floats) take the masked form.  They went
// float by float through the plain kernel, some 20 instructions per element and a grid-wide agreement; forward / backward, us, there
// and here: [4096,23,7,7] 44 / 45 and 20 / 30, [647,340,351] 317 / 618 and 158 / 268, [2571,573,75] 450 / 610 and 240 / 369, [4160,7,33]
// 21 / 20 and 8 / 10, residual [2374,147,83] 226 / 271 and 94 / 157.  Error against float64 over 60 shapes, there and here, geometric mean:
// mean 4.9e-8 and 2.5e-8, variance 4.8e-8 and 3.0e-8, dgamma 1.5e-7 and 1.2e-7, dbeta 1.3e-7 and 7.9e-8.
//
// What bounds it: HBM and the loads in flight.  Nothing is staged in shared memory, so the blocks per SM are limited by
// registers only and some stream while others fold and wait; the kernel that holds the slices in shared memory
// (bn_segres.cu) runs its load, six dependent phases and store one after the other.
// Forward / backward: [1024,2048,7,7] 203 / 436 us there, 179 / 298 us here (0.70 / 0.63 of the copy bandwidth),
// [256,1024,14,14] backward 164 -> 147; where a unit does not fit sixteen blocks' shared memory and the plain kernel
// served the layer, [4096,512,7,7] 490 / 797 -> 206 / 338, [1024,64,15,15] 87 / 178 -> 31 / 54, residual
// [1024,2048,7,7] 383 / 1151 -> 248 / 420.
//
// Reference kernels this replaces: routines_gpu/batch_norm.cu:24-57, 125-163, 314-336 (forward), :181-206, 240-280,
// 354-376, 408-444, 476-515 (backward), flat_map.cu:172-194 (ReLU).
#include <math.h>

#include "bn_device.cuh"
#include "bn_host.h"

namespace anode_b200 {

// Most threads of a block, and blocks per SM.  [1024,2048,7,7] forward / backward: three of 256 threads (80 registers)
// 180 / 298 us, two of 448 (72) 193 / 319, two of 352 (88) 190 / 304, four of 256 (64) 251 / 392.
constexpr uint32_t kStreamThreads = 256, kStreamBlocks = 3;
constexpr uint32_t kStreamRecords = 1024;    // most channels * blocks of a unit
constexpr uint32_t kStreamChannels = 128;    // most channels of a unit

// RAG: runs that begin anywhere (the masked form).  A thread's samples lie a multiple of four floats apart, so its 16-byte vectors,
// from the boundary below the run's start to the one above its end, always lie over the run in the same way: floats lo to hi of a
// vector are the run's, the others belong to a neighbour, have sums of their own in the thread and are left out when it is folded.
template <int DIR, bool EXTRA, bool RAG>
__global__ void __launch_bounds__(kStreamThreads, kStreamBlocks) bn_stream_kernel(const FusedArgs a, const StreamGeom g)
{
  // samples in flight per thread (more of them spill; four of the masked residual backward, too)
  constexpr int kBatch = DIR == 0 && !EXTRA ? 8 : RAG && DIR == 1 && EXTRA ? 3 : 4;
  __shared__ double2 part[2][kStreamThreads];            // per thread: its sums for the one or two channels of its column
  __shared__ double2 rec[kStreamRecords];                // [channel][block of the cluster]
  __shared__ float4 coef0[kStreamChannels];              // mean, gamma/std, beta, -
  __shared__ float2 coef1[kStreamChannels];              // backward: factor of x - mean, constant
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = (blockDim.x + 31) >> 5;
  const uint32_t csh = (uint32_t)__ffs((int)g.cluster) - 1u;
  const uint32_t u = blockIdx.x >> csh, rank = blockIdx.x & (g.cluster - 1u);
  const uint32_t dim0 = a.plan.dim0, C = a.plan.C, N = a.plan.N;
  // remote shared memory may only be written once its block runs (collected right before the first remote store)
  if (g.cluster > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t c0 = u * g.cb, cw = C - c0 < g.cb ? C - c0 : g.cb;
  const uint32_t run = cw * dim0, L4 = RAG ? (run + 6) / 4 : run / 4, rs = C * dim0;
  const uint32_t grp = tid / L4, v = tid - grp * L4;
  const uint32_t n0 = rank * g.rows, rows = n0 < N ? (N - n0 < g.rows ? N - n0 : g.rows) : 0;
  const uint32_t step = g.groups * rs;                   // float offsets are below 2^32 (check_dims) wherever k < nk
  const uint32_t start = (n0 + grp) * rs + c0 * dim0, mis = RAG ? start & 3u : 0u;
  const uint32_t off0 = start - mis + 4 * v;
  const uint32_t lo = RAG && v == 0 ? mis : 0u, hi = !RAG || 4 * v + 4 <= run + mis ? 4u : 4 * v < run + mis ? run + mis - 4 * v : 0u;
  const bool whole = !RAG || (lo == 0 && hi == 4);
  const uint32_t nk = grp < g.groups && grp < rows && lo < hi ? (rows - grp - 1) / g.groups + 1 : 0;      // this thread's samples
  // the column's four floats lie in channel chA up to float eB, in the next one from there on
  const uint32_t chA = grp < g.groups && lo < hi ? (4 * v + lo - mis) / dim0 : 0;
  const uint32_t eB = (chA + 1) * dim0 + mis - 4 * v;
  const uint32_t chB = eB < hi && chA + 1 < cw ? chA + 1 : chA;
  // Of a tensor that ends inside a vector the floats up to its end are read one by one.
  const uint32_t end = RAG ? N * rs - 4 : 0u;
  auto load = [&](const float *p, uint32_t off, uint64_t pol) {
    if (!RAG || off <= end) return Pack<4>::load(p + off, pol);
    Pack<4> r = pack_fill<4>(0.f);
#pragma unroll
    for (int e = 0; e < 3; ++e) if (off + e < end + 4) r.v[e] = p[off + e];
    return r;
  };
  auto store = [&](const Pack<4> &o, float *p, bool later) {      // later: the block reads it again
    if (whole) { if (later) o.put(p); else o.store_stream(p); return; }
#pragma unroll
    for (int e = 0; e < 4; ++e) if ((uint32_t)e >= lo && (uint32_t)e < hi) p[e] = o.v[e];
  };
  const float slope = a.neg_slope;                       // activation: t * (t > 0 ? 1 : slope)
  const bool early = DIR == 1 && EXTRA && a.dres_early;  // dz is stored in the first walk and read back in the second
  const uint64_t keep = policy_keep(), drop = policy_drop();
  pdl_wait();
  pdl_trigger();

  float mean[4], scale[4], beta[4];
  if (DIR == 1) {
    const float mA = a.mean_in[c0 + chA], mB = a.mean_in[c0 + chB];
    const float sA = (a.gamma ? a.gamma[c0 + chA] : 1.0f) * inv_std(a.var_in[c0 + chA]);
    const float sB = (a.gamma ? a.gamma[c0 + chB] : 1.0f) * inv_std(a.var_in[c0 + chB]);
    const float bA = a.gamma && a.beta ? a.beta[c0 + chA] : 0.f, bB = a.gamma && a.beta ? a.beta[c0 + chB] : 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) { const bool b = (uint32_t)e >= eB; mean[e] = b ? mB : mA; scale[e] = b ? sB : sA; beta[e] = b ? bB : bA; }
  }

  // ---- first walk
  Pack<4> vx[kBatch], vd[DIR == 1 ? kBatch : 1];         // after the walk: the last batch (vd: its dz)
  float s[4] = {0.f, 0.f, 0.f, 0.f}, q[4] = {0.f, 0.f, 0.f, 0.f}, K[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t kb = 0;
  for (uint32_t k = 0; k < nk; k += kBatch) {
    kb = k;
    Pack<4> vm[DIR == 1 && EXTRA ? kBatch : 1];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const uint32_t off = off0 + (k + i) * step;
      vx[i] = pack_fill<4>(0.f);
      if (k + i < nk) {
        vx[i] = load(a.x, off, keep);
        if (DIR == 1) vd[i] = load(a.dy, off, early ? drop : keep);
        if (DIR == 1 && EXTRA) vm[i] = load(a.ymask, off, early ? drop : keep);
      }
    }
    if (DIR == 0) {
      if (k == 0) {
        // shift of the sums: the mean of the column's first batch
        const float inv = __fdividef(1.0f, (float)(nk < kBatch ? nk : kBatch));
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float t = 0.f;
#pragma unroll
          for (int i = 0; i < kBatch; ++i) t += vx[i].v[e];
          K[e] = fabsf(t) < 1e36f ? t * inv : 0.f;      // (an infinity or a NaN is no shift, the sums show it)
        }
      }
      // batch by batch, so that a long column's sums are rounded once per batch
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float bs = 0.f, bq = 0.f;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const float d = k + i < nk ? vx[i].v[e] - K[e] : 0.f;
          bs += d; bq = fmaf(d, d, bq);
        }
        s[e] += bs; q[e] += bq;
      }
    } else {
#pragma unroll
      for (int i = 0; i < kBatch; ++i)
        if (k + i < nk) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float d = vx[i].v[e] - mean[e];
            const float yb = EXTRA ? vm[i].v[e] : fmaf(d, scale[e], beta[e]);
            vd[i].v[e] *= yb > 0.0f ? 1.0f : slope;      // dz = dy * act'(y)  (routines_gpu/flat_map.cu:191-192)
            s[e] += vd[i].v[e]; q[e] = fmaf(vd[i].v[e], d, q[e]);
          }
          if (EXTRA && early) store(vd[i], a.dres + (off0 + (k + i) * step), true);
        }
    }
  }

  // ---- the thread's sums for its channels: of x and x^2 about zero (from the shifted sums, in double precision: nothing
  // that the f32 sums hold is lost), or the backward sums
  {
    double2 p[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      double t1 = (double)s[e], t2 = (double)q[e];
      if (DIR == 0) {
        const double n = (double)nk, k = (double)K[e];
        t2 = fma(k, fma(n, k, 2.0 * t1), t2); t1 = fma(n, k, t1);
      }
      const bool b = (uint32_t)e >= eB;
      if (RAG && ((uint32_t)e < lo || (uint32_t)e >= hi)) t1 = t2 = 0.0;
      p[0].x += b ? 0.0 : t1; p[0].y += b ? 0.0 : t2;
      p[1].x += b ? t1 : 0.0; p[1].y += b ? t2 : 0.0;
    }
    part[0][tid] = p[0]; part[1][tid] = p[1];
  }
  __syncthreads();

  // ---- the block's sums: one warp per channel over the threads whose column touches it, in a fixed order
  if (g.cluster > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (uint32_t ci = warp; ci < cw; ci += warps) {
    const uint32_t f0 = ci * dim0, nv = RAG ? (dim0 + 6) / 4 : (f0 + dim0 - 1) / 4 - f0 / 4 + 1;
    double t1 = 0.0, t2 = 0.0;
    for (uint32_t i = lane; i < nv * g.groups; i += 32) {
      const uint32_t gi = i / nv, m = RAG ? ((n0 + gi) * rs + c0 * dim0) & 3u : 0u, vi = (f0 + m) / 4 + i - gi * nv;
      if (RAG && 4 * vi >= f0 + dim0 + m) continue;
      const double2 p = part[ci > 0 && 4 * vi < f0 + m ? 1 : 0][gi * L4 + vi];     // (a column that starts in the channel before)
      t1 += p.x; t2 += p.y;
    }
    t1 = warp_sum_all(t1); t2 = warp_sum_all(t2);
    if (g.cluster > 1) { if (lane < g.cluster) st_cluster_d2(&rec[ci * g.cluster + rank], lane, t1, t2); }
    else if (lane == 0) rec[ci] = make_double2(t1, t2);
  }
  if (g.cluster > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }

  // ---- merged in rank order by every block; block 0 writes the channel's results
  for (uint32_t ci = tid; ci < cw; ci += blockDim.x) {
    const uint32_t c = c0 + ci;
    double t1 = 0.0, t2 = 0.0;
    for (uint32_t r = 0; r < g.cluster; ++r) { const double2 p = rec[ci * g.cluster + r]; t1 += p.x; t2 += p.y; }
    const float gm = a.gamma ? a.gamma[c] : 1.0f;
    const float bt = (a.gamma && a.beta) ? a.beta[c] : 0.0f;
    if (DIR == 0) {
      const double md = t1 * g.inv_count;
      const float mf = (float)md;
      const float vf = (float)(not_below_zero(t2 - t1 * md) * g.inv_count + (double)a.epsilon);      // biased, epsilon folded in (batch_norm.cu:160)
      coef0[ci] = make_float4(mf, gm * inv_std(vf), bt, 0.f);
      if (rank == 0) {
        a.mean[c] = mf; a.var[c] = vf;
        if (a.run_mean) { const float o = a.run_mean[c]; a.run_mean[c] = o + a.avg_rate * (mf - o); }
        if (a.run_var) { const float o = a.run_var[c]; a.run_var[c] = o + a.avg_rate * (vf - o); }
      }
    } else {
      const float rstd = inv_std(a.var_in[c]);
      const double rs2 = (double)rstd * t2;              // sum(dz * xhat)
      const double A = (double)gm * (double)rstd;
      coef1[ci] = make_float2((float)(-A * (double)rstd * rs2 * g.inv_count), (float)(-A * t1 * g.inv_count));
      if (rank == 0) {
        if (a.dbeta) a.dbeta[c] = (float)t1;
        if (a.dgamma) a.dgamma[c] = (float)rs2;
      }
    }
  }
  __syncthreads();
  if (!nk) return;

  // ---- second walk, last batch first
  float cB[4], cC[4];
  if (DIR == 0) {
    const float4 cA = coef0[chA], cBf = coef0[chB];
#pragma unroll
    for (int e = 0; e < 4; ++e) { const bool b = (uint32_t)e >= eB; mean[e] = b ? cBf.x : cA.x; scale[e] = b ? cBf.y : cA.y; beta[e] = b ? cBf.z : cA.z; }
  } else {
    const float2 cA = coef1[chA], cBf = coef1[chB];
#pragma unroll
    for (int e = 0; e < 4; ++e) { const bool b = (uint32_t)e >= eB; cB[e] = b ? cBf.x : cA.x; cC[e] = b ? cBf.y : cA.y; }
  }
  for (uint32_t k = kb;; k -= kBatch) {
    if (DIR == 0) {
      if (k != kb) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) vx[i] = load(a.x, off0 + (k + i) * step, drop);      // (only the last batch is short)
      }
#pragma unroll
      for (int h = 0; h < kBatch; h += 4) {
        Pack<4> ve[EXTRA ? 4 : 1];
        if (EXTRA) {
#pragma unroll
          for (int i = 0; i < 4; ++i) if (k + h + i < nk) ve[i] = load(a.res, off0 + (k + h + i) * step, drop);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (k + h + i < nk) {
            Pack<4> o;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              float yb = fmaf(vx[h + i].v[e] - mean[e], scale[e], beta[e]);
              if (EXTRA) yb += ve[i].v[e];
              o.v[e] = yb * (yb > 0.0f ? 1.0f : slope);
            }
            store(o, a.out + (off0 + (k + h + i) * step), false);
          }
      }
    } else {
      if (a.accumulate) {      // what is added to, on its way to L2 (registers for all of a batch would spill)
#pragma unroll
        for (int i = 0; i < kBatch; ++i) if (k + i < nk) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.out + (off0 + (k + i) * step)));
      }
      if (k != kb) {
        const float *second = early ? a.dres : a.dy;
        Pack<4> vm[EXTRA ? kBatch : 1];
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          const uint32_t off = off0 + (k + i) * step;
          vx[i] = load(a.x, off, drop);
          vd[i] = load(second, off, drop);
          if (EXTRA && !early) vm[i] = load(a.ymask, off, drop);
        }
        if (!early) {
#pragma unroll
          for (int i = 0; i < kBatch; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float yb = EXTRA ? vm[i].v[e] : fmaf(vx[i].v[e] - mean[e], scale[e], beta[e]);
              vd[i].v[e] *= yb > 0.0f ? 1.0f : slope;
            }
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i)
        if (k + i < nk) {
          const uint32_t off = off0 + (k + i) * step;
          Pack<4> o;
          if (a.accumulate) o = load(a.out, off, drop);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float dx = fmaf(scale[e], vd[i].v[e], fmaf(cB[e], vx[i].v[e] - mean[e], cC[e]));
            o.v[e] = a.accumulate ? o.v[e] + dx : dx;
          }
          store(o, a.out + off, false);
          if (EXTRA && !early && a.dres) store(vd[i], a.dres + off, false);
        }
    }
    if (k == 0) break;
  }
}

// ---- host side -------------------------------------------------------------------------------

// Bytes that the resident blocks may have between their two walks.  It wants to fit L2, but a large cluster waits longer
// for its slowest block and leaves more SMs without a place for a whole cluster: [1024,2048,7,7] takes 199 / 343 us
// with 64 MB (clusters of 8 / 16), 180 / 298 with 96 MB (4 / 8) and the same with 128 MB.
constexpr uint64_t kStreamWindow = 96ull << 20;
constexpr uint64_t kStreamSplit = 72ull << 20;

static bool stream_geom(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, StreamGeom &g)
{
  if (dim0 < 4 || (uint64_t)C * dim0 % 4 != 0) return false;
  uint32_t q = 4; if (dim0 % 2 == 0) q = 2; if (dim0 % 4 == 0) q = 1;      // cb*dim0 must be a multiple of 4
  // runs of at least 512 bytes, then the channel count that leaves the fewest of a block's threads without a column, as
  // long as there are units for a block at every place of the device (of runs up to a kilobyte, for some 64 blocks)
  // (forward / backward, us, with the fewest idle threads alone and now: [6688,120,11] 32 and 160 blocks, 151 / 350 and
  // 22 / 37; [724,524,11] 96 and 352, 24 / 41 and 10 / 14)
  uint32_t best = 0, best_used = 0;
  for (uint32_t cb = q; cb <= C && cb <= kStreamChannels && (uint64_t)cb * dim0 <= 4 * kStreamThreads; cb += q) {
    const uint32_t L4 = cb * dim0 / 4, used = kStreamThreads / L4 * L4;
    if (best * dim0 >= 128 && (used * 16 <= best_used * 17 ||
                               ceil_div_u32(C, cb) * 16 < (cb * dim0 <= 256 ? 64u : kStreamBlocks * sm_count()))) continue;
    best = cb; best_used = used;
  }
  if (!best) return false;
  const uint32_t L4 = best * dim0 / 4;
  g.cb = best; g.units = ceil_div_u32(C, best);
  g.groups = kStreamThreads / L4; if (g.groups > N) g.groups = N;
  const uint64_t unit_bytes = 16ull * L4 * N * (dir == 1 ? 2 : 1);
  // Large layers: clusters that keep to the window.  Small ones: as many blocks as are resident at once, a few more at
  // most, and four samples per thread at least; a second wave only repeats each block's fixed steps: [43,832,183] 1664
  // blocks and 416, 19.3 / 25.7 us and 12.7 / 18.2; [995,1892,6] 1264 and 316, 38 / 54 and 21 / 41.  (Backward passes over
  // more than 72 MB gain by what a second or third wave takes out of L2's way: [264,968,37] one wave 34.7 us, two 31.8.)
  const uint32_t wave = kStreamBlocks * sm_count();
  const bool split = dir == 1 && unit_bytes * g.units > kStreamSplit;
  const uint32_t most = split ? 3 * wave : wave * 8 / 7, least = split ? 9 : 4;
  uint32_t cl = 1;
  while (cl < 16 && cl * 2 * g.cb <= kStreamRecords &&
         (wave * unit_bytes / cl > kStreamWindow || (g.units * cl * 2 <= most && N / (cl * 2) >= g.groups * least))) cl *= 2;
  // A wave and less than a third of another: the rest of the blocks costs most of a second wave.  Another unit and cluster may make
  // nearly a whole one, with nearly all threads.  Forward / backward, us, before and after: [128,2048,7,7] 512 and 412 blocks 26.4 / 33.0 and
  // 21.2 / 33.0 (backward in three waves either way), [64,2048,7,7] 17.9 / 25.8 and 15.4 / 20.5, [32,2048,7,7] 11.4 / 15.4 and 10.0 / 13.8,
  // [150,1000,6,6] 500 and 400 blocks 16.8 / 22.2 and 12.7 / 17.9.
  // The SMs of a cluster lie together, so larger ones leave places empty, and one that does not fit makes a second wave: in clusters of eight 376
  // blocks are resident and 400 are not, in clusters of four 412 are and 432 not.  [112,1000,7,7], 500 blocks and 400 in clusters of eight,
  // 17.2 / 22.4 and 19.5 / 27.9, [723,2048,4,4], 512 and 432 in clusters of four, 50 and 58, but [140,940,7,7], 470 and 376, 17.5 and 16.6.
  // The residual backward pass wants six samples per thread, too: [20,2000,7,7] 11.9 and, with five, 12.9.
  uint32_t run = L4;      // vectors
  if (!split && g.units * cl > wave && g.units * cl * 3 <= wave * 4 && g.groups * L4 > 192) {      // (of fewer threads four blocks are resident)
    uint32_t most_threads = wave * kStreamThreads * 25 / 32;
    for (uint32_t cb = q; cb <= C && cb <= kStreamChannels && (uint64_t)cb * dim0 <= 4 * kStreamThreads; cb += q) {
      const uint32_t V = cb * dim0 / 4, units = ceil_div_u32(C, cb), groups = kStreamThreads / V < N ? kStreamThreads / V : N;
      if (cb * dim0 < 128) continue;
      for (uint32_t n = 1; n <= 8 && n * cb <= kStreamRecords && N / n >= groups * (dir == 1 && extra ? 6 : least); n *= 2) {
        const uint32_t blocks = units * n, resident = n == 8 ? wave * 17 / 20 : n == 4 ? wave * 15 / 16 : wave;
        if (blocks <= resident && blocks * groups * V > most_threads && wave * (16ull * V * N * (dir == 1 ? 2 : 1)) / n <= kStreamWindow) {
          most_threads = blocks * groups * V;
          cl = n; run = V; g.cb = cb; g.units = units; g.groups = groups;
        }
      }
    }
  }
  g.cluster = cl;
  g.rows = ceil_div_u32(N, cl);
  if (g.groups > g.rows) g.groups = g.rows;
  g.threads = (g.groups * run + 31) / 32 * 32;
  g.inv_count = 1.0 / ((double)dim0 * (double)N);
  return true;
}

// Estimated us of units of `cb` channels and clusters of `cl` blocks: a fixed part per wave of blocks (clusters of 8 and 16 fill 85 and
// 78 per cent of the device's places), and the larger of a thread's chain of batches and the bytes moved, where the cache lines that
// two runs share come twice, what exceeds L2 between the two walks comes again, and idle threads leave bandwidth unused.  The
// figures are fitted to 570 launches of the masked form, 60 shapes (16 to 480 floats a row, 3 to 1500 channels, 0.6 to 120 M elements, four
// directions) with up to 30 units and clusters each: what is chosen by it is 3 per cent above the best of them on average.
// (parts: a last wave counts as much of one as it fills.)
static double stream_cost(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, bool masked, uint32_t cb, uint32_t cl, uint32_t groups, uint32_t L4,
                          bool parts = false)
{
  const uint32_t wave = kStreamBlocks * sm_count(), run = cb * dim0, rows = ceil_div_u32(N, cl), used = groups < rows ? groups : rows;
  const double bytes = 4.0 * dim0 * C * N * (dir == 0 ? (extra ? 3 : 2) : extra ? 5 : 3);
  const double sample = (dir == 0 && !extra ? 1.5 : 2.0) / (dir == 0 ? (extra ? 4 : 8) : extra && masked ? 3 : 4);      // us per sample of a thread
  const double window = 77e6, rate = 5.15e6;      // bytes that L2 keeps; bytes per us
  const uint64_t blocks = (uint64_t)ceil_div_u32(C, cb) * cl, places = cl == 16 ? wave * 25 / 32 : cl == 8 ? wave * 17 / 20 : cl == 4 ? wave * 15 / 16 : wave;
  const double waves = parts && blocks > places ? (double)blocks / places : (double)((blocks + places - 1) / places);
  const double resident = (double)(blocks < places ? blocks : places);
  const double over = 4.0 * run * N * (dir == 1 ? 2 : 1) / cl * resident / window - 1;
  const double again = (dir == 1 ? 0.5 : 0.17) * (over < 0 ? 0 : over > 1 ? 1 : over), lanes = resident * used * L4 / ((double)wave * kStreamThreads);
  const double moved = bytes * (1 + 9.0 / run) * (1 + again) / rate * (0.9 + 0.1 / lanes);
  const double chain = waves * ceil_div_u32(rows, used) * sample;
  return 0.6 + waves * (3.0 + 0.024 * cl) + pow(pow(moved, 2.5) + pow(chain, 2.5), 0.4);
}

// The next number of channels to look at: all up to eight steps of q, then an eighth more each time.
static uint32_t next_unit(uint32_t cb, uint32_t q) { return cb + (cb / 8 > q ? cb / 8 / q * q : q); }

static void stream_set(StreamGeom &g, uint32_t C, uint32_t N, uint32_t cb, uint32_t cl, uint32_t groups, uint32_t L4)
{
  g.cb = cb; g.units = ceil_div_u32(C, cb); g.cluster = cl; g.rows = ceil_div_u32(N, cl);
  g.groups = groups < g.rows ? groups : g.rows;
  g.threads = (g.groups * L4 + 31) / 32 * 32;
}

// What the estimate of runs of aligned channels, with the last wave in parts, is multiplied by where it is held against the kernel for long
// rows (long_plan).  The smaller one of the two is launched: of 450 passes of 250 to 510 floats a row, forward, residual forward, backward and
// residual backward are 2.9, 0.8, 0.4 and 1.0 per cent above the better one (121 to 161 each, of forward passes 7), always this kernel would be
// 22, 4.5, 5.6 and 3.0; of 241 passes without such runs, with whole waves and no factor, 1.7, 3.2, 2.0 and 0.8, and 1.8, 5.0, 9.2 and 6.6.
// [207,54,262] backward 13.8 us here and 18.0, [169,32,254] residual backward 10.4 and 11.0, [197,44,270] backward 16.3 and 11.0.
constexpr double kStreamAligned = 0.87;

// The geometry that is launched: stream_geom's, or the one of the least estimated time where that is this much less.  Us so and with
// stream_geom's alone, forward, backward, residual forward and backward: [3865,36,18] 8.9, 11.7, 10.7, 15.4 and 11.0, 17.4, 16.9, 23.3, [1148,44,80]
// 9.4, 14.6, 11.7, 19.3 and 13.4, 21.2, 18.0, 25.6, [20,1998,102] 9.7, 13.8, 11.4, 18.7 and 14.0, 16.6, 16.6, 19.6, [148,750,38] 9.4, 15.1, 12.6, 20.4 and
// 19.9, 26.4, 23.1, 30.0; 5 to 9 per cent less over 120 shapes.  (Without the margin some were slower, [1217,108,87] 23.5 and 27.4.)
constexpr double kStreamOther = 0.85;
bool stream_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, StreamGeom &g)
{
  if (!stream_geom(dim0, C, N, dir, extra, g)) return false;
  const uint32_t q = dim0 % 4 == 0 ? 1 : dim0 % 2 == 0 ? 2 : 4;
  double best = kStreamOther * stream_cost(dim0, C, N, dir, extra, false, g.cb, g.cluster, g.groups, g.cb * dim0 / 4);
  for (uint32_t cb = q; cb <= C && cb <= kStreamChannels && cb * dim0 <= 4 * kStreamThreads; cb = next_unit(cb, q)) {
    const uint32_t L4 = cb * dim0 / 4, groups = kStreamThreads / L4 < N ? kStreamThreads / L4 : N;
    if (cb * dim0 < 32 && cb + q <= C) continue;
    for (uint32_t cl = 1; cl <= 16 && cl * cb <= kStreamRecords && (cl == 1 || N / cl >= groups * 2); cl *= 2) {
      const double cost = stream_cost(dim0, C, N, dir, extra, false, cb, cl, groups, L4);
      if (cost < best) { best = cost; stream_set(g, C, N, cb, cl, groups, L4); }
    }
  }
  g.cost = (float)(kStreamAligned * stream_cost(dim0, C, N, dir, extra, false, g.cb, g.cluster, g.groups, g.cb * dim0 / 4, true));
  return true;
}

// The masked form (RAG): runs of any channels.  The samples of a thread lie a multiple of four floats apart, so the groups of a
// block are an even number or a multiple of four where C*dim0 asks for it (unless a thread has one sample anyway), and rows are
// no longer than leaves place for those.  (The least idle threads and the aligned form's clusters, as chosen by stream_geom, were 11 per
// cent slower over 70 shapes, a third at 3 to 10 channels.)
bool masked_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, StreamGeom &g)
{
  const uint32_t rs = C * dim0, m = rs % 4 == 0 ? 1u : rs % 2 == 0 ? 2u : 4u;
  StreamGeom aligned;
  if (dim0 < 4 || stream_geom(dim0, C, N, dir, extra, aligned)) return false;
  double best = 0;
  for (uint32_t cb = 1; cb <= C && cb <= kStreamChannels && ((uint64_t)cb * dim0 + 6) / 4 <= kStreamThreads; cb = next_unit(cb, 1)) {
    const uint32_t L4 = (cb * dim0 + 6) / 4;
    if (cb * dim0 < 16 && cb < C) continue;
    uint32_t groups = kStreamThreads / L4;
    groups = groups >= N ? N : groups / m * m;
    if (groups == 0) break;
    for (uint32_t cl = 1; cl <= 16 && cl * cb <= kStreamRecords && (cl == 1 || N / cl >= groups * 2); cl *= 2) {
      const double cost = stream_cost(dim0, C, N, dir, extra, true, cb, cl, groups, L4);
      if (best == 0 || cost < best) { best = cost; g.cost = (float)cost; stream_set(g, C, N, cb, cl, groups, L4); }
    }
  }
  g.inv_count = 1.0 / ((double)dim0 * (double)N);
  return best != 0;
}

// Whether stream_geom's grid is one wave of blocks, all resident, that fills the device: nothing of a second wave to pay for.
bool stream_one_wave(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra)
{
  StreamGeom g;
  if (!stream_geom(dim0, C, N, dir, extra, g)) return false;
  const uint32_t wave = kStreamBlocks * sm_count(), blocks = g.units * g.cluster;
  return g.cluster <= 4 && blocks * 20 >= wave * 17 && blocks <= (g.cluster == 4 ? wave * 15 / 16 : wave);
}

// The rules that choose between this kernel and the others, here and in chan_preferred and band_plan, look at stream_geom's geometry, on
// which their lines were drawn; what is launched in its place (stream_plan) is estimated to be the faster one, so they err to this side only.
static bool stream_extra(const FusedArgs &a, int dir) { return (dir == 0 ? a.res : a.ymask) != nullptr; }

// Blocks of a cluster, and of the grid, in stream_geom's geometry for this call; 0 where the kernel does not apply.
uint32_t stream_cluster(const FusedArgs &a, int dir, bool aligned, uint32_t &blocks)
{
  StreamGeom g;
  if (!stream_applies(a, dir, aligned) || !stream_geom(a.plan.dim0, a.plan.C, a.plan.N, dir, stream_extra(a, dir), g)) return 0u;
  blocks = g.units * g.cluster;
  return g.cluster;
}

bool stream_applies(const FusedArgs &a, int dir, bool aligned)
{
  StreamGeom g;
  return aligned && a.mode == MODE_FUSED && a.world <= 1 && stream_geom(a.plan.dim0, a.plan.C, a.plan.N, dir, stream_extra(a, dir), g);
}

// Where this kernel is taken (after the register-resident kernel): all rows that the tiled kernel does not serve, and of
// those it does serve (`tiled_ok`) the short ones and the medium ones of layers and channels that are not too large
// (tiled_takes; short of that line by the channel's size, as measured when the tiled kernel read every tile twice: of rows of
// 784 and 1024 floats it would have more now, see there).
constexpr uint32_t kStreamShortRow = 512, kStreamMediumRow = 600, kStreamLongRow = 1024;
// Layers of few channels leave the device to a few clusters whose threads walk hundreds of samples.  With rows that the
// tiled kernel serves it is the faster one there, forward / backward, here and there: [7663,4,412] 47 / 119 and 31 / 54,
// [5111,9,420] 54 / 102 and 43 / 77, but [4976,11,260] 43 / 76 and 43 / 78 (104 samples a thread), [295,122,588] 39 / 66
// and 42 / 77 (74).  For odd rows below that the plain kernel is, in the residual epilogue's forward pass only:
// [45953,8,21] 162 and 121, [17770,12,27] 94 and 72, [11845,12,73] 94 and 75, but [18431,12,37] 70 and 90 (192 samples),
// [129340,8,10] 224 and 330, [57124,7,32] 167 and 189.
constexpr uint32_t kStreamLongWalk = 112, kStreamFewBlocks = 48;
bool stream_preferred(const FusedArgs &a, int dir, bool aligned, bool tiled_ok)
{
  const uint32_t dim0 = a.plan.dim0;
  StreamGeom g;
  if (!stream_applies(a, dir, aligned) || !stream_geom(dim0, a.plan.C, a.plan.N, dir, stream_extra(a, dir), g)) return false;
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  const uint32_t walk = ceil_div_u32(g.rows, g.groups), blocks = g.units * g.cluster;
  if (tiled_ok && walk >= kStreamLongWalk) return false;
  if (!tiled_ok && extra && dir == 0 && dim0 > 16 && dim0 % 4 != 0 && blocks <= kStreamFewBlocks && walk >= 2 * kStreamLongWalk) return false;
  if (tiled_ok && tiled_takes(dim0, (uint64_t)dim0 * a.plan.C * a.plan.N, dir, extra)) return false;
  if (!tiled_ok || dim0 <= kStreamShortRow) return true;
  const uint64_t most = (extra ? 1u << 18 : dir == 1 ? 1u << 17 : 1u << 16) * (dim0 <= kStreamMediumRow ? 4ull : 1ull);
  return dim0 <= kStreamLongRow && (uint64_t)dim0 * a.plan.N <= most;
}

// ANODE_E_LAUNCH when the device refuses the cluster shape (the caller takes the next kernel that applies).
int launch_stream(FusedArgs &a, int dir, cudaStream_t stream)
{
  StreamGeom g;
  const bool masked = !stream_geom_of(a, dir, g);
  if (masked && !masked_geom_of(a, dir, g)) return ANODE_E_LAUNCH;
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  // dres may be stored before x is read again only where it is not x itself
  a.dres_early = a.dres && a.dres != a.x ? 1u : 0u;
  auto kernel = dir == 0 ? (extra ? bn_stream_kernel<0, true, false> : bn_stream_kernel<0, false, false>)
                         : (extra ? bn_stream_kernel<1, true, false> : bn_stream_kernel<1, false, false>);
  if (masked) kernel = dir == 0 ? (extra ? bn_stream_kernel<0, true, true> : bn_stream_kernel<0, false, true>)
                                : (extra ? bn_stream_kernel<1, true, true> : bn_stream_kernel<1, false, true>);
  return launch_clusters(kernel, a, g, g.units * g.cluster, g.threads, g.cluster, stream);
}

}  // namespace anode_b200

// ---- diagnostics: geometry of the streaming kernel for a shape (no GPU needed) -----------------
extern "C" int anode_gpu_batch_norm_stream_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  StreamGeom g{};
  const bool ok = stream_plan(dim0, dim1, dim2, dir, false, g);
  const uint32_t v[7] = {ok ? 1u : 0u, g.cb, g.units, g.cluster, g.rows, g.groups, g.threads};
  for (int i = 0; i < 7; ++i) out[i] = v[i];
  return ANODE_OK;
}

extern "C" int anode_gpu_batch_norm_stream_masked_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  StreamGeom g{};
  const bool ok = masked_plan(dim0, dim1, dim2, dir, residual != 0, g);
  const uint32_t v[7] = {ok ? 1u : 0u, g.cb, g.units, g.cluster, g.rows, g.groups, g.threads};
  for (int i = 0; i < 7; ++i) out[i] = ok || i == 0 ? v[i] : 0u;
  return ANODE_OK;
}
