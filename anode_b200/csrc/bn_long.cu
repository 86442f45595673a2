// Fused batch-norm (+activation, +residual) for small layers of long rows, e.g. [1, 3, 64, 64, 64] or [41, 6, 64, 64]: few channels,
// each too large for the registers of a few blocks.
//
// A thread-block CLUSTER of up to sixteen blocks owns one channel; its threads take the channel's 16-byte vectors in turn and walk
// them twice, as the streaming kernel (bn_stream.cu) does with runs of short rows:
//   1. statistics: kBatch 128-bit loads in flight per thread, shifted sums (or the backward sums) in registers, added over the block
//      in double precision; each block pushes its sums into every block of the cluster, one cluster barrier;
//   2. every block merges them in rank order and walks its vectors again: the last batch is still in registers, the others come from L2.
// RAG: rows whose length is no multiple of four floats, from the 16-byte boundary below a row's start to the one above its end; a
// vector's lanes outside the row are left out.
//
// What bounds it: the chain launch -> loads -> cluster barrier -> stores, and for larger channels the batches of a thread (a vector
// costs 0.23 us of a thread forward, 0.4 backward, ragged ones 1.7 times that, forward 2.1, for their place and lanes: with 27 M elements
// DRAM is at 0.46 and 0.49 of its peak and warps wait for loads, on ragged rows at 0.40 and 0.46, and they wait for instructions as
// well).  The tiled kernel, which these layers had, is launched cooperatively and agrees over the whole grid, some ten us a launch
// whatever the size.  Forward / backward, us, there and here: [4,4,42672] 12.9 / 12.4 and 6.0 / 6.7, [1,4,254072] 14.4 / 13.9 and
// 6.2 / 8.5, [227,8,1116] 16.5 / 14.8 and 7.6 / 10.3; ragged rows on the register-resident kernel, [8,217,2678] 18.5 / 29.8 and 12.7 / 16.1.
// Error against float64, relative, geometric mean, on the tiled kernel (398 passes) and here: mean 2.4e-8 and 2.2e-8, variance 4.6e-8 and
// 2.7e-8, dgamma (the one there with an older inv_std) 1.6e-7 and 8.6e-8, dbeta 1.2e-7 and 6.5e-8; on the register-resident one (219)
// 2.4e-8 and 2.3e-8, 2.8e-8 and 2.7e-8, 1.3e-7 and 8.2e-8, 9.9e-8 and 5.7e-8.
//
// Reference kernels this replaces: routines_gpu/batch_norm.cu:24-57, 125-163, 314-336 (forward), :181-206, 240-280,
// 354-376, 408-444, 476-515 (backward), flat_map.cu:172-194 (ReLU).
#include <math.h>

#include "bn_device.cuh"
#include "bn_host.h"

namespace anode_b200 {

constexpr uint32_t kLongThreads = 256, kLongCluster = 16;

template <int DIR, bool EXTRA, bool RAG>
__global__ void __launch_bounds__(kLongThreads, kLongBlocks) bn_long_kernel(const FusedArgs a, const LongGeom g)
{
  constexpr int kBatch = DIR == 0 && !EXTRA ? 8 : DIR == 1 && EXTRA ? 3 : 4;      // vectors in flight per thread and tensor
  __shared__ double2 part[kLongThreads / 32], rec[kLongCluster];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t csh = (uint32_t)__ffs((int)g.cluster) - 1u;
  const uint32_t c = blockIdx.x >> csh, rank = blockIdx.x & (g.cluster - 1u);
  const uint32_t dim0 = a.plan.dim0, rs = a.plan.C * dim0;
  // remote shared memory may only be written once its block runs (collected right before the first remote store)
  if (g.cluster > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t j0 = rank * kLongThreads + tid;
  const uint32_t cnt = j0 < g.total ? (g.total - j0 - 1) / g.stride + 1 : 0;
  const uint32_t row0 = j0 / g.per_row, col0 = j0 - row0 * g.per_row;
  const uint32_t at0 = row0 * rs + c * dim0;             // float offsets are below 2^32 (check_dims) wherever k < cnt
  const float slope = a.neg_slope;                       // activation: t * (t > 0 ? 1 : slope)
  const bool early = DIR == 1 && EXTRA && a.dres_early;  // dz is stored in the first walk and read back in the second
  const uint64_t keep = policy_keep(), drop = policy_drop();

  // the row at `at`, its vector `col`: the vector's offset, and the lanes that are the row's
  auto place = [&](uint32_t at, uint32_t col, uint32_t &lanes) {
    lanes = 15u;
    if (!RAG) return at + 4 * col;
    const uint32_t mis = at & 3u, past = dim0 + mis, v = 4 * col;
    lanes = v >= past ? 0u : (past - v >= 4 ? 15u : (1u << (past - v)) - 1u) & (col == 0 ? 15u << mis : 15u);
    return at - mis + v;
  };
  auto advance = [&](uint32_t &at, uint32_t &col) {
    at += g.step_rows * rs; col += g.step_col;
    if (col >= g.per_row) { col -= g.per_row; at += rs; }
  };
  // (of the vector in which the tensor ends, the last channel's, what lies inside is read)
  const bool tail = RAG && c + 1 == a.plan.C && (a.plan.N * rs & 3u);
  const uint32_t end = a.plan.N * rs - 4;
  auto load = [&](const float *p, uint32_t off, uint32_t lanes, uint64_t pol) {
    if (!tail || off <= end) return Pack<4>::load(p + off, pol);
    Pack<4> r = pack_fill<4>(0.f);
#pragma unroll
    for (int e = 0; e < 3; ++e) if (lanes >> e & 1u) r.v[e] = p[off + e];
    return r;
  };
  auto store = [&](const Pack<4> &o, float *p, uint32_t lanes, bool later) {      // later: the block reads it again
    if (!RAG || lanes == 15u) { if (later) o.put(p); else o.store_stream(p); return; }
#pragma unroll
    for (int e = 0; e < 4; ++e) if (lanes >> e & 1u) p[e] = o.v[e];
  };
  pdl_wait();
  pdl_trigger();

  const float gm = a.gamma ? a.gamma[c] : 1.0f;
  const float bt = (a.gamma && a.beta) ? a.beta[c] : 0.0f;
  float mean = 0.f, rstd = 0.f, scale = 0.f;
  if (DIR == 1) { mean = a.mean_in[c]; rstd = inv_std(a.var_in[c]); scale = gm * rstd; }

  // ---- first walk
  Pack<4> vx[kBatch], vd[DIR == 1 ? kBatch : 1];         // after the walk: the last batch (vd: its dz)
  float s[4] = {0.f, 0.f, 0.f, 0.f}, q[4] = {0.f, 0.f, 0.f, 0.f}, K = 0.f;
  uint32_t at = at0, col = col0, atb = at0, colb = col0, kb = 0, floats = 0;      // atb, colb, kb: where the last batch begins
  for (uint32_t k = 0; k < cnt; k += kBatch) {
    kb = k; atb = at; colb = col;
    Pack<4> vm[DIR == 1 && EXTRA ? kBatch : 1];
    uint32_t lanes[kBatch], off[DIR == 1 && EXTRA ? kBatch : 1];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      const uint32_t o = place(at, col, lanes[i]);
      if (k + i >= cnt) lanes[i] = 0u;
      if (DIR == 1 && EXTRA) off[i] = o;
      vx[i] = pack_fill<4>(0.f);
      if (DIR == 1) vd[i] = pack_fill<4>(0.f);
      if (lanes[i]) {
        vx[i] = load(a.x, o, lanes[i], keep);
        if (DIR == 1) vd[i] = load(a.dy, o, lanes[i], early ? drop : keep);
        if (DIR == 1 && EXTRA) vm[i] = load(a.ymask, o, lanes[i], early ? drop : keep);
      }
      advance(at, col);
    }
    // lanes that are not the channel's take a value that adds nothing
    auto others = [&](Pack<4> &v, uint32_t lanes, float f) {
      if (lanes != 15u) {
#pragma unroll
        for (int e = 0; e < 4; ++e) if (!(lanes >> e & 1u)) v.v[e] = f;
      }
    };
    if (DIR == 0) {
      if (k == 0) {
        // shift of the sums: the mean of the thread's first batch
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          others(vx[i], lanes[i], 0.f);
          t += (vx[i].v[0] + vx[i].v[1]) + (vx[i].v[2] + vx[i].v[3]);
          floats += (uint32_t)__popc(lanes[i]);
        }
        K = fabsf(t) < 1e36f && floats ? __fdividef(t, (float)floats) : 0.f;      // (an infinity or a NaN is no shift, the sums show it)
      } else {
#pragma unroll
        for (int i = 0; i < kBatch; ++i) floats += (uint32_t)__popc(lanes[i]);
      }
      // batch by batch, so that a long walk's sums are rounded once per batch
      float bs[4] = {0.f, 0.f, 0.f, 0.f}, bq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        others(vx[i], lanes[i], K);
#pragma unroll
        for (int e = 0; e < 4; ++e) { const float d = vx[i].v[e] - K; bs[e] += d; bq[e] = fmaf(d, d, bq[e]); }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) { s[e] += bs[e]; q[e] += bq[e]; }
    } else {
      float bs[4] = {0.f, 0.f, 0.f, 0.f}, bq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        others(vx[i], lanes[i], mean); others(vd[i], lanes[i], 0.f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d = vx[i].v[e] - mean;
          const float yb = EXTRA ? vm[i].v[e] : fmaf(d, scale, bt);
          vd[i].v[e] *= yb > 0.0f ? 1.0f : slope;        // dz = dy * act'(y)  (routines_gpu/flat_map.cu:191-192)
          bs[e] += vd[i].v[e]; bq[e] = fmaf(vd[i].v[e], d, bq[e]);
        }
        if (EXTRA && early && lanes[i]) store(vd[i], a.dres + off[i], lanes[i], true);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) { s[e] += bs[e]; q[e] += bq[e]; }
    }
  }

  // ---- the block's sums, of x and x^2 about zero (from the shifted ones, in double precision) or the backward sums
  double t1 = ((double)s[0] + (double)s[1]) + ((double)s[2] + (double)s[3]), t2 = ((double)q[0] + (double)q[1]) + ((double)q[2] + (double)q[3]);
  if (DIR == 0) {
    const double n = (double)floats, k = (double)K;
    t2 = fma(k, fma(n, k, 2.0 * t1), t2); t1 = fma(n, k, t1);
  }
  t1 = warp_sum_all(t1); t2 = warp_sum_all(t2);
  if (lane == 0) part[warp] = make_double2(t1, t2);
  __syncthreads();
  if (warp == 0) {
    const double2 p = lane < kLongThreads / 32 ? part[lane] : make_double2(0.0, 0.0);
    t1 = warp_sum_all(p.x); t2 = warp_sum_all(p.y);
  }
  if (g.cluster > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp == 0 && lane < g.cluster) st_cluster_d2(&rec[rank], lane, t1, t2);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    if (tid == 0) rec[0] = make_double2(t1, t2);
    __syncthreads();
  }

  // ---- merged in rank order by every thread; block 0 writes the channel's results
  t1 = 0.0; t2 = 0.0;
  for (uint32_t r = 0; r < g.cluster; ++r) { const double2 p = rec[r]; t1 += p.x; t2 += p.y; }
  float cB = 0.f, cC = 0.f;
  if (DIR == 0) {
    const double md = t1 * g.inv_count;
    mean = (float)md;
    const float vf = (float)(not_below_zero(t2 - t1 * md) * g.inv_count + (double)a.epsilon);      // biased, epsilon folded in (batch_norm.cu:160)
    scale = gm * inv_std(vf);
    if (rank == 0 && tid == 0) {
      a.mean[c] = mean; a.var[c] = vf;
      if (a.run_mean) { const float o = a.run_mean[c]; a.run_mean[c] = o + a.avg_rate * (mean - o); }
      if (a.run_var) { const float o = a.run_var[c]; a.run_var[c] = o + a.avg_rate * (vf - o); }
    }
  } else {
    const double rs2 = (double)rstd * t2;                // sum(dz * xhat)
    const double A = (double)gm * (double)rstd;
    cB = (float)(-A * (double)rstd * rs2 * g.inv_count);
    cC = (float)(-A * t1 * g.inv_count);
    if (rank == 0 && tid == 0) {
      if (a.dbeta) a.dbeta[c] = (float)t1;
      if (a.dgamma) a.dgamma[c] = (float)rs2;
    }
  }

  // ---- second walk, the batch in registers first
  at = atb; col = colb;
  for (uint32_t k = kb, left = cnt; left > 0;) {
    uint32_t off[kBatch], lanes[kBatch];
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      off[i] = place(at, col, lanes[i]);
      if (k + i >= cnt) lanes[i] = 0u;
      advance(at, col);
    }
    if (left != cnt) {
      const float *second = early ? a.dres : a.dy;
      Pack<4> vm[DIR == 1 && EXTRA ? kBatch : 1];
#pragma unroll
      for (int i = 0; i < kBatch; ++i)
        if (lanes[i]) {
          vx[i] = load(a.x, off[i], lanes[i], drop);
          if (DIR == 1) vd[i] = load(second, off[i], lanes[i], drop);
          if (DIR == 1 && EXTRA && !early) vm[i] = load(a.ymask, off[i], lanes[i], drop);
        }
      if (DIR == 1 && !early) {
#pragma unroll
        for (int i = 0; i < kBatch; ++i)
          if (lanes[i]) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float yb = EXTRA ? vm[i].v[e] : fmaf(vx[i].v[e] - mean, scale, bt);
              vd[i].v[e] *= yb > 0.0f ? 1.0f : slope;
            }
          }
      }
    }
    Pack<4> ve[DIR == 0 && EXTRA ? kBatch : 1];
    if (DIR == 0 && EXTRA) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) if (lanes[i]) ve[i] = load(a.res, off[i], lanes[i], drop);
    }
    Pack<4> old[DIR == 1 ? kBatch : 1];
    if (DIR == 1 && a.accumulate) {
#pragma unroll
      for (int i = 0; i < kBatch; ++i) if (lanes[i]) old[i] = load(a.out, off[i], lanes[i], drop);
    }
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (lanes[i]) {
        Pack<4> o;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (DIR == 0) {
            float yb = fmaf(vx[i].v[e] - mean, scale, bt);
            if (EXTRA) yb += ve[i].v[e];
            o.v[e] = yb * (yb > 0.0f ? 1.0f : slope);
          } else {
            const float dx = fmaf(scale, vd[i].v[e], fmaf(cB, vx[i].v[e] - mean, cC));
            o.v[e] = a.accumulate ? old[i].v[e] + dx : dx;
          }
        }
        store(o, a.out + off[i], lanes[i], false);
        if (DIR == 1 && EXTRA && !early && a.dres) store(vd[i], a.dres + off[i], lanes[i], false);
      }
    // the batch that was held, then the others from the first on
    if (left == cnt) { if (kb == 0) break; left = kb; k = 0; at = at0; col = col0; }
    else { if (left <= kBatch) break; left -= kBatch; k += kBatch; }
  }
}

// ---- host side -------------------------------------------------------------------------------

// The cluster of the least estimated time, as for the streaming kernel's masked form (masked_plan); the figures are fitted to 155 shapes
// of 0.3 to 23 M elements in four directions, from which the estimate is off by ten per cent on average.  In the geometry's cost, which is
// held against other kernels' times, ragged vectors take 1.7 times as long, forward 2.1 (fitted to 782 launches from memory and as many
// from L2, from which it is off by nine per cent; without those factors, by 12 and 13 on ragged rows, and 20 too low).
bool long_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, LongGeom &g)
{
  if (dim0 < 16 || C > 0xfffffu) return false;
  g.per_row = dim0 % 4 ? (uint32_t)((dim0 + 6ull) / 4) : dim0 / 4;
  const uint64_t total = (uint64_t)g.per_row * N;
  if (total > 0x3fffffffu) return false;
  g.total = (uint32_t)total;
  const uint32_t wave = kLongBlocks * sm_count();
  const double bytes = 4.0 * dim0 * C * N * (dir == 0 ? (extra ? 3 : 2) : extra ? 5 : 3);
  const double each = dir == 0 ? (extra ? 0.32 : 0.225) : 0.41;      // us per vector of a thread
  const double ragged = dim0 % 4 == 0 ? 1.0 : dir == 0 && !extra ? 2.1 : 1.7;
  double best = 0;
  for (uint32_t cl = 1; cl <= kLongCluster; cl *= 2) {
    const uint64_t blocks = (uint64_t)C * cl, places = cl == 16 ? wave * 25 / 32 : cl == 8 ? wave * 17 / 20 : cl == 4 ? wave * 15 / 16 : wave;
    const double waves = (double)((blocks + places - 1) / places), resident = (double)(blocks < places ? blocks : places);
    const uint64_t walk = (total + cl * kLongThreads - 1) / (cl * kLongThreads);
    const double over = 4.0 * dim0 * N * (dir == 1 ? 2 : 1) / cl * resident / 77e6 - 1;
    const double again = (dir == 1 ? 0.5 : 0.17) * (over < 0 ? 0 : over > 1 ? 1 : over), lanes = resident / wave;
    const double moved = bytes * (1 + again) / 5.15e6 * (0.9 + 0.1 / lanes), chain = waves * walk * each;
    const double fixed = 0.5 + waves * (2.4 + 0.024 * cl), cost = fixed + pow(pow(moved, 2.5) + pow(chain, 2.5), 0.4);
    if (best == 0 || cost < best) {
      best = cost; g.cluster = cl;
      g.cost = (float)(fixed + pow(pow(moved, 2.5) + pow(chain * ragged, 2.5), 0.4));
    }
  }
  g.stride = g.cluster * kLongThreads;
  g.step_rows = g.stride / g.per_row; g.step_col = g.stride - g.step_rows * g.per_row;
  g.inv_count = 1.0 / ((double)dim0 * (double)N);
  return true;
}

// ANODE_E_LAUNCH when the device refuses the cluster shape (the caller takes the next kernel that applies).
int launch_long(FusedArgs &a, const LongGeom &g, int dir, cudaStream_t stream)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr, rag = a.plan.dim0 % 4 != 0;
  // dres may be stored before x is read again only where it is not x itself
  a.dres_early = a.dres && a.dres != a.x ? 1u : 0u;
  auto kernel = dir == 0 ? (extra ? (rag ? bn_long_kernel<0, true, true> : bn_long_kernel<0, true, false>)
                                  : (rag ? bn_long_kernel<0, false, true> : bn_long_kernel<0, false, false>))
                         : (extra ? (rag ? bn_long_kernel<1, true, true> : bn_long_kernel<1, true, false>)
                                  : (rag ? bn_long_kernel<1, false, true> : bn_long_kernel<1, false, false>));
  return launch_clusters(kernel, a, g, a.plan.C * g.cluster, kLongThreads, g.cluster, stream);
}

}  // namespace anode_b200

// ---- diagnostics: geometry for a shape (no GPU needed) -----------------------------------------
extern "C" int anode_gpu_batch_norm_long_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  LongGeom g{};
  const bool ok = long_plan(dim0, dim1, dim2, dir, residual != 0, g);
  const uint32_t v[7] = {ok ? 1u : 0u, g.cluster, g.stride, g.per_row, g.total, g.step_rows, g.step_col};
  for (int i = 0; i < 7; ++i) out[i] = ok || i == 0 ? v[i] : 0u;
  return ANODE_OK;
}
