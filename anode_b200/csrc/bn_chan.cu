// Fused batch-norm (+activation, +residual) for channels that fit the registers of a few thread blocks: small layers,
// where a kernel's latency is its time, and any row length or alignment.
//
// A channel belongs to a TEAM of threads: one warp, one block, or a thread-block cluster of up to eight blocks.  Every
// thread loads its elements of the channel into registers, all loads in flight at once, and the tensor is read once:
//   1. warp moments (two passes over registers: mean, then squares about it), or the warp's backward sums;
//   2. each warp pushes its record into the shared memory of every block of the cluster (one remote store per lane)
//      and the cluster barrier follows: the only synchronisation of the kernel, and none at all in a one-warp team;
//   3. every warp merges all records in a fixed order in double precision (bit-identical coefficients everywhere);
//   4. y (or dx) is computed from the registers and stored.
//
// What bounds it: on small layers the chain launch -> load -> barrier -> store, 3 - 4 us; the plain kernel's grid-wide
// partials, counters and flags took 6 - 15 us for the same layers (figures at chan_preferred).  Elements a team does not own to the full are predicated, so the split is by
// the flat index inside the channel (row-major over samples): odd rows cost an add and a compare per element, no division.
//
// Reference kernels this replaces: routines_gpu/batch_norm.cu:24-57, 125-163, 314-336 (forward), :181-206, 240-280,
// 354-376, 408-444, 476-515 (backward), flat_map.cu:172-194 (ReLU).
#include <atomic>

#include "bn_device.cuh"
#include "bn_host.h"

namespace anode_b200 {

constexpr uint32_t kChanThreads = 512;       // most threads of a block
constexpr uint32_t kChanCluster = 8;         // most blocks of a team (the portable cluster size)
constexpr uint32_t kChanWarpTeams = 4;       // one-warp teams per block

// Threads that two blocks of an SM are compiled for: 64 registers each at most, or for teams of a few floats a thread 48 or 56, where blocks
// that do not divide an SM's 1024 threads would leave a second wave (chan_dense).  Us with 64 and so, forward, [225,56,80] 6.4 and 4.3,
// [3,239,1451] 6.0 and 4.3, [6,278,354] 5.5 and 3.8; but with one wave either way backward [451,21,48] 3.6 and 4.3, [108,84,29] 3.6 and 4.3.
constexpr uint32_t chan_bound(int floats, bool dense) { return !dense ? kChanThreads : floats == 4 ? 640u : 576u; }

struct ChanGeom {
  uint32_t vec, floats;      // floats per load (4 or 1) and per thread (the template's F)
  uint32_t threads, cluster; // team = cluster * threads; threads == 32: one-warp teams, kChanWarpTeams to a block
  uint32_t d0v, total;       // vectors per row and per channel
  uint32_t team;             // threads of a team = distance between a thread's vectors
  uint32_t step_off, step_col, wrap;   // a step of `team` vectors: floats forward, columns forward, floats added when the column wraps
  double inv_count;
};

// float4 into the shared memory of block `rank` of the cluster, at the address `p` has in this block
__device__ __forceinline__ void st_cluster_f4(void *p, uint32_t rank, float4 v)
{
  const uint32_t local = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(remote), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// F: floats a thread holds per tensor; ADDS: the output is added to (the forms without it that do so, too: kLate)
template <int DIR, int VEC, int F, bool EXTRA, bool DENSE, bool ADDS>
__global__ void __launch_bounds__(chan_bound(F, DENSE), 2) bn_chan_kernel(const FusedArgs a, const ChanGeom g)
{
  constexpr int E = F / VEC;
  __shared__ float4 rec[kChanCluster * kChanThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool solo = g.threads == 32;                      // one-warp teams
  const uint32_t csh = (uint32_t)__ffs((int)g.cluster) - 1u;
  const uint32_t c = solo ? blockIdx.x * kChanWarpTeams + warp : blockIdx.x >> csh;
  const uint32_t rank = solo ? 0u : blockIdx.x & (g.cluster - 1u);
  const uint32_t C = a.plan.C;
  // remote shared memory may only be written once its block runs: announce this block now, collect the others' word
  // right before the first remote store
  if (g.cluster > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
  const uint32_t t = solo ? lane : rank * g.threads + tid;
  const uint32_t row = t / g.d0v;
  const uint32_t col0 = t - row * g.d0v;
  const uint32_t off0 = row * (C * a.plan.dim0) + c * a.plan.dim0 + col0 * VEC;      // below 2^32 (check_dims)
  const uint32_t cnt = t < g.total ? (g.total - t - 1) / g.team + 1 : 0;          // this thread's vectors, <= E
  pdl_wait();
  pdl_trigger();
  if (c >= C) return;                                     // (one-warp teams only: the last block may be ragged)

  const float gm = a.gamma ? a.gamma[c] : 1.0f;
  const float bt = (a.gamma && a.beta) ? a.beta[c] : 0.0f;
  const bool owner = rank == 0 && (solo || warp == 0) && lane == 0;
  float mean = 0.f, scale = 0.f, rstd = 0.f, rm = 0.f, rv = 0.f;
  if (DIR == 1) { mean = a.mean_in[c]; rstd = inv_std(a.var_in[c]); scale = gm * rstd; }
  else if (owner) { if (a.run_mean) rm = a.run_mean[c]; if (a.run_var) rv = a.run_var[c]; }
  const float slope = a.neg_slope;      // activation: t * (t > 0 ? 1 : slope)

  // Accumulating writes: what they add to is loaded with the inputs where a thread has four floats of it, else brought to L2 with them and
  // loaded ahead of the first write ([100,300,7,7] 14.6 us where each load waited for the store before it, and 8.9 so; [2,2048,14,108] 22.7
  // and 19.1).  In forms of their own: assigning calls have nothing of it to check ([16,899,6,6] 3.9 us and 3.8, [108,84,29] 4.2 and 3.7).
  // Sixteen single floats more would spill, so they are brought to L2 only, and the residual epilogue has three tensors already: there each
  // load waits (kLate; in forms of their own those are 4 per cent slower, [184,1311,8,8] 79 and 83).
  constexpr bool kEarly = ADDS && F == 4, kLate = DIR == 1 && (EXTRA || (VEC == 1 && F == 16));
  static_assert(!ADDS || (DIR == 1 && !kLate), "no such form");
  Pack<VEC> vx[E], ve[(DIR == 1 || EXTRA) ? E : 1];       // ve: dy, later dz (backward) or the residual (forward)
  Pack<VEC> old[ADDS ? E : 1];
  {
    uint32_t off = off0, col = col0;
    Pack<VEC> vm[(DIR == 1 && EXTRA) ? E : 1];            // the saved output, which carries the mask
#pragma unroll
    for (int k = 0; k < E; ++k) {
      vx[k] = pack_fill<VEC>(0.f);
      if (DIR == 1 || EXTRA) ve[k] = pack_fill<VEC>(0.f);
      if (DIR == 1 && EXTRA) vm[k] = pack_fill<VEC>(0.f);
      if (k < cnt) {
        vx[k] = Pack<VEC>::load(a.x + off);
        if (DIR == 1) ve[k] = Pack<VEC>::load(a.dy + off);
        if (kEarly) old[k] = Pack<VEC>::load(a.out + off);
        else if (ADDS || (kLate && !EXTRA && a.accumulate)) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.out + off));
        if (DIR == 0 && EXTRA) ve[k] = Pack<VEC>::load(a.res + off);
        if (DIR == 1 && EXTRA) vm[k] = Pack<VEC>::load(a.ymask + off);
      }
      off += g.step_off; col += g.step_col;
      if (col >= g.d0v) { col -= g.d0v; off += g.wrap; }
    }
    if (DIR == 1) {
      // x becomes x - mean, dy becomes dz = dy * act'(y)  (routines_gpu/flat_map.cu:191-192)
#pragma unroll
      for (int k = 0; k < E; ++k)
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float d = vx[k].v[i] - mean;
          const float yb = EXTRA ? vm[k].v[i] : fmaf(d, scale, bt);
          vx[k].v[i] = k < cnt ? d : 0.f;
          ve[k].v[i] *= yb > 0.0f ? 1.0f : slope;
        }
    }
  }

  // ---- the warp's record
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  if (DIR == 0) {
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < E; ++k)
#pragma unroll
      for (int i = 0; i < VEC; ++i) s += vx[k].v[i];
    s = warp_sum_all(s);
    const float n = (float)(__reduce_add_sync(0xffffffffu, cnt) * VEC);
    const float m = n > 0.f ? __fdividef(s, n) : 0.f;
    float q = 0.f, dev = 0.f;      // dev: what the division and the sum's rounding left in the mean
#pragma unroll
    for (int k = 0; k < E; ++k)
      if (k < cnt) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) { const float d = vx[k].v[i] - m; dev += d; q = fmaf(d, d, q); }
      }
    q = warp_sum_all(q); dev = warp_sum_all(dev);
    // (a sum that holds an infinity is one, whatever is left beside it)
    r = make_float4(n, m, q, fabsf(m) <= 3.402823466e38f ? dev : 0.f);
  } else {
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int k = 0; k < E; ++k)
#pragma unroll
      for (int i = 0; i < VEC; ++i) { s1 += ve[k].v[i]; s2 = fmaf(ve[k].v[i], vx[k].v[i], s2); }
    r.x = warp_sum_all(s1); r.y = warp_sum_all(s2);
  }

  // ---- all records of the team, merged by every warp
  double t0 = 0.0, t1 = 0.0;
  auto add = [&](const float4 &p) {
    if (DIR == 0) {
      // sum and sum of squares about zero: sum(x) = n*m + dev, sum(x^2) = q + m*(n*m + 2*dev)
      const double n = (double)p.x, m = (double)p.y, e = (double)p.w;
      t0 += fma(n, m, e); t1 += fma(m, fma(n, m, 2.0 * e), (double)p.z);
    } else { t0 += (double)p.x; t1 += (double)p.y; }
  };
  if (solo) {
    add(r);
  } else {
    const uint32_t warps = g.threads >> 5;
    if (g.cluster > 1) {
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      if (lane < g.cluster) st_cluster_f4(&rec[rank * warps + warp], lane, r);
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
      if (lane == 0) rec[warp] = r;
      __syncthreads();
    }
    for (uint32_t i = lane; i < warps * g.cluster; i += 32) add(rec[i]);
    t0 = warp_sum_all(t0); t1 = warp_sum_all(t1);
  }

  // ---- coefficients and per-channel results
  float cB = 0.f, cC = 0.f;
  if (DIR == 0) {
    const double md = t0 * g.inv_count;
    mean = (float)md;
    const float var = (float)(not_below_zero(t1 - t0 * md) * g.inv_count + (double)a.epsilon);      // biased, epsilon folded in (batch_norm.cu:160)
    scale = gm * inv_std(var);
    if (owner) {
      a.mean[c] = mean; a.var[c] = var;
      if (a.run_mean) a.run_mean[c] = rm + a.avg_rate * (mean - rm);
      if (a.run_var) a.run_var[c] = rv + a.avg_rate * (var - rv);
    }
  } else {
    const double rs2 = (double)rstd * t1;                 // sum(dz * xhat)
    const double A = (double)gm * (double)rstd;
    cB = (float)(-A * (double)rstd * rs2 * g.inv_count);
    cC = (float)(-A * t0 * g.inv_count);
    if (owner) {
      if (a.dbeta) a.dbeta[c] = (float)t0;
      if (a.dgamma) a.dgamma[c] = (float)rs2;
    }
  }

  // ---- apply
  uint32_t off = off0, col = col0;
  if (ADDS && !kEarly) {
    uint32_t at = off0, to = col0;
#pragma unroll
    for (int k = 0; k < E; ++k) {
      if (k < cnt) old[k] = Pack<VEC>::load(a.out + at);
      at += g.step_off; to += g.step_col;
      if (to >= g.d0v) { to -= g.d0v; at += g.wrap; }
    }
  }
#pragma unroll
  for (int k = 0; k < E; ++k) {
    if (k < cnt) {
      Pack<VEC> o;
      if (kLate && a.accumulate) o = Pack<VEC>::load(a.out + off);
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        if (DIR == 0) {
          float yb = fmaf(vx[k].v[i] - mean, scale, bt);
          if (EXTRA) yb += ve[k].v[i];
          o.v[i] = yb * (yb > 0.0f ? 1.0f : slope);
        } else {
          const float dx = fmaf(scale, ve[k].v[i], fmaf(cB, vx[k].v[i], cC));
          o.v[i] = ADDS ? old[ADDS ? k : 0].v[i] + dx : kLate && a.accumulate ? o.v[i] + dx : dx;
        }
      }
      o.put(a.out + off);
      if (DIR == 1 && EXTRA && a.dres) ve[k].put(a.dres + off);
    }
    off += g.step_off; col += g.step_col;
    if (col >= g.d0v) { col -= g.d0v; off += g.wrap; }
  }
}

// ---- host side -------------------------------------------------------------------------------

typedef void (*ChanKernel)(const FusedArgs, const ChanGeom);

template <int DIR, bool EXTRA, bool ADDS, int VEC>
static ChanKernel chan_kernel_of(uint32_t f, bool dense)
{
  if (f == 4) return dense ? bn_chan_kernel<DIR, VEC, 4, EXTRA, true, ADDS> : bn_chan_kernel<DIR, VEC, 4, EXTRA, false, ADDS>;
  if (f == 8) return dense ? bn_chan_kernel<DIR, VEC, 8, EXTRA, true, ADDS> : bn_chan_kernel<DIR, VEC, 8, EXTRA, false, ADDS>;
  if (f == 16) return bn_chan_kernel<DIR, VEC, 16, EXTRA, false, ADDS && VEC == 4>;
  if constexpr (DIR == 0 && !EXTRA) return bn_chan_kernel<DIR, VEC, 32, EXTRA, false, ADDS>;
  return nullptr;
}
template <int DIR, bool EXTRA, bool ADDS = false>
static ChanKernel chan_kernel_of(const ChanGeom &g, bool dense)
{
  return g.vec == 4 ? chan_kernel_of<DIR, EXTRA, ADDS, 4>(g.floats, dense) : chan_kernel_of<DIR, EXTRA, ADDS, 1>(g.floats, dense);
}
static ChanKernel chan_kernel_of(const ChanGeom &g, int dir, bool extra, bool adds, bool dense)
{
  if (dir == 0) return extra ? chan_kernel_of<0, true>(g, dense) : chan_kernel_of<0, false>(g, dense);
  return extra ? chan_kernel_of<1, true>(g, dense) : adds ? chan_kernel_of<1, false, true>(g, dense) : chan_kernel_of<1, false>(g, dense);
}

// Blocks of a form that an SM holds, 0 where the device does not say: asked for once per form and block size.  The register counts are the
// compiler's: the backward form of four floats in 16-byte loads has 56 without the bound, not 64, and of 48 registers an SM holds 40 warps, not 42.
static uint32_t chan_resident(const ChanGeom &g, int dir, bool extra, bool adds, bool dense, uint32_t threads)
{
  static std::atomic<uint8_t> kept[2][2][2][2][2][2][kChanThreads / 32 + 1];      // one more than the answer
  std::atomic<uint8_t> &k = kept[dir][extra][adds][g.vec == 4][g.floats == 8][dense][threads / 32];
  uint8_t n = k.load(std::memory_order_relaxed);
  if (!n) {
    int blocks = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, chan_kernel_of(g, dir, extra, adds, dense), (int)threads, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    k.store(n = (uint8_t)(blocks + 1), std::memory_order_relaxed);
  }
  return n - 1u;
}

// Whether the grid is one wave of blocks in the form of fewer registers, and more than one in the other ([1265,36,9], 36 clusters of eight:
// forward 6.4 and 4.7 us, residual forward 6.9 and 5.1; a twentieth more blocks than fit gain, too, [2,1938,10,14] forward 4.9 and 4.6).  Of 48
// registers in the place of 56, with one wave either way, backward [16,899,6,6] takes 4.1 and 3.9, [10,912,8,8] 4.0 and 3.9; but residual
// backward [94,224,4,6] 4.8 and 4.9, [136,469,2,4], from L2, 3.4 and 3.5: there as if the ordinary form had 64.
static bool chan_dense(const ChanGeom &g, int dir, bool extra, bool adds, uint32_t blocks, uint32_t threads)
{
  if (g.floats > 8 || blocks < 128) return false;      // (a wave is more than that)
  // (the SMs of a cluster lie together: clusters of four fill 94 per cent of the places, of eight 90: 256 blocks fit where
  // 296 would, 288 do not)
  auto places = [&](bool dense) {
    uint32_t n = chan_resident(g, dir, extra, adds, dense, threads);
    if (!dense && dir == 1 && extra && n > 1024 / threads) n = 1024 / threads;
    n *= sm_count();
    return g.cluster == 8 ? n * 9 / 10 : g.cluster == 4 ? n * 15 / 16 : n;
  };
  const uint32_t ordinary = places(false);
  return ordinary && blocks > ordinary && blocks <= places(true) * 21 / 20;
}

// blocks of the grid and threads of a block
static void chan_grid(const ChanGeom &g, uint32_t C, uint32_t &blocks, uint32_t &threads)
{
  const bool solo = g.threads == 32;
  blocks = solo ? ceil_div_u32(C, kChanWarpTeams) : C * g.cluster;
  threads = solo ? 32 * kChanWarpTeams : g.threads;
}

static bool chan_geom(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, bool aligned, ChanGeom &g)
{
  g.vec = aligned && dim0 % 4 == 0 ? 4u : 1u;
  const uint64_t total = (uint64_t)(dim0 / g.vec) * N;
  const uint32_t fmax = dir == 0 && !extra ? 32u : 16u;
  if (total > (uint64_t)kChanThreads * kChanCluster * (fmax / g.vec)) return false;
  g.d0v = dim0 / g.vec; g.total = (uint32_t)total;
  // floats per thread: as few as leave the whole problem on the device at once (about 1024 threads per SM)
  uint32_t f = 4;
  const uint32_t most = sm_count() * 1024;
  while (f < fmax && ((uint64_t)C * total * g.vec > (uint64_t)f * most ||
                      total > (uint64_t)kChanThreads * kChanCluster * (f / g.vec))) f *= 2;
  const uint32_t e = f / g.vec;
  const uint32_t need = (uint32_t)((total + e - 1) / e);             // threads of the team
  g.floats = f; g.cluster = 1;
  if (need <= 32) {
    g.threads = 32;
  } else {
    while (need > g.cluster * kChanThreads) g.cluster *= 2;
    g.threads = (ceil_div_u32(need, g.cluster) + 31) / 32 * 32;
  }
  g.team = g.threads * g.cluster;
  const uint32_t drow = g.team / g.d0v;
  g.step_col = g.team - drow * g.d0v;
  g.step_off = drow * (C * dim0) + g.step_col * g.vec;
  g.wrap = C * dim0 - dim0;
  g.inv_count = 1.0 / ((double)dim0 * (double)N);
  return true;
}

bool chan_applies(const FusedArgs &a, int dir, bool aligned)
{
  ChanGeom g;
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  return a.mode == MODE_FUSED && a.world <= 1 && chan_geom(a.plan.dim0, a.plan.C, a.plan.N, dir, extra, aligned, g);
}

// Where this kernel is taken: wherever a team can hold the channel, except on large layers where the team would be of
// more than half the largest size (its load, exchange and store then follow one another on most of the device) and
// where the elements would be fetched one by one although aligned runs of several channels, or long ragged rows, can be
// had (the scalar walk costs some 22 instructions per element).
// Forward + backward at the places of other kernels, there and here: [2,512,7,7] 11.5 -> 4.5 us, [32,64,28,28] 20.7 ->
// 9.8, [1,53,39,25] 17.9 -> 5.2, [1,260,128,128] 34.0 -> 16.7, [1,1240,45,30] 60.5 -> 13.8, [40,2048,146,5] 630 -> 413.
// The other way round, us here and there: streaming kernel, forward [512,1024,14,14] 213 and 185, backward
// [256,1024,14,14] 164 and 147, residual epilogue 156 / 222 and 137 / 209; [64,2048,7,7] 19.0 / 25.5 and 13.4 / 20.2,
// but [300,100,7,7] 5.9 / 8.6 and 6.7 / 8.3.  Tiled kernel, forward [128,512,28,28] 105 and 87, [39,255,45,45] 62 and
// 44, but [349,255,15,15] 64 and 68, [45,33,45,45] 12.9 and 15.5.
// Elements from which on the others are asked (rows without aligned runs of several channels, residual backward, on the
// tiled kernel: [26,551,431], 6.2 M, 57 and 47; [15,528,631], 5.0 M, 39 and 41).  Scalar rows with such runs go earlier where
// the teams take more than one wave of blocks, so that their load, exchange and store come twice: backward passes and the
// residual epilogue, us here and on the streaming kernel: residual backward [103,304,53] 15.2 and 8.8, residual forward
// [115,704,29] 11.8 and 7.4, backward [230,384,31] 13.7 and 8.8; but one wave, backward [19,728,145] 8.0 and 9.4, few
// samples, [15,1516,130] 10.8 and 12.5, clusters of sixteen, [336,212,29] 8.7 and 12.9.  With 20 to 31 samples a block of the
// streaming kernel has few rows to stream, and only grids of one wave without clusters of four gain: backward / residual forward
// [31,320,222] 14.2 / 14.7 and 10.8 / 9.4, [28,15964,5] 17.7 / 19.3 and 12.2 / 10.8, [27,1376,67] 13.6 / 14.0 and 11.6 / 10.4, but
// [31,6844,14], 685 blocks, 13.9 / 15.4 and 15.8 / 15.8, [27,5376,17], clusters of four, 12.9 / 14.1 and 15.8 / 14.7.  The residual
// backward, three tensors a thread, stalls in these teams at any number of waves: from 20 samples and a million elements it goes,
// [30,948,39], 1.1 M, 13.4 and 8.7, [81,680,35] 15.9 and 11.7, [28,340,218] 26.1 and 12.5, [31,6844,14] 27.1 and 19.2, but
// [20,848,43], 0.7 M, 6.5 and 6.4, [181,168,21], 0.6 M, 7.1 and 7.9; and units of 52 or 92 channels, which a block of few samples folds one by
// one, stay here in small layers and with fewer than 26 samples: [25,3720,11] 11.1 and 14.3, [31,3708,11] 13.2 and 15.1, [24,10100,11] 25.8 and 29.5,
// [21,5652,19] 22.4 and 23.1, but [28,6520,11] 20.8 and 19.4, [29,5156,19] 28.3 and 18.4.  (Those were all that lost by it of 280 residual
// backward passes of 1 - 3 M elements and 18 to 400 samples.)  Rows of 1 - 3 floats, which the
// threads fetch from far apart, on the shared-memory kernel: [1024,512,3] residual backward 25.8 and 18.5, [1540,632,2]
// backward 24.4 and 18.7, [1457,828,1] residual forward 23.6 and 20.6.
// Backward passes and the residual epilogue of large layers of medium and long aligned rows go to the tiled kernel although a
// team holds the channel, unless a channel is but a tile or two there.  Us here and there: backward [8,1024,56,56] 74 and 59,
// [16,512,56,56] 82 and 59, [35,512,28,28] 42 and 36, but [64,1024,18,18] 69 and 71, [1,2048,100,100] 51 and 54; residual
// [16,512,56,56] 80 / 109 and 62 / 96, [8,1024,56,56] 68 / 100 and 61 / 98, but [2,512,128,128] 41 / 61 and 44 / 65,
// [25,1024,28,28] 51 / 76 and 57 / 80.  (Forward passes: [64,512,28,28] 52 and 52, [25,1024,28,28] 36 and 47.)
// Nor below rows of 480 floats: 1024 channels of 31 K floats, backward, residual forward and backward, here and there, rows of
// 324 86 / 78 / 120 and 107 / 91 / 137, 400 84 / 77 / 117 and 95 / 84 / 122, but 484 85 / 78 / 118 and 88 / 81 / 118, 676
// 85 / 77 / 117 and 77 / 77 / 117, and of 25 K floats 484 77 / 70 / 105 and 68 / 63 / 96.
constexpr uint32_t kChanTiledRow = 480;
constexpr uint64_t kChanTiled = 16u << 20, kChanTiledExtra = 18u << 20, kChanTiledChannel = 24u << 10;
// Aligned rows below 320 floats go to the band kernel (the streaming kernel's form for large layers) from these sizes on.  Us here
// and there, forward: [80,1024,14,14] 16 M 29.3 and 31.3, [100,1024,16,16] 26 M 46.7 and 47.8, [100,1000,10,30] 30 M 54.6 and 52.1,
// [180,1024,14,14] 36 M 68 and 58, [256,1024,14,14] 99 and 81; backward: [50,2048,12,12] 15 M 37.2 and 35.0, [100,1024,14,14] 20 M 55 and 49,
// [256,1024,14,14] 164 and 106; residual forward, 15 M 32.1 and 34.7, 16 M 40 and 36, 20 M 52 and 46; residual backward 15 M 53.7 and 55.7, 20 M 79
// and 74.  (The last three lines lie higher than today's times ask for.)
constexpr uint32_t kChanBandRow = 320;
constexpr uint64_t kChanBand[2][2] = {{28000000, 18000000}, {18000000, 18000000}};      // [direction][residual]
constexpr uint64_t kChanLarge = 8u << 20, kChanLargeScalar = 3u << 20, kChanLargeExtra = 5u << 20;
constexpr uint64_t kChanWaves = 1500000, kChanShortest = 1200000, kChanShortestExtra = 1000000;
constexpr uint32_t kChanFewSamples = 32, kChanFewestSamples = 20;
constexpr uint32_t kChanLongRow = 300, kChanUnit = 32, kChanWideSamples = 26;
bool chan_preferred(const FusedArgs &a, int dir, bool aligned, bool tiled_ok)
{
  ChanGeom g;
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  if (a.mode != MODE_FUSED || a.world > 1) return false;
  if (!chan_geom(a.plan.dim0, a.plan.C, a.plan.N, dir, extra, aligned, g)) return false;
  const uint64_t channel = (uint64_t)a.plan.dim0 * a.plan.N, elements = channel * a.plan.C;
  const uint32_t most = dir == 0 && !extra ? 32u : 16u;
  BandGeom band;
  if (g.vec == 4) {
    if (tiled_ok && (dir == 1 || extra) && a.plan.dim0 >= kChanTiledRow && channel >= kChanTiledChannel &&
        elements >= (extra ? kChanTiledExtra : kChanTiled) && tiled_takes(a.plan.dim0, elements, dir, extra)) return false;
    if (a.plan.dim0 < kChanBandRow && elements >= kChanBand[dir][extra] && band_geom_of(a, dir, band) &&
        stream_preferred(a, dir, aligned, tiled_ok)) return false;
    if (elements < kChanLarge || channel <= (uint64_t)kChanThreads * kChanCluster * most / 2) return true;
    return !stream_preferred(a, dir, aligned, tiled_ok) &&
           !(tiled_ok && ((dir == 0 && !extra) || tiled_takes(a.plan.dim0, elements, dir, extra)));
  }
  if (elements < kChanLargeScalar) {
    const bool extra_bwd = extra && dir == 1 && a.plan.dim0 >= 4;
    if ((dir == 0 && !extra) || elements < (extra_bwd ? kChanShortestExtra : kChanShortest)) return true;
    if (a.plan.dim0 < 4) {
      const uint32_t blocks = segres_blocks(a, dir, aligned);
      return blocks == 0 || blocks > 2 * sm_count();
    }
    const uint64_t places = (uint64_t)sm_count() * (2 * kChanThreads / g.threads);
    const bool waves = elements >= kChanWaves && a.plan.N >= kChanFewSamples && (uint64_t)a.plan.C * g.cluster > places;
    uint32_t blocks = 0;
    const uint32_t cluster = stream_cluster(a, dir, aligned, blocks);
    if (!waves) {
      if (a.plan.N < kChanFewestSamples || !stream_preferred(a, dir, aligned, tiled_ok)) return true;
      const bool wide = cluster >= 4 && (uint64_t)blocks * kChanUnit < (uint64_t)a.plan.C * cluster;      // (more channels to a unit)
      if (extra_bwd && wide && (elements < kChanWaves || a.plan.N < kChanWideSamples)) return true;
      if (!extra_bwd && (elements < kChanWaves || (uint64_t)a.plan.C * g.cluster <= places || cluster > 2 || blocks > 3 * sm_count())) return true;
    }
    return cluster == 0 || cluster > 8;
  }
  if (stream_preferred(a, dir, aligned, tiled_ok)) return false;
  if (elements >= kChanLarge && segres_applies(a, dir, aligned)) return false;
  return elements < (extra && dir == 1 ? kChanLargeExtra : kChanLarge) || !(tiled_ok && a.plan.dim0 >= kChanLongRow);
}

int launch_chan(FusedArgs &a, int dir, bool aligned, cudaStream_t stream)
{
  ChanGeom g;
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  if (!chan_geom(a.plan.dim0, a.plan.C, a.plan.N, dir, extra, aligned, g)) return ANODE_E_LAUNCH;
  uint32_t blocks, threads;
  chan_grid(g, a.plan.C, blocks, threads);
  const bool adds = dir == 1 && a.accumulate;
  ChanKernel k = chan_kernel_of(g, dir, extra, adds, chan_dense(g, dir, extra, adds, blocks, threads));
  if (!k) return ANODE_E_LAUNCH;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  // The launch may overlap the tail of the kernel before it on the stream; every block waits for that kernel's
  // results (griddepcontrol.wait) before it touches memory.
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = g.cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = g.cluster > 1 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, k, a, g) != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

}  // namespace anode_b200

// ---- diagnostics: the form launched for a shape, of aligned tensors ------------------------------
extern "C" int anode_gpu_batch_norm_register_form(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  for (int i = 0; i < 8; ++i) out[i] = 0;
  ChanGeom g;
  const bool extra = residual != 0;
  if (!chan_geom(dim0, dim1, dim2, dir, extra, true, g)) return ANODE_OK;
  uint32_t blocks, threads;
  chan_grid(g, dim1, blocks, threads);
  out[0] = 1; out[1] = g.floats; out[2] = g.cluster; out[3] = blocks; out[4] = threads;
  if (g.floats <= 8) for (int dense = 0; dense < 2; ++dense) out[5 + dense] = chan_resident(g, dir, extra, false, dense != 0, threads);
  out[7] = chan_dense(g, dir, extra, false, blocks, threads);
  return ANODE_OK;
}
