// The front end's own composition (src/ops.rs:999-1014: mean, variance, two running averages, normalize) and its adjoint
// (the seven ops that src/ops_gpu.rs:4344-4352, 3997-4003 and 3787-3791 emit), one launch each, without scratch memory
// (large layers of few channels: the normalization is a launch of its own, normalized_apart).
//
// A thread-block cluster of up to eight blocks owns a channel and visits it two or three times, the sums of a visit going
// through distributed shared memory before the next one begins:
//   forward   sum x -> mean; sum (x-mean)^2 -> var, running averages; y = (x-mean) * rsqrt(var)
//   adjoint   sums of dy*(x-mean), dy and x-mean -> dvar, dmean; dx = dy*rsqrt(var) + dvar*(x-mean)*2/norm + dmean/norm
// Where a channel fits the cluster's registers it is read once; else the later visits find it in L2, a cluster's share being
// small.  Forward passes that the register-resident and streaming kernels of the fused calls serve (short rows) are
// theirs; the expressions here are the reference's op by op (rsqrtf; mean need not be the batch's in the adjoint).
//
// What bounds the composition, [64,128,28,28] (26 MB tensors): seventeen launches and twenty passes over L2 took 114.5 us,
// composition and adjoint in one launch each and the two ReLU maps 47.
#include <cooperative_groups.h>

#include "bn_device.cuh"
#include "bn_host.h"

namespace cg = cooperative_groups;

namespace anode_b200 {

constexpr uint32_t kComposeThreads = 512, kComposeCluster = 8;
constexpr uint64_t kComposeSmall = 128u << 10;      // floats of a small channel (launch_compose)
constexpr int kComposeHold = 4;       // vectors per tensor that a thread holds (64 registers: two blocks per SM)
constexpr uint64_t kComposeWindow = 100u << 20;      // bytes between the two walks of an adjoint, where all blocks are resident (launch_compose)
constexpr int kComposeScalars = 8;    // floats in flight per thread and tensor where rows are loaded float by float

struct ComposeArgs {
  uint32_t dim0, C, N;
  float epsilon, avg_rate;
  const float *x, *dy, *mean_in, *var_in;
  float *out, *mean, *var, *run_mean, *run_var;      // adjoint: dx, dmean, dvar; forward: no out, no third visit
};

// Sums of K values over the threads of the cluster, in a fixed order, to every thread.
template <int K>
__device__ __forceinline__ void cluster_sums(cg::cluster_group &cluster, double (&v)[K], double (*part)[kComposeThreads / 32],
                                             double (*gather)[kComposeCluster])
{
  const uint32_t tid = threadIdx.x, cs = cluster.num_blocks(), rank = cluster.block_rank(), warps = blockDim.x / 32;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    v[k] = warp_sum(v[k]);
    if ((tid & 31) == 0) part[k][tid >> 5] = v[k];
  }
  __syncthreads();
  if (tid < K * cs) {
    const uint32_t k = tid / cs, r = tid - k * cs;
    double s = 0.0;
    for (uint32_t w = 0; w < warps; ++w) s += part[k][w];
    cluster.map_shared_rank(&gather[k][0], r)[rank] = s;
  }
  cluster.sync();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    v[k] = 0.0;
    for (uint32_t r = 0; r < cs; ++r) v[k] += gather[k][r];
  }
}

// HOLD: the thread's vectors (at most kComposeHold) stay in registers
template <int DIR, int VEC, bool HOLD>
__global__ void __launch_bounds__(kComposeThreads, 2) bn_compose_kernel(const ComposeArgs g)
{
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t cs = cluster.num_blocks(), rank = cluster.block_rank();
  const uint32_t c = blockIdx.x / cs;
  __shared__ double part[3][kComposeThreads / 32], gather[2][3][kComposeCluster];
  // remote shared memory may only be written once its block runs (collected before the first sums)
  if (cs > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

  // the thread's vectors are j0, j0 + stride, ... of the channel, B of them in flight; places by walking (row, column) along
  // (float offsets are below 2^32, check_dims)
  // Four chains of additions per thread (that of dy * (x - mean) three or four).  Where the cluster is chosen for the waves of blocks
  // (launch_compose) they are emptied into double precision after every batch, so that a chain is two to four additions however much a
  // thread walks: the adjoint's sums are no further from float64 than with the larger clusters, relative error of dmean of [300,16,56,56] 7.1e-8
  // and, without, 1.1e-7.  It costs three to six per cent where the cluster is the same anyway, which a third vector in flight makes good, us
  // without and with both: [3483,7,16,16] 35.9 and 32.8, [2426,4,16,16] 24.5 and 22.7, but [192,6,28,28] 7.3 and 7.7, [52,32,35,60] 12.5 and 14.2.
  constexpr int B = HOLD ? kComposeHold : VEC == 1 ? kComposeScalars : DIR == 0 ? kComposeHold : kComposeHold - 1;      // (four of the adjoint's spill)
  constexpr int D = HOLD || VEC == 1 ? kComposeHold : kComposeHold - 1;
  const uint32_t per_row = g.dim0 / VEC, total = per_row * g.N, rs = g.C * g.dim0;
  const uint32_t stride = cs * blockDim.x, j0 = rank * blockDim.x + threadIdx.x;
  const uint32_t row0 = j0 / per_row, drow = stride / per_row;
  const uint32_t col0 = j0 - row0 * per_row, dcol = stride - drow * per_row;
  const uint32_t off0 = c * g.dim0 + row0 * rs + col0 * VEC;
  const uint32_t step = drow * rs + dcol * VEC, wrap = rs - per_row * VEC;
  const uint32_t cnt = j0 < total ? (total - j0 - 1) / stride + 1 : 0;
  pdl_wait();
  pdl_trigger();

  Pack<VEC> vx[B], vd[DIR == 1 ? B : 1];
  // visit(f, turn): f(x, dy, offset, number of the vector in its batch) for every vector, B loads in flight, and turn() after every
  // batch; the first visit of a held channel loads it
  bool loaded = false;
  auto visit = [&](auto f, auto turn) {
    uint32_t off = off0, col = col0;
    for (uint32_t k = 0; k < cnt; k += B) {
      uint32_t at[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        at[u] = off;
        if (k + u < cnt && !(HOLD && loaded)) {
          vx[u] = Pack<VEC>::load(g.x + off);
          if (DIR == 1) vd[u] = Pack<VEC>::load(g.dy + off);
        }
        off += step; col += dcol;
        if (col >= per_row) { col -= per_row; off += wrap; }
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
        if (k + u < cnt) f(vx[u], vd[DIR == 1 ? u : 0], at[u], u);
      if (HOLD) break;
      if (DIR == 1 || VEC == 1) turn();
    }
    loaded = true;
  };
  const float norm = (float)g.dim0 * (float)g.N;

  auto nothing = [] {};
  if constexpr (DIR == 0) {
    float acc[kComposeHold] = {};
    double v[1] = {0.0};
    auto empty = [&] { v[0] += ((double)acc[0] + (double)acc[1]) + ((double)acc[2] + (double)acc[3]); acc[0] = acc[1] = acc[2] = acc[3] = 0.f; };
    visit([&](const Pack<VEC> &x, const Pack<VEC> &, uint32_t, int u) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[u % kComposeHold] += x.v[i];
    }, empty);
    empty();
    if (cs > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    cluster_sums(cluster, v, part, gather[0]);
    const float m = (float)v[0] / norm;                               // batch_norm.cu:54
    v[0] = 0.0;
    visit([&](const Pack<VEC> &x, const Pack<VEC> &, uint32_t, int u) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) { const float d = x.v[i] - m; acc[u % kComposeHold] += d * d; }
    }, empty);
    empty();
    cluster_sums(cluster, v, part, gather[1]);
    const float var = (float)v[0] / norm + g.epsilon;                 // batch_norm.cu:160
    if (rank == 0 && threadIdx.x == 0) {
      g.mean[c] = m; g.var[c] = var;
      if (g.run_mean) { const float o = g.run_mean[c]; g.run_mean[c] = o + g.avg_rate * (m - o); }
      if (g.run_var) { const float o = g.run_var[c]; g.run_var[c] = o + g.avg_rate * (var - o); }
    }
    if (!g.out) return;
    const float r = rsqrtf(var);                                      // batch_norm.cu:333
    visit([&](const Pack<VEC> &x, const Pack<VEC> &, uint32_t at, int) {
      Pack<VEC> o;
#pragma unroll
      for (int i = 0; i < VEC; ++i) o.v[i] = (x.v[i] - m) * r;
      o.put(g.out + at);
    }, nothing);
  } else {
    const float m = g.mean_in[c], va = g.var_in[c], r = rsqrtf(va);
    float a1[D] = {}, a2[kComposeHold] = {}, a3[kComposeHold] = {};
    double v[3] = {0.0, 0.0, 0.0};
    auto empty = [&] {
#pragma unroll
      for (int u = 0; u < D; ++u) { v[0] += (double)a1[u]; a1[u] = 0.f; }
      v[1] += (double)a2[0] + (double)a2[1] + ((double)a2[2] + (double)a2[3]); v[2] += (double)a3[0] + (double)a3[1] + ((double)a3[2] + (double)a3[3]);
      a2[0] = a2[1] = a2[2] = a2[3] = a3[0] = a3[1] = a3[2] = a3[3] = 0.f;
    };
    visit([&](const Pack<VEC> &x, const Pack<VEC> &dy, uint32_t, int u) {
#pragma unroll
      for (int i = 0; i < VEC; ++i) {
        const int chain = (u + i) % kComposeHold;
        const float d = x.v[i] - m;
        a1[(u + i) % D] = fmaf(dy.v[i], d, a1[(u + i) % D]); a2[chain] += dy.v[i]; a3[chain] += d;
      }
    }, empty);
    empty();
    if (cs > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    cluster_sums(cluster, v, part, gather[0]);
    const float dvar = (float)((double)(-0.5f * r / va) * v[0]);                            // batch_norm.cu:492
    const float dmean = (float)(-(double)r * v[1]) + (float)((double)(-dvar * 2.0f) * v[2]) / norm;      // :420, :255, :277
    if (rank == 0 && threadIdx.x == 0) { g.var[c] = dvar; g.mean[c] = dmean; }
    const float k1 = dvar * 2.0f / norm, k0 = dmean / norm;                                 // :203, :92
    visit([&](const Pack<VEC> &x, const Pack<VEC> &dy, uint32_t at, int) {
      Pack<VEC> o;
#pragma unroll
      for (int i = 0; i < VEC; ++i) o.v[i] = fmaf(dy.v[i], r, fmaf(x.v[i] - m, k1, k0));
      o.put(g.out + at);
    }, nothing);
  }
}

// Forward passes over aligned rows whose few clusters leave SMs idle: the normalization goes over the whole device in a launch
// of its own, where the clusters of eight have a block for every SM at most and a channel is large.  Us in one launch, in two,
// and op by op:
//   1 channel   3 M 59, 33, 46, 25 M 702, 440, 492      3   3 M 23, 18, 27, 10 M 78, 50, 66, 50 M 544, 390, 423
//   8 channels  10 M 29, 29, 43, 25 M 121, 101, 116     16  25 M 83, 77, 88, 50 M 160, 148, 161
// but 12 channels 10 M 23.4, 24.5, 37, and of 36 200 M 630, 650, 598.  (Rows that threads load float by float gain little by
// it: 8 channels, 10 M 56, 67, 136.)
constexpr uint64_t kApartChannel = 1u << 20;
static bool normalized_apart(uint32_t dim0, uint32_t C, uint32_t N, bool aligned)
{
  return dim0 % 4 == 0 && aligned && (uint64_t)dim0 * N >= kApartChannel && (uint64_t)C * kComposeCluster <= sm_count();
}

template <int DIR>
static int launch_compose(const ComposeArgs &g, bool aligned, cudaStream_t stream)
{
  const bool vec = g.dim0 % 4 == 0 && aligned;
  const uint64_t total = (uint64_t)(vec ? g.dim0 / 4 : g.dim0) * g.N;
  // The smallest cluster that holds the channel, else one of eight; but the adjoint, and forward passes that load the floats of small
  // channels one by one, no larger than makes two blocks per SM, what is resident: more blocks only repeat the fixed steps of a cluster.
  // (Two where a thread of one block would have 64 floats and more; two that hold the channel.)  Adjoint with the cluster that
  // holds the channel or eight, and so, us: [64,128,28,28] 25.2 and 20.0, [32,64,56,56] 25.9 and 19.6, [64,512,28,28] 88 and 76, [64,128,27,27]
  // 32.4 and 21.2, [40,300,15,15] 39.5 and 15.4, [256,1024,7,7] 132 and 49, [16,95,55,55] 24.6 and 19.6.  Forward [32,512,27,27] 66 and 40,
  // but [65,1024,55,55] 684 and 798.
  // The adjoint's second walk wants to find the channels in flight in L2 (kComposeWindow): with the cluster by waves alone, and larger ones up to
  // eight while they exceed it, [256,150,28,28] 121 and 90, [256,512,28,28] 330 and 283, [91,512,32,32] 149 and 129.
  // (Less where blocks leave and others come: [207,646,28,28] with 96 MB 317 and, with 48, 285; [408,143,14,14], resident, with 91 MB 36.6 and 41.4.
  // Not where eight would exceed it by far, [1285,108,28,28] 336 and 353, nor scalar rows, which wait for less, [958,128,353] 149 and 159.)
  // And clusters of four and eight do not fill the device, their SMs lie together: [64,n,28,28] with 70 of four 12.4, with 72 17.7 ([1184,71,33], 71 of them, 12.4 and, of two, 13.5).
  const bool waves = DIR == 1 || (!vec && total <= kComposeSmall);
  const uint32_t lanes = vec ? 4u : 1u, wave = 2 * sm_count();
  auto holds = [&](uint32_t n) { return total <= (uint64_t)n * kComposeThreads * kComposeHold; };
  auto window = [&](uint32_t n) { return (g.C < wave / n ? g.C : wave / n) * total * lanes * 8; };
  const bool near = DIR == 1 && vec && window(kComposeCluster) <= kComposeWindow * 3 / 2;
  uint32_t cs = 1;
  while (cs < kComposeCluster && !holds(cs) &&
         (!waves || (uint64_t)g.C * cs * 2 <= (cs == 1 || DIR == 0 ? wave : wave * 24 / 25) ||
          (cs == 1 && (total * lanes >= 64ull * kComposeThreads || (vec && holds(2)))) || (near && window(cs) > ((uint64_t)g.C * cs <= wave ? kComposeWindow : kComposeWindow * 4 / 5)))) cs *= 2;
  if (DIR == 1 && vec && !holds(cs) && holds(kComposeCluster)) {
    // A cluster that holds the channel needs no second walk.  It is the faster one where the others leave a few SMs with one block more than the
    // rest or with a wave of their own, and beyond a wave where its threads are nearly full of what they hold.  Us without and with:
    // [64,75,28,28] 16.6 and 15.9, [48,75,28,28] 13.2 and 11.9, [64,150,28,28] 29.5 and 27.0, [24,310,28,28] 23.2 and 18.8; [14,969,40,55] 94 and 77,
    // [5,512,112,112] 90 and 87, but two thirds full, [45,512,32,32], 67 and 74.
    const uint64_t blocks = (uint64_t)g.C * cs;
    uint32_t n = 2 * cs;
    while (!holds(n)) n *= 2;
    if ((blocks * 2 > wave && blocks * 10 <= wave * 7ull) || (blocks > wave && blocks < 3ull * wave && blocks % wave && blocks % wave * 4 <= wave) ||
        (blocks > wave && total * 8 >= 7ull * n * kComposeThreads * kComposeHold)) cs = n;
  }
  const bool hold = holds(cs);
  // threads of a block: a vector each where all of them are resident at once, else up to what one holds
  const uint64_t each = (total + cs - 1) / cs;
  uint32_t threads = kComposeThreads;
  for (uint32_t k = 1; k <= kComposeHold; ++k) {
    const uint64_t t = ((each + k - 1) / k + 31) / 32 * 32;
    if (t < threads && (hold || k == 1)) threads = (uint32_t)t;
    if (!hold || (uint64_t)g.C * cs * threads <= 1024ull * sm_count()) break;
  }
  if ((uint64_t)g.C * cs > 0x7fffffffull) return ANODE_E_DIMS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(g.C * cs);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // (as in bn_legacy.cu)
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  auto kernel = vec ? (hold ? bn_compose_kernel<DIR, 4, true> : bn_compose_kernel<DIR, 4, false>)
                    : (hold ? bn_compose_kernel<DIR, 1, true> : bn_compose_kernel<DIR, 1, false>);
  if (cudaLaunchKernelEx(&cfg, kernel, g) != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

}  // namespace anode_b200

using namespace anode_b200;

extern "C" int anode_gpu_batch_normalize_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate, const float *x, float *y, float *mean, float *var,
    float *run_mean, float *run_var, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  const int rc = check_dims(dim0, dim1, dim2);
  if (rc) return rc;
  if (!x || !y || !mean || !var) return ANODE_E_NULL;
  if (!aligned4(x) || !aligned4(y)) return ANODE_E_ALIGN;
  const bool aligned = aligned16(x) && aligned16(y);
  // a fused call without affine step and activation, as far as its kernel needs no scratch
  FusedArgs a{};
  a.plan = plan_for(dim0, dim1, dim2, aligned);
  a.ws_capacity = workspace_part_bytes(dim0, dim1, dim2);
  a.x = x; a.out = y; a.mean = mean; a.var = var; a.run_mean = run_mean; a.run_var = run_var;
  a.epsilon = epsilon; a.avg_rate = avg_rate; a.neg_slope = 1.0f;
  a.mode = MODE_FUSED;
  a.count_total = (double)dim0 * (double)dim2;
  const int kind = pick_kernel_kind(a, 0, aligned);
  if (kind == ANODE_KERNEL_REGISTER && launch_chan(a, 0, aligned, stream) == ANODE_OK) return ANODE_OK;
  if (kind == ANODE_KERNEL_STREAM && launch_stream(a, 0, stream) == ANODE_OK) return ANODE_OK;
  ComposeArgs g{};
  g.dim0 = dim0; g.C = dim1; g.N = dim2; g.epsilon = epsilon; g.avg_rate = avg_rate;
  g.x = x; g.out = y; g.mean = mean; g.var = var; g.run_mean = run_mean; g.run_var = run_var;
  if (!normalized_apart(dim0, dim1, dim2, aligned)) return launch_compose<0>(g, aligned, stream);
  g.out = nullptr;
  const int stats = launch_compose<0>(g, aligned, stream);
  if (stats) return stats;
  anode_gpu_batch_norm_3d1_packed_f32(dim0, dim1, dim2, x, mean, var, y, cfg, stream);
  if (cudaGetLastError() != cudaSuccess) return ANODE_E_LAUNCH;
  return ANODE_OK;
}

extern "C" int anode_gpu_batch_normalize_adjoint_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, const float *dy, const float *x, const float *mean, const float *var,
    float *dx, float *dmean, float *dvar, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  const int rc = check_dims(dim0, dim1, dim2);
  if (rc) return rc;
  if (!dy || !x || !mean || !var || !dx || !dmean || !dvar) return ANODE_E_NULL;
  if (!aligned4(x) || !aligned4(dy) || !aligned4(dx)) return ANODE_E_ALIGN;
  ComposeArgs g{};
  g.dim0 = dim0; g.C = dim1; g.N = dim2;
  g.x = x; g.dy = dy; g.mean_in = mean; g.var_in = var; g.out = dx; g.mean = dmean; g.var = dvar;
  return launch_compose<1>(g, aligned16(x) && aligned16(dy) && aligned16(dx), stream);
}
