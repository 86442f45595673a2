// Batch-norm with given statistics fused with the activation that follows it: the inference branch
// of batch_normalize_2d/3d (src/ops.rs:1010-1011: `switch(online, avg_mean, mean)` feeding
// BatchNormalize2dOp, evaluation loop examples/run_imagenet_mpi.rs:841-843) followed by
// positive_clip (routines_gpu/flat_map.cu:172-179) or leaky ReLU (flat_map.cu:44-52), in one pass:
//
//   y = act(gamma[c]*(x - mean[c])*var[c]^-1/2 + beta[c]),   act(t) = t * (t > 0 ? 1 : neg_slope)
//
// (var is what anode stores: biased variance + epsilon.)  One read and one write of the tensor:
// 8 bytes per element, HBM-bound.  A thread owns one 16-byte column of the sample (its channel
// never changes), computes its coefficients once and walks down the samples.
// On small layers the launch gap and the chain coefficients -> load -> store are the time, on ragged ones (float by float) what a
// thread has in flight: a thread loads four samples at a time, the first four ahead of its coefficients, and the grid is no
// larger than gives most threads four.  With one sample in flight and a thread for each of up to 32 blocks per SM, and so, us
// from buffer to buffer: [8,256,28,28] 4.1 and 3.3, [32,256,14,14] 4.1 and 2.9, [64,512,7,7] 6.8 and 3.7, [32,64,56,56] 11.7 and 9.9,
// [256,2048,7,7] 37.0 and 33.8, [64,95,55,55] 44.6 and 27.6, [256,256,56,56] 254 and 247 (1.01 of the copy bandwidth).
#include <initializer_list>

#include "bn_device.cuh"
#include "bn_host.h"

namespace anode_b200 {

constexpr uint32_t kInferThreads = 256;
constexpr uint32_t kInferFlight = 4;      // samples in flight per thread
constexpr uint64_t kInferCut = 1500000;   // floats of a single sample from which on its rows are cut

// The inputs carry no __restrict__: it would let the compiler treat their loads as reads of memory that nothing writes while
// the kernel runs and move them above pdl_wait(), where the kernel before this one may still be writing them (the running
// averages of a training step, the activations of the layer below).
// N samples, `step` floats apart, of C channels of `len` floats, `row` floats apart (a single sample's rows may be cut into pieces that
// take the place of samples, see the launch).
// PLACE: a thread's place from its row, else from its column, as long as nothing is cut ([1,3,5000011], whose threads have one float each, 73.4 us
// and 70.6; but 16-byte loads, [64,512,7,7] 3.9 and 4.0).
template <int VEC, bool PLACE>
__global__ void __launch_bounds__(kInferThreads) bn_infer_kernel(uint32_t len, uint32_t C, uint32_t N, uint32_t row, uint32_t step, float neg_slope,
                                                                 const float *x, const float *mean, const float *var,
                                                                 const float *gamma, const float *beta, float *y)
{
  const uint64_t per_sample = (uint64_t)C * len;                  // floats
  const uint64_t col = ((uint64_t)blockIdx.x * kInferThreads + threadIdx.x) * VEC;
  if (col >= per_sample) return;
  // channel of each of this thread's elements, and its coefficients (a sample has less than 2^32 floats, check_dims)
  uint32_t c = (uint32_t)col / len, off = (uint32_t)col - c * len;
  // this thread's samples: blockIdx.y, + gridDim.y, ...; `left` of the batch from the next one on
  uint32_t left = N - blockIdx.y;
  const size_t down = (size_t)gridDim.y * step;
  size_t at = (size_t)blockIdx.y * step + (PLACE ? (size_t)c * row + off : (size_t)col);
  Pack<VEC> p[kInferFlight];
  auto load = [&] {
#pragma unroll
    for (int u = 0; u < kInferFlight; ++u)
      if (u * gridDim.y < left) p[u] = Pack<VEC>::load(x + at + u * down);
  };
  pdl_wait();
  // the first samples' floats are on their way while the coefficients are made
  load();
  float sc[VEC], sh[VEC], mu[VEC];
  uint32_t prev = 0xffffffffu;
  float s0 = 0.f, b0 = 0.f, m0 = 0.f;
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    if (c != prev) {
      const float g = gamma ? gamma[c] : 1.0f;
      m0 = mean[c]; s0 = g * inv_std(var[c]); b0 = (gamma && beta) ? beta[c] : 0.0f;
      prev = c;
    }
    mu[i] = m0; sc[i] = s0; sh[i] = b0;
    if (++off == len) { off = 0; ++c; }
  }
  for (;;) {
#pragma unroll
    for (int u = 0; u < kInferFlight; ++u)
      if (u * gridDim.y < left) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
          const float t = fmaf(p[u].v[i] - mu[i], sc[i], sh[i]);
          p[u].v[i] = t * (t > 0.0f ? 1.0f : neg_slope);
        }
        p[u].store_stream(y + at + u * down);
      }
    if (left <= kInferFlight * gridDim.y) break;
    left -= kInferFlight * gridDim.y; at += kInferFlight * down;
    load();
  }
}

}  // namespace anode_b200

using namespace anode_b200;

extern "C" int anode_gpu_batch_norm_act_infer_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float neg_slope,
    const float *x, const float *mean, const float *var, const float *gamma, const float *beta,
    float *y, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  const int rc = check_dims(dim0, dim1, dim2);
  if (rc) return rc;
  if (!x || !y || !mean || !var) return ANODE_E_NULL;
  if (!aligned4(x) || !aligned4(y)) return ANODE_E_ALIGN;
  const bool vec = aligned16(x) && aligned16(y) && (uint64_t)dim1 * dim0 % 4 == 0;
  // A single sample leaves a thread one load: its rows are cut into pieces, which take the place of samples (us in one piece, and in four,
  // from memory: [1,515,64,64,64] 236.5 and 157.1, [1,16,96,96,96] 26.9 and 18.6, [1,132,128,128] 6.05 and 4.6, [1,92,128,128] 4.5 and 3.6).
  // The line is not drawn by measurements: some smaller ones would gain, too, [1,91,128,128] 4.6 and 3.7, [1,256,56,56] 3.7 and 2.9, while
  // [1,700,31,33], in three, stays at 2.9.
  uint32_t len = dim0, samples = dim2, step = dim1 * dim0;
  if (dim2 == 1 && (uint64_t)dim1 * dim0 >= kInferCut && (!vec || dim0 % 4 == 0)) {
    const uint32_t lanes = vec ? 4u : 1u;
    for (uint32_t n : {4u, 8u, 5u, 3u, 7u, 2u})
      if (dim0 % (n * lanes) == 0) { len = dim0 / n; samples = n; step = len; break; }
  }
  dim2 = samples;
  const uint64_t per_sample = (uint64_t)dim1 * len;
  const uint64_t cols = vec ? per_sample / 4 : per_sample;
  const uint64_t bx = (cols + kInferThreads - 1) / kInferThreads;
  if (bx > 0x7fffffffull) return ANODE_E_DIMS;
  // Samples per thread: a multiple of four that makes no more than `most` blocks per SM (eight are resident: where the launch is the
  // time one wave and a half, [8,95,55,55] 4.1 us with twelve and 5.0 with 16 to 64; on large layers more of them keep HBM busier,
  // [256,256,56,56] 266 us with twelve, 253 with 32 and 248 with 64, but [256,2048,7,7] 34.6, 33.9 and 35.7), or fewer than four where
  // that leaves SMs with one block ([8,256,28,28] 2.9 us with two of them, 3.5 with four and more).
  // (32-bit arithmetic: a 64-bit division costs what two per cent of the call do)
  const uint64_t elements = per_sample * dim2;
  const uint32_t sms = sm_count(), most = sms * (!vec || elements < (16u << 20) ? 12 : elements < (64u << 20) ? 32 : 64), wide = (uint32_t)bx;
  const uint32_t rows = most / wide;                 // blocks one below the other, at most
  uint32_t each = rows ? dim2 / rows + (dim2 % rows != 0) : dim2, by = 1;
  if (each < dim2) each = (each + kInferFlight - 1) / kInferFlight * kInferFlight;
  for (;; each /= 2) {
    by = dim2 / each + (dim2 % each != 0);           // (no more than `most`, so below 65536)
    if (each <= 1 || wide >= 2 * sms || wide * by >= 2 * sms) break;
  }
  const dim3 grid(wide, by);
  // The launch may overlap the tail of the kernel before it (every block waits for that kernel's results before it
  // touches memory): in a network at a serving batch the layers last a few microseconds each.
  cudaLaunchConfig_t cfg_ = {};
  cfg_.gridDim = grid; cfg_.blockDim = dim3(kInferThreads); cfg_.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg_.attrs = attr; cfg_.numAttrs = 1;
  const auto kernel = vec ? bn_infer_kernel<4, true> : len != dim0 ? bn_infer_kernel<1, true> : bn_infer_kernel<1, false>;
  const cudaError_t e = cudaLaunchKernelEx(&cfg_, kernel, len, dim1, dim2, dim0, step, neg_slope, x, mean, var, gamma, beta, y);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}
