// Host-side declarations shared by the translation units of libanode_routines_gpu.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "../../include/anode_routines_gpu.h"
#include "bn_band.cuh"
#include "bn_fused.cuh"

namespace anode_b200 {

// Geometry of the streaming kernel (bn_stream.cu)
struct StreamGeom {
  uint32_t cb, units;        // channels per unit
  uint32_t cluster, rows;    // blocks per unit, samples per block
  uint32_t groups, threads;  // sample groups of a block: thread = group * vectors per run + vector
  float cost;                // estimated us (of a prepared call's geometry)
  double inv_count;
};

// Geometry of its counterpart for long rows (bn_long.cu), and its blocks per SM
constexpr uint32_t kLongBlocks = 3;
struct LongGeom {
  uint32_t cluster, stride;         // blocks per channel, distance between a thread's vectors
  uint32_t per_row, total;          // vectors per row and per channel
  uint32_t step_rows, step_col;     // a step of `stride` vectors
  float cost;                       // estimated us
  double inv_count;
};

// Launch of a grid of clusters that may overlap the tail of the kernel before it on the stream (every block waits for that kernel's
// results before it touches memory).  ANODE_E_LAUNCH where the device refuses it.
template <typename Geom>
inline int launch_clusters(void (*kernel)(const FusedArgs, const Geom), const FusedArgs &a, const Geom &g, uint32_t blocks, uint32_t threads,
                           uint32_t cluster, cudaStream_t stream)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;      // (as launch_chan)
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = 2;
  if (cluster > 8) {
    // larger than the portable size: asked for once per kernel and device
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, bool> allowed;
    int dev = 0;
    (void)cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair((const void *)kernel, dev);
    auto it = allowed.find(key);
    if (it == allowed.end()) {
      const bool ok = cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
      if (!ok) (void)cudaGetLastError();
      it = allowed.emplace(key, ok).first;
    }
    if (!it->second) return ANODE_E_LAUNCH;
  }
  if (cudaLaunchKernelEx(&cfg, kernel, a, g) != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

struct Tunables {
  uint32_t tile_floats;     // target floats per tile
  uint32_t slack_steps;     // extra lookahead steps beyond the minimum
  uint32_t blocks_per_sm;   // persistent blocks planned per SM
  uint32_t ring_slots;      // shared-memory slots per block (forward)
  uint32_t ring_slots_bwd;  // shared-memory slots per block (backward; a slot holds x and dy)
  uint32_t ring_floats_fwd; // floats per slot (forward: x)
  uint32_t ring_floats_bwd; // floats per tensor per slot (backward: x and dy)
  uint32_t ring_blocks_per_sm;
};
const Tunables &tunables();

uint32_t sm_count();
Plan plan_for(uint32_t dim0, uint32_t C, uint32_t N, bool aligned16);
int check_dims(uint32_t dim0, uint32_t dim1, uint32_t dim2);
bool aligned16(const void *p);
bool aligned4(const void *p);

int prepare_fwd(FusedArgs &a, uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate,
                int relu, const float *x, const float *gamma, const float *beta, float *y, float *mean,
                float *var, float *run_mean, float *run_var, void *ws, size_t ws_bytes);
int prepare_bwd(FusedArgs &a, uint32_t dim0, uint32_t dim1, uint32_t dim2, int relu, int accumulate,
                const float *dy, const float *x, const float *mean, const float *var, const float *gamma,
                const float *beta, float *dx, float *dgamma, float *dbeta, void *ws, size_t ws_bytes);
int launch_pipeline(FusedArgs &a, int dir, cudaStream_t stream);
// the kernel that serves a prepared call (ANODE_KERNEL_*, -1 for none), and its launch
int pick_kernel_kind(const FusedArgs &a, int dir, bool aligned);
int launch_best(FusedArgs &a, int dir, bool aligned, cudaStream_t stream);
int kernel_choice();
// large layers of aligned rows that the tiled kernel serves faster than the streaming kernel
bool tiled_takes(uint32_t dim0, uint64_t elements, int dir, bool extra);
// the cluster kernel for short rows (bn_segres.cu)
bool segres_applies(const FusedArgs &a, int dir, bool aligned);
uint32_t segres_blocks(const FusedArgs &a, int dir, bool aligned);     // blocks of its launch, 0 where it does not apply
bool segres_preferred(const FusedArgs &a, int dir, bool aligned);      // take it even where the tiled kernel applies
int launch_segres(FusedArgs &a, int dir, cudaStream_t stream);
// the register-resident kernel (bn_chan.cu); one GPU, any alignment
bool chan_applies(const FusedArgs &a, int dir, bool aligned);
bool chan_preferred(const FusedArgs &a, int dir, bool aligned, bool tiled_ok);
int launch_chan(FusedArgs &a, int dir, bool aligned, cudaStream_t stream);
// the streaming cluster kernel for large layers of short rows (bn_stream.cu); one GPU
bool stream_applies(const FusedArgs &a, int dir, bool aligned);
uint32_t stream_cluster(const FusedArgs &a, int dir, bool aligned, uint32_t &blocks);
bool stream_preferred(const FusedArgs &a, int dir, bool aligned, bool tiled_ok);
int launch_stream(FusedArgs &a, int dir, cudaStream_t stream);
bool stream_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, StreamGeom &g);      // geometry of a shape, and of a prepared call
bool stream_geom_of(const FusedArgs &a, int dir, StreamGeom &g);
// its masked form for rows without an aligned run: the geometry of a shape, and of a prepared call on aligned tensors
bool masked_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, StreamGeom &g);
bool masked_geom_of(const FusedArgs &a, int dir, StreamGeom &g);
// its counterpart for small layers of long rows (bn_long.cu), likewise
bool long_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, LongGeom &g);
bool long_geom_of(const FusedArgs &a, int dir, LongGeom &g);
int launch_long(FusedArgs &a, const LongGeom &g, int dir, cudaStream_t stream);
bool stream_one_wave(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra);      // its grid, where it fills the device once
// its form for the largest of them (bn_band.cu): the geometry of a shape where it is taken, and of a prepared call
bool band_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, BandGeom &g);
bool band_geom_of(const FusedArgs &a, int dir, BandGeom &g);
int launch_band(FusedArgs &a, const BandGeom &g, int dir, cudaStream_t stream);
uint64_t workspace_part_bytes(uint32_t dim0, uint32_t C, uint32_t N);
uint64_t workspace_static_bytes(uint32_t dim0, uint32_t C, uint32_t N);
uint64_t ring_ws_bytes(const FusedArgs &a, int dir, bool aligned);
// the slice-resident kernel (bn_resident.cu)
bool resident_applies(const FusedArgs &a, int dir, bool aligned);
uint64_t resident_ws_bytes(uint32_t dim0, uint32_t C, uint32_t N);
int launch_resident(FusedArgs &a, int dir, uint64_t ws_off, cudaStream_t stream);
long long wait_limit_cycles();
uint64_t control_region_bytes(uint32_t dim0, uint32_t C, uint32_t N, bool aligned);

// synchronized launches (bn_sync.cu), for the host-buffer step
int sync_launch(FusedArgs &a, int dir, bool aligned, struct ::AnodeSyncComm *comm, size_t fused_ws_bytes, cudaStream_t stream);
size_t sync_gather_bytes(uint32_t C, const struct ::AnodeSyncComm *comm);
int sync_world(const struct ::AnodeSyncComm *comm);

}  // namespace anode_b200
