/* Diagnostic exports of libanode_routines_gpu: the planners behind the fused batch-norm kernels, as
 * plain index arithmetic that runs without a GPU.  They exist for the tests of the tile plans and
 * schedules and for measurements (which kernel serves a shape); no counterpart in the reference,
 * whose kernels take their launch shape from KernelConfig (routines_gpu/common.cuh:51-67). */
#ifndef ANODE_ROUTINES_GPU_DIAG_H
#define ANODE_ROUTINES_GPU_DIAG_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

/* Kernel that serves direction `dir` (0 forward, 1 backward) of a fused call, with a workspace of the full size: an ANODE_KERNEL_*
 * value of anode_routines_gpu.h.  STREAM and LONG may be launched in the place of PLAIN, REGISTER or TILED, and BAND in the place of
 * STREAM; anode_gpu_batch_norm_fused_launched_kernel tells.  residual: the residual-epilogue calls; aligned: every tensor on a
 * 16-byte boundary; world: ranks of a synchronized call whose communicator has an exchange buffer (1: a call on one
 * GPU).  ANODE_KERNEL_AUTO (0): a synchronized call that no kernel with the exchange inside serves (a reduce, an
 * exchange and an apply kernel are launched). */
int anode_gpu_batch_norm_fused_serving_kernel(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual,
                                              int aligned, int world);

/* Kernel that such a call on one GPU launches first; another one only where the device refuses its clusters. */
int anode_gpu_batch_norm_fused_launched_kernel(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, int aligned);

/* ANODE_KERNEL_* value of the kernel that this thread's last fused call launched, in one launch or with the exchange apart, BAND and
 * STREAM told apart; -1 before the first one. */
int anode_gpu_batch_norm_fused_last_kernel(void);

/* Family, among the first four ANODE_KERNEL_* values, that the shape of a plain fused call on 16-byte aligned tensors
 * belongs to.  (The REGISTER and STREAM kernels and the TILED kernel's ragged rows count as the family whose shapes they
 * take over on one GPU; for the kernel that is launched ask anode_gpu_batch_norm_fused_launched_kernel.) */
int anode_gpu_batch_norm_fused_kernel_kind(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir);

/* The same for the residual-epilogue calls (anode_gpu_batch_norm_add_act_fused_*). */
int anode_gpu_batch_norm_add_act_fused_kernel_kind(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir);

/* Tile plan of the tiled and plain kernels.  out (15 values): regime, vec, cb, units, rows_per_tile,
 * piece_len, pieces, sample_blocks, tiles_per_unit, total_tiles, grid, lookahead_steps, div_mul,
 * workspace bytes (low, high).  Zero for resident_blocks / tile_floats / slack_steps = the library's
 * own values. */
int anode_gpu_batch_norm_fused_plan(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                    uint32_t resident_blocks, uint32_t tile_floats, uint32_t slack_steps,
                                    uint32_t *out, uint32_t out_len);
/* One tile of that plan.  out (8 values): unit, c0, cw, n0, rows, col0, len, base. */
int anode_gpu_batch_norm_fused_plan_tile(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                         uint32_t resident_blocks, uint32_t tile_floats, uint32_t tile, uint64_t *out);
/* `count` tiles first, first + stride, ... as the kernels' division-free iterator walks them (8 values each). */
int anode_gpu_batch_norm_fused_plan_walk(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                         uint32_t resident_blocks, uint32_t tile_floats,
                                         uint32_t first, uint32_t stride, uint32_t count, uint64_t *out);

/* Geometry of the cluster kernel.  out (6 values): applies, channels per unit, blocks per cluster, samples
 * per block, units, shared-memory bytes. */
int anode_gpu_batch_norm_segres_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, uint32_t *out);

/* Geometry of the streaming kernel.  out (7 values): applies, channels per unit, units, blocks per cluster, samples per
 * block, sample groups of a block, threads (of an ordinary call, without the residual epilogue). */
int anode_gpu_batch_norm_stream_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, uint32_t *out);

/* The same of its masked form, which serves rows without an aligned run of channels (and of the residual epilogue's calls). */
int anode_gpu_batch_norm_stream_masked_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out);

/* Geometry of the kernel for small layers of long rows.  out (7 values): applies, blocks per channel, distance between a thread's
 * vectors, vectors per row and per channel, rows and columns of such a distance. */
int anode_gpu_batch_norm_long_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out);

/* Launch of the register-resident kernel for a shape of aligned tensors.  out (8 values): applies, floats of a thread, blocks of a
 * team, blocks of the grid, threads of a block, blocks that an SM holds of the ordinary form and of the one of fewer registers
 * (teams of four or eight floats a thread; 0 otherwise, and where there is no device), whether the latter is launched. */
int anode_gpu_batch_norm_register_form(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out);

/* Geometry of the band kernel, the streaming kernel's form for large layers.  out (16 values): taken by a call with a workspace
 * of the full size (zeros behind a 0: the kernel cannot take the shape at all), channels per unit, units, sample groups of a tile,
 * samples per thread, samples of a tile, tiles per unit, blocks, steps between a tile's two visits, boxes per band, vectors of
 * a box's row, bytes of a box, slots, bytes of a slot, shared-memory bytes, log2 of the lanes per channel in the service warps. */
int anode_gpu_batch_norm_band_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out);

/* Geometry of the tiled kernel (bn_ring.cuh) for direction `dir` of a fused call on 16-byte aligned tensors.
 * out (12 values): applies, rows per tile, floats per row piece, tiles per unit, slots, bytes per slot, dynamic
 * shared memory bytes of the layout (the one-launch forms take the SM's whole), KiB between a tile's two visits, the
 * fraction (in 1/1000) of such a window that L2 would keep by itself (anode_gpu_batch_norm_tiled_keep: what tensor memory takes off it), thread blocks, steps between a tile's two visits, tiles. */
int anode_gpu_batch_norm_tiled_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, uint32_t *out);

/* Which of a block's tiles stay in tensor memory between their two visits (tiled kernel, one launch per direction).
 * out (10 values): tiles kept at a time (0: none), whether tile number `tile` of a block is kept, its place, the number
 * under which consumer warp `warp` is dealt vectors of that place, the warp's first column, kept tiles before this one,
 * vectors of the largest tile, consumer warps, columns per set of one vector per lane, steps between a tile's two visits. */
int anode_gpu_batch_norm_tiled_keep(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual,
                                    uint32_t tile, uint32_t warp, uint32_t *out);

/* Floats of the last of the pieces that the tiled kernel cuts a row into (the whole row where it cuts none), for direction
 * `dir` of a call on 16-byte aligned tensors, with or without the residual epilogue; 0 where it does not apply. */
uint32_t anode_gpu_batch_norm_tiled_last_piece(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual);

/* anode_gpu_batch_norm_fused_set_wait_limit_ms in SM clock cycles, for tests of what follows when a wait inside a kernel runs out. */
int anode_gpu_batch_norm_fused_set_wait_limit_cycles(uint32_t cycles);

/* Plan of the slice-resident kernel for `planes` tensors per shared-memory slot.  out (16 values): applies,
 * rows per piece, parts per row, floats per part, pieces per channel, blocks per team, teams, grid, pieces
 * per block and channel, slot bytes, slots, resident-ring slots, streaming-ring slots, resident pieces per
 * channel, load-ahead slots, shared-memory bytes. */
int anode_gpu_batch_norm_resident_plan(uint32_t dim0, uint32_t dim1, uint32_t dim2, uint32_t planes, uint32_t *out);
/* Event sequence of thread block `block` of that plan, 4 values per event (kind, channel index in the
 * team's list, piece, slot); returns the number of events (at most max_events are written) or a negative
 * ANODE_E_* code. */
long long anode_gpu_batch_norm_resident_schedule(uint32_t dim0, uint32_t dim1, uint32_t dim2, uint32_t planes,
                                                 uint32_t block, uint32_t *out, uint64_t max_events);

#ifdef __cplusplus
}
#endif
#endif
