// Host side of the fused batch-norm (+ReLU) entry points: argument checks, the tile plan,
// and the cooperative launch of the persistent kernels of bn_fused.cuh.
#include "bn_host.h"
// the warp-specialised kernel, instantiated with 8 and with 16 consumer warps
#define ANODE_RING_NS ring8
#define ANODE_RING_CONSUMERS 256
#include "bn_ring.cuh"
#undef ANODE_RING_NS
#undef ANODE_RING_CONSUMERS
#define ANODE_RING_NS ring16
#define ANODE_RING_CONSUMERS 512
#include "bn_ring.cuh"
#undef ANODE_RING_NS
#undef ANODE_RING_CONSUMERS

namespace anode_b200 {

// Ragged rows (a length that is no multiple of four floats): the shortest one the tiled kernel can take, forward and
// backward.  A row costs the producer a bulk copy per tensor, so below some length the plain kernel's 4-byte accesses
// are the faster form.  20 M elements, 33 channels, forward / backward in us, tiled against plain: 9 x 9 144 / 270
// against 116 / 160, 11 x 11 105 / 195 (116 / 161), 13 x 13 82 / 150 (116 / 161), 25 x 25 45 / 79 (117 / 160),
// 63 x 63 43 / 62 (113 / 155).
constexpr uint32_t kRaggedMinRow[2] = {112, 160};
// Workspace header: (exit counter, parity) of the tiled kernel's plans (words 3 and 4 are the slice-resident kernel's)
constexpr uint32_t kRingHdr = 4, kRingHdrRagged = 32, kRingHdrExtra = 40, kBandHdr = 48, kBandHdrExtra = 56;

// ---- planner constants, from sweeps on B200 -------------------------------------------------------
#ifndef ANODE_SLACK_STEPS
#define ANODE_SLACK_STEPS 2
#endif
#ifndef ANODE_RING_SLOTS_FWD
#define ANODE_RING_SLOTS_FWD 3
#endif
#ifndef ANODE_RING_SLOTS_BWD
#define ANODE_RING_SLOTS_BWD 4
#endif
#ifndef ANODE_RING_FLOATS_FWD
#define ANODE_RING_FLOATS_FWD 16384
#endif
#ifndef ANODE_RING_FLOATS_BWD
#define ANODE_RING_FLOATS_BWD 8192
#endif
const Tunables &tunables()
{
  static const Tunables t = {
      32768,    // tile_floats
      ANODE_SLACK_STEPS,        // slack_steps
      4,        // blocks_per_sm
      ANODE_RING_SLOTS_FWD,     // ring_slots
      ANODE_RING_SLOTS_BWD,     // ring_slots_bwd
      ANODE_RING_FLOATS_FWD,    // ring_floats_fwd
      ANODE_RING_FLOATS_BWD,    // ring_floats_bwd
      1,        // ring_blocks_per_sm
  };
  return t;
}

// Which kernel serves the fused calls: ANODE_KERNEL_AUTO picks by shape; any other value is tried first
// where that kernel applies (set by tests and measurements, process-wide).
static std::atomic<int> g_kernel_choice{ANODE_KERNEL_AUTO};
int kernel_choice() { return g_kernel_choice.load(std::memory_order_relaxed); }

uint32_t sm_count()
{
  // one entry per device ordinal; 148 (B200) when no device can be queried, so that the
  // planning helpers stay callable on a machine without a GPU
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return 148; }
  int v = cache[dev].load(std::memory_order_relaxed);
  if (v == 0) {
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) {
      (void)cudaGetLastError();
      v = 148;
    }
    cache[dev].store(v, std::memory_order_relaxed);
  }
  return (uint32_t)v;
}

// What planning derives from a shape alone.  A call asks for it several times and a training loop makes the
// same few calls over and over, so each thread keeps the answers for the shapes it saw last (a fixed number of
// entries, nothing shared between threads).  Planning on every call cost 10 - 50 us of host time, several times
// the kernel's own time on small layers (the slice-resident kernel's planner alone searches hundreds of layouts).
struct ShapeInfo {
  uint32_t dim0, C, N, sms;      // key; sms == 0: empty
  Plan plan[2];                  // tile plan: [pointers 16-byte aligned]
  bool ring_ok[2][2];            // warp-specialised kernel for aligned pointers: [direction][residual epilogue]
  Plan ring_plan[2][2];
  RingGeom ring_geom[2][2];
  uint64_t tiled_bytes, static_bytes, part_bytes;      // see fill_shape_info
  bool band_ok[2][2];            // the streaming kernel's form for the largest layers, likewise
  BandGeom band[2][2];
  // the streaming kernel and its masked form (one of them at most), and its counterpart for long rows, likewise: searched for when a
  // call first asks for them (0 not yet, 1 no, 2 yes), since most shapes never do and a search takes some ten microseconds
  mutable uint8_t stream_ok[2][2], masked_ok[2][2], long_ok[2][2];
  mutable StreamGeom stream[2][2];
  mutable LongGeom long_rows[2][2];
};
constexpr uint32_t kShapeCache = 64;      // entries per thread, direct mapped

static void fill_shape_info(ShapeInfo &s);

static const ShapeInfo &shape_info(uint32_t dim0, uint32_t C, uint32_t N)
{
  thread_local std::unique_ptr<ShapeInfo[]> cache;
  if (!cache) cache.reset(new ShapeInfo[kShapeCache]());
  const uint32_t sms = sm_count();
  const uint32_t h = (dim0 * 0x9e3779b1u) ^ (C * 0x85ebca6bu) ^ (N * 0xc2b2ae35u);
  ShapeInfo &s = cache[(h >> 16) % kShapeCache];
  if (s.dim0 != dim0 || s.C != C || s.N != N || s.sms != sms) {
    s.sms = 0;
    s.dim0 = dim0; s.C = C; s.N = N;
    fill_shape_info(s);
    s.sms = sms;
  }
  return s;
}

Plan plan_for(uint32_t dim0, uint32_t C, uint32_t N, bool aligned16) { return shape_info(dim0, C, N).plan[aligned16 ? 1 : 0]; }

constexpr uint32_t kRingSmemBudget = 227u * 1024u;      // a block's most
constexpr uint64_t kRingLargeWindowMax = 48ull << 20;     // what L2 keeps of a window between a tile's two visits

// vectors that a row takes in a slot, and those of the largest tile
static uint32_t ring_pitch(const Plan &p)
{
  const uint32_t len = p.piece_len < p.dim0 ? p.piece_len : p.dim0;
  return p.dim0 % 4 != 0 ? ragged_pitch(len) : len / 4;
}
static uint32_t ring_tile_vecs(const Plan &p) { return p.rows_per_tile * ring_pitch(p); }

// consumer warps of direction `dir` (the two instantiations of bn_ring.cuh)
static uint32_t ring_warps(int dir) { return dir == 0 ? 8u : 16u; }

// Bytes between the two visits of a tile: what L2 has to hold for the apply visit to find its tile there.
static uint64_t ring_window_bytes(const Plan &p, int dir)
{
  return (uint64_t)p.lookahead_steps * p.grid * p.rows_per_tile * p.piece_len * 4 * (dir == 1 ? 2 : 1);
}

// Forward passes on ragged rows from this length on: no tile stays in tensor memory.  The two forms of a ragged visit are long, and
// consumers that run one of them alone are faster than tensor memory makes them; on shorter rows the producer's copies, one per
// row and tensor, bound the kernel, and a kept tile needs one less.  Us with tensor memory, and without: [64,95,55,55] 39.8 and 35.5,
// [512,128,55,55] 328 and 295, [256,64,111,111] 328 and 305, [300,301,31,31] 149 and 146, but [1024,101,21,21] 84.7 and 85.3.  (A form
// with nothing but kept tiles: 40.4, 308, 303, 138.)  Not where L2 does not keep what lies between two visits, nor in layers of few
// channels, which come near that line from one size to the next: [1252,6,7485] 97 and 101, [952,3,14225] 75.5 and 76.6, but
// [598,11,1991] 29 and 25.
// Residual epilogue, with tensor memory, and without either: 40 M elements of 131 channels, rows of 301 119 and 144, 451 107 and 116,
// 601 103 and 103, 713 104 and 99, 1201 109 and 99; [34,123,6374] 96 and 70, [50,119,12674] 268 and 202, [200,100,5041] 357 and 273
// (where every second visit was one from L2, in an older form of both: 76, 238, 279).
constexpr uint32_t kRaggedKeepMost = 640, kRaggedKeepChannels = 24;
static bool ring_keeps(const Plan &p, int dir, bool extra)
{
  if (dir != 0 || p.dim0 % 4 == 0 || p.dim0 < kRaggedKeepMost) return true;
  return !extra && (p.C < kRaggedKeepChannels || ring_window_bytes(p, dir) > kRingLargeWindowMax);
}

// Fused mode: the tiles that stay in tensor memory.
static void ring_keep(const Plan &p, int dir, bool extra, RingGeom &g)
{
  g.keep_slots = 0; g.keep_period = 1;
  if (!ring_keeps(p, dir, extra)) return;
  plan_keep(g, ring_tile_vecs(p), dir == 1 ? 2u : 1u, ring_warps(dir), p.lookahead_steps);
}

// Shared-memory layout of the warp-specialised kernel for plan `p` (see bn_ring.cuh).
static RingGeom ring_geom(const Plan &p, int dir, bool extra, uint32_t slots, uint32_t slot_floats)
{
  RingGeom g{};
  g.slots = slots; g.slot_floats = slot_floats; g.hdr = kRingHdr;
  uint32_t off = kRingCtlBytes;
  const uint32_t cwarps = ring_warps(dir), planes = (dir == 1 ? 2u : 1u) + (extra ? 1u : 0u);
  g.res_stride = p.cb > cwarps ? p.cb : cwarps;   // regime R: one partial per consumer warp
  g.off_res = off;  off += (uint32_t)align_up_u64((uint64_t)kResQ * g.res_stride * 16, 128);
  g.off_coef = off; off += (uint32_t)align_up_u64((uint64_t)kCoefQ * kCoefBox * 16, 128);
  g.off_slots = off;
  g.slot_stride = (uint32_t)align_up_u64((uint64_t)slot_floats * 4 * planes + 32, 128);
  g.smem_bytes = off + slots * g.slot_stride;
  return g;
}

// Steps between a tile's two visits: the fewest, and `slack` more for a channel's statistics to come together.  Two, but
//  - three where a channel has no more tiles than there are blocks, so that each visit waits for another channel: backward
//    passes of many steps ([256,256,56,56] 414 - 425 -> 393 us), forward passes of few ([64,95,55,55] 41.0 -> 39.3,
//    [128,256,32,32] 53.6 -> 50.2; at 90 steps equal);
//  - one in backward passes whose window is over what L2 keeps even with a part of it in tensor memory
//    ([4,32,128,128,128] 605 -> 572 us; where the window fits one step is slower: [256,64,112,112] 394 -> 450).
static uint32_t ring_lookahead(const Plan &p, int dir)
{
  uint32_t slack = tunables().slack_steps;
  const uint32_t least = ceil_div_u32(p.tiles_per_unit, p.grid), steps = ceil_div_u32(p.total_tiles, p.grid);
  if (p.tiles_per_unit <= p.grid && (dir == 1 ? steps >= 32 : steps < 64)) ++slack;
  if (dir == 1 && slack > 1) {
    RingGeom g{};
    plan_keep(g, ring_tile_vecs(p), 2, ring_warps(dir), least + slack);
    const uint64_t window = (uint64_t)(least + slack) * p.grid * ring_tile_vecs(p) * 32;
    if (window * (g.keep_period - g.keep_slots) / g.keep_period > kRingLargeWindowMax) slack = 1;
  }
  return least + slack;
}

// Plan for the warp-specialised kernel, or false when it does not apply (scalar paths, tiles that
// do not fit a slot, too little shared memory): the caller then uses the plain kernel.
// Plan and geometry for `slots` slots of `slot_floats` floats (per tensor); false when they do not fit.
static bool ring_plan_with(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, uint32_t slots, uint32_t slot_floats, Plan &p, RingGeom &g)
{
  const Tunables &t = tunables();
  slot_floats = (slot_floats / 4) * 4;
  if (slot_floats < 1024) slot_floats = 1024;
  slots = slots < 2 ? 2 : (slots > kMaxSlots ? kMaxSlots : slots);
  uint32_t bps = t.ring_blocks_per_sm ? t.ring_blocks_per_sm : 1;
  // rows that are no multiple of four floats take up to 6 floats more in a slot (ragged_pitch)
  const bool ragged = dim0 % 4 != 0;
  if (ragged && dim0 < kRaggedMinRow[dir]) return false;
  uint32_t target = slot_floats;
  if (ragged) target = 4 * ragged_pitch(dim0) <= slot_floats ? slot_floats / (4 * ragged_pitch(dim0)) * dim0 : slot_floats - 8;
  p = make_plan(dim0, C, N, true, sm_count() * bps, target, t.slack_steps);
  // short rows (regime S) belong to the cluster kernel or the plain kernel
  if (p.regime != 0) return false;
  if (ragged) {
    // no last piece of a row of fewer than four floats (ragged_whole)
    while (p.pieces > 1 && dim0 - (p.pieces - 1) * p.piece_len < 4) {
      p.piece_len -= 4; p.pieces = ceil_div_u32(dim0, p.piece_len);
      p.tiles_per_unit = p.sample_blocks * p.pieces; p.total_tiles = p.units * p.tiles_per_unit;
      p.grid = p.total_tiles < sm_count() * bps ? p.total_tiles : sm_count() * bps;
    }
    // Equal tiles: the last of a channel would hold what is left over and cost a step all the same.  Forward, before and
    // now: [846,106,131] 67.8 and 61.8 us, [371,210,135] 65.8 and 55.5, [64,95,55,55] 41.9 and 42.0.
    p.rows_per_tile = ceil_div_u32(N, p.sample_blocks);
    p.vec = 4;
  }
  p.lookahead_steps = ring_lookahead(p, dir);
  // a tile must fit one slot
  const uint64_t tile_max = 4ull * ring_tile_vecs(p);
  if (tile_max > slot_floats) return false;
  slot_floats = (uint32_t)((tile_max + 31) / 32 * 32);     // slots no larger than the largest tile
  g = ring_geom(p, dir, extra, slots, slot_floats);
  while (g.smem_bytes > kRingSmemBudget && slots > 2) { --slots; g = ring_geom(p, dir, extra, slots, slot_floats); }
  return g.smem_bytes <= kRingSmemBudget;
}

// Backward pass: three slots of larger tiles are faster than four of the standard ones as long as the larger
// window they make still fits what L2 keeps ([256,256,56,56]: 0.50 -> 0.44 ms; with a 56 MB window 10 % slower).
constexpr uint32_t kRingLargeSlotsBwd = 3, kRingLargeFloatsBwd = 9408;

// The residual epilogue's slots hold a third tensor (a second one in the forward pass, used by the apply visits only).
#ifndef ANODE_RING_SLOTS_FWD_EXTRA
#define ANODE_RING_SLOTS_FWD_EXTRA 4
#endif
#ifndef ANODE_RING_FLOATS_FWD_EXTRA
#define ANODE_RING_FLOATS_FWD_EXTRA 9408
#endif
// (Forward, small layers: where the planner halves that for want of tiles and ends below what it makes of this.  Residual
// forward pass with the one and with the other, us: [149,5,2888] 19.9 and 15.3, [94,7,1197] 16.6 and 14.6, [113,15,1364]
// 16.0 and 14.7.)
#ifndef ANODE_RING_FLOATS_FWD_EXTRA_SMALL
#define ANODE_RING_FLOATS_FWD_EXTRA_SMALL 6656
#endif
#ifndef ANODE_RING_SLOTS_BWD_EXTRA
#define ANODE_RING_SLOTS_BWD_EXTRA 3
#endif
#ifndef ANODE_RING_FLOATS_BWD_EXTRA
#define ANODE_RING_FLOATS_BWD_EXTRA 6272
#endif
static bool make_ring_plan(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, Plan &p, RingGeom &g)
{
  const Tunables &t = tunables();
  auto tile = [](const Plan &q) { return (uint64_t)q.rows_per_tile * q.piece_len; };
  if (extra) {
    if (dir == 1) return ring_plan_with(dim0, C, N, dir, true, ANODE_RING_SLOTS_BWD_EXTRA, ANODE_RING_FLOATS_BWD_EXTRA, p, g);
    const bool ok = ring_plan_with(dim0, C, N, dir, true, ANODE_RING_SLOTS_FWD_EXTRA, ANODE_RING_FLOATS_FWD_EXTRA, p, g);
    Plan ps; RingGeom gs;
    if (ring_plan_with(dim0, C, N, dir, true, ANODE_RING_SLOTS_FWD_EXTRA, ANODE_RING_FLOATS_FWD_EXTRA_SMALL, ps, gs) &&
        (!ok || tile(ps) > tile(p))) { p = ps; g = gs; return true; }
    return ok;
  }
  if (!ring_plan_with(dim0, C, N, dir, false, dir == 0 ? t.ring_slots : t.ring_slots_bwd,
                      dir == 0 ? t.ring_floats_fwd : t.ring_floats_bwd, p, g)) return false;
  if (dir == 1) {
    Plan pl; RingGeom gl;
    if (ring_plan_with(dim0, C, N, dir, false, kRingLargeSlotsBwd, kRingLargeFloatsBwd, pl, gl) && gl.slots == kRingLargeSlotsBwd &&
        tile(pl) > tile(p) && ring_window_bytes(pl, dir) <= kRingLargeWindowMax) {
      p = pl; g = gl;
    }
  }
  return true;
}

bool ring_plan_for(uint32_t dim0, uint32_t C, uint32_t N, bool aligned, int dir, bool extra, Plan &p, RingGeom &g)
{
  if (!aligned) return false;
  const ShapeInfo &s = shape_info(dim0, C, N);
  if (!s.ring_ok[dir][extra]) return false;
  p = s.ring_plan[dir][extra]; g = s.ring_geom[dir][extra];
  return true;
}

// Plan of the warp-specialised kernel for a prepared call, or false when it does not serve it.  Ragged rows and the
// residual epilogue are one-launch, one-GPU forms.
static bool ring_serves(const FusedArgs &a, int dir, bool aligned)
{
  const bool extra = a.res || a.ymask || a.dres;
  if (!aligned || ((extra || a.plan.dim0 % 4 != 0) && (a.mode != MODE_FUSED || a.world > 1))) return false;
  const ShapeInfo &s = shape_info(a.plan.dim0, a.plan.C, a.plan.N);
  return s.ring_ok[dir][extra] && s.ring_plan[dir][extra].ws_bytes <= a.ws_capacity;
}
static bool ring_plan_of(const FusedArgs &a, int dir, bool aligned, Plan &p, RingGeom &g)
{
  return ring_serves(a, dir, aligned) && ring_plan_for(a.plan.dim0, a.plan.C, a.plan.N, aligned, dir, a.res || a.ymask || a.dres, p, g);
}

// Bytes of a part up to the end of that plan's words; 0 when the kernel does not serve the call.
uint64_t ring_ws_bytes(const FusedArgs &a, int dir, bool aligned)
{
  Plan p; RingGeom g;
  return ring_plan_of(a, dir, aligned, p, g) ? p.ws_bytes : 0;
}

// Whether the tiled kernel, which can serve the call, is the faster form.  Not for the residual epilogue on ragged rows below
// these lengths (forward, backward).  The lines were drawn when the kernel read every tile twice, us here and on the plain
// kernel: forward [2123,21,139] 51 and 48, but [998,17,145] 25 and 36; backward [1841,15,165] 60 and 47, [177,77,183] 39 and
// 36, but [966,13,191] 31 and 35.  With tiles in tensor memory it is the faster one below them, too: 41 and 61, 23 and 40; 41
// and 48, 29 and 36, 25 and 36.
constexpr uint32_t kRaggedMinRowExtra[2] = {144, 184};
static bool tiled_preferred(const FusedArgs &a, int dir)
{
  return !(a.res || a.ymask || a.dres) || a.plan.dim0 % 4 == 0 || a.plan.dim0 >= kRaggedMinRowExtra[dir];
}

// Layers of 16-byte aligned rows from which on the tiled kernel is faster than the streaming kernel: it reads a layer once,
// the other one twice, but a tile costs it some 2 us whatever its size.  One line for all rows of 320 floats and more, drawn
// where the shortest of them cross; longer rows cross earlier ([100,128,28,28], 10 M, backward and residual forward / backward:
// streaming kernel 40 and 33 / 50, tiled 29 and 28 / 42).  Forward / backward in us, tiled and streaming:
//   rows of 256   24 M elements 46 / 84 and 49 / 83, 67 M [4096,64,16,16] 107 / 229 and 131 / 228, [512,512,16,16] 105 / 231, 104 / 177
//   rows of 324   10 M 25 / 36 and 21 / 35, 14 M 31 / 48 and 29 / 50, 24 M 45 / 75 and 56 / 78
//   rows of 576   10 M 22 / 30 and 18 / 30, 14 M 26 / 38 and 26 / 43, 24 M 40 / 60 and 43 / 73
//   rows of 784    7 M 19 / 23 and 17 / 24, 10 M 21 / 28 and 22 / 37, 24 M 40 / 56 and 57 / 80
// residual epilogue
//   rows of 256   24 M 76 / 106 and 72 / 99;  324  10 M 32 / 46 and 27 / 46, 14 M 42 / 60 and 40 / 65, 24 M 63 / 94 and 76 / 108
//   rows of 784   10 M 25 / 39 and 29 / 47, 14 M 34 / 53 and 43 / 65
constexpr uint32_t kTiledRow = 320;
constexpr uint64_t kTiledFwd = 18u << 20, kTiledBwd = 12u << 20, kTiledFwdExtra = 12u << 20, kTiledBwdExtra = 11u << 20;
bool tiled_takes(uint32_t dim0, uint64_t elements, int dir, bool extra)
{
  if (dim0 % 4 != 0) return false;
  if (dim0 < kTiledRow) return dir == 0 && !extra && elements >= kTiledFwd + kTiledFwd / 4;
  return elements >= (dir == 0 ? (extra ? kTiledFwdExtra : kTiledFwd) : extra ? kTiledBwdExtra : kTiledBwd);
}

typedef void (*RingKernel)(const FusedArgs, const RingGeom);

static RingKernel pick_ring_kernel(const Plan &p, int dir, bool extra, bool adds, uint32_t &threads)
{
  const bool ragged = p.dim0 % 4 != 0;
  threads = dir == 0 ? ring8::kRingThreads : ring16::kRingThreads;
  if (dir == 0) {
    if (!ring_keeps(p, dir, extra)) return extra ? ring8::bn_ring_kernel<0, true, true, false> : ring8::bn_ring_kernel<0, false, true, false>;
    if (extra) return ragged ? ring8::bn_ring_kernel<0, true, true> : ring8::bn_ring_kernel<0, true, false>;
    return ragged ? ring8::bn_ring_kernel<0, false, true> : ring8::bn_ring_kernel<0, false, false>;
  }
  if (adds) {
    if (extra) return ragged ? ring16::bn_ring_kernel<1, true, true, true, true> : ring16::bn_ring_kernel<1, true, false, true, true>;
    return ragged ? ring16::bn_ring_kernel<1, false, true, true, true> : ring16::bn_ring_kernel<1, false, false, true, true>;
  }
  if (extra) return ragged ? ring16::bn_ring_kernel<1, true, true> : ring16::bn_ring_kernel<1, true, false>;
  return ragged ? ring16::bn_ring_kernel<1, false, true> : ring16::bn_ring_kernel<1, false, false>;
}

int launch_ring(FusedArgs &a, const RingGeom &g_in, int dir, cudaStream_t stream)
{
  RingGeom g = g_in;
  uint32_t threads = 0;
  const bool extra = a.res || a.ymask || a.dres;
  RingKernel k = pick_ring_kernel(a.plan, dir, extra, dir == 1 && a.accumulate, threads);
  // the reduce visits may store dres before the apply visits read x only where it is not x itself
  a.dres_early = a.dres && a.dres != a.x ? 1u : 0u;
  static std::mutex mu;
  static std::map<std::pair<const void *, uint32_t>, int> occ;     // (kernel, smem) -> blocks per SM
  int per_sm = 0;
  // Blocks of kernels that use tensor memory take the SM's whole shared memory: a block of another kernel beside them could
  // hold columns they need, or wait for theirs, and blocks that wait for one another across SMs must not also wait for columns.
  const uint32_t smem = a.mode == MODE_FUSED && ring_keeps(a.plan, dir, extra) ? kRingSmemBudget : g.smem_bytes;
  {
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair((const void *)k, smem);
    auto it = occ.find(key);
    if (it == occ.end()) {
      if (cudaFuncSetAttribute((const void *)k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRingSmemBudget) != cudaSuccess ||
          cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, (int)threads, smem) != cudaSuccess) {
        (void)cudaGetLastError();
        per_sm = 0;
      }
      occ[key] = per_sm;
    } else {
      per_sm = it->second;
    }
  }
  const uint32_t fit = (uint32_t)per_sm * sm_count();
  if (fit == 0) return ANODE_E_LAUNCH;
  if (a.plan.grid > fit) {
    a.plan.grid = fit;
    a.plan.lookahead_steps = ring_lookahead(a.plan, dir);
  }
  a.use_rec = a.mode == MODE_FUSED ? 1u : 0u;
  plan_walk(g, a.plan, ring_pitch(a.plan), ring_warps(dir) * 32);
  g.copies = ceil_div_u32(16 * ring_pitch(a.plan), kRingCopyBytes);
  g.keep_slots = 0; g.keep_period = 1;
  if (a.mode == MODE_FUSED) ring_keep(a.plan, dir, extra, g);
  // A window larger than what L2 keeps would cycle through it whole (config 3, backward: 67 MB); marking only
  // the part that fits lets that part stay (backward 4.42 -> 4.27 ms).  Smaller windows keep everything.
  uint64_t window = ring_window_bytes(a.plan, dir) * (g.keep_period - g.keep_slots) / g.keep_period;
  if (a.ymask && !a.dres_early) window += window / 2;      // x, dy and the saved output come twice
  g.keep_frac = window > kRingLargeWindowMax ? (float)((double)kRingLargeWindowMax / (double)window) : 1.0f;
  void *params[] = {(void *)&a, (void *)&g};
  cudaError_t e;
  if (a.mode == MODE_FUSED)
    e = cudaLaunchCooperativeKernel((const void *)k, dim3(a.plan.grid), dim3(threads), params, smem, stream);
  else
    e = cudaLaunchKernel((const void *)k, dim3(a.plan.grid), dim3(threads), params, smem, stream);
  if (e != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

// The caller's workspace holds two independent parts, one per direction (forward first): a
// direction's kernels keep state in their part from launch to launch (which partial buffer is
// current, words waiting to be cleared), laid out by that direction's own tile plan, so forward
// and backward launches must not share one.  The status word is the first word of the whole.
static void fill_shape_info(ShapeInfo &s)
{
  const Tunables &t = tunables();
  // the plan depends on pointer alignment, which is not known when a workspace is sized: cover both cases
  uint64_t need = 0;
  for (int al = 0; al < 2; ++al) {
    s.plan[al] = make_plan(s.dim0, s.C, s.N, al != 0, sm_count() * t.blocks_per_sm, t.tile_floats, 1);
    if (s.plan[al].ws_bytes > need) need = s.plan[al].ws_bytes;
  }
  for (int dir = 0; dir < 2; ++dir)
    for (int ex = 0; ex < 2; ++ex)
      s.ring_ok[dir][ex] = make_ring_plan(s.dim0, s.C, s.N, dir, ex != 0, s.ring_plan[dir][ex], s.ring_geom[dir][ex]);
  const bool ragged = s.dim0 % 4 != 0;
  if (!ragged)
    for (int dir = 0; dir < 2; ++dir)
      if (s.ring_ok[dir][0] && s.ring_plan[dir][0].ws_bytes > need) need = s.ring_plan[dir][0].ws_bytes;
  s.tiled_bytes = align_up_u64(need, 256);
  s.static_bytes = align_up_u64(s.tiled_bytes + resident_ws_bytes(s.dim0, s.C, s.N), 256);
  // The tiled kernel keeps tagged words from launch to launch, laid out by its plan.  Ragged rows and the residual
  // epilogue have plans of their own beside the plain kernel's and the ordinary call's on the same workspace, so their
  // words (and their two header words) lie apart, behind everything else.
  s.part_bytes = s.static_bytes;
  for (int dir = 0; dir < 2; ++dir)
    for (int ex = 0; ex < 2; ++ex) {
      if (!s.ring_ok[dir][ex] || (!ex && !ragged)) continue;
      Plan &p = s.ring_plan[dir][ex];
      // the fused form of this kernel uses the tagged words only
      uint64_t off = s.static_bytes;
      if (ex && ragged && s.ring_ok[dir][0]) off = align_up_u64(s.ring_plan[dir][0].ws_bytes, 256);
      const uint64_t end = align_up_u64(off + 16ull * p.total_tiles * p.cb, 256);
      if (end > 0xffffffffull) { s.ring_ok[dir][ex] = false; continue; }
      p.off_tag = (uint32_t)off; p.off_part = (uint32_t)end; p.ws_bytes = end;
      s.ring_geom[dir][ex].hdr = ex ? kRingHdrExtra : kRingHdrRagged;
      if (end > s.part_bytes) s.part_bytes = end;
    }
  // so does the band kernel; a part serves one direction, so both directions' words may begin at the same place
  const uint64_t bands = s.part_bytes;
  for (int dir = 0; dir < 2; ++dir) {
    uint64_t at = bands;
    for (int ex = 0; ex < 2; ++ex) {
      BandGeom &g = s.band[dir][ex];
      s.band_ok[dir][ex] = band_plan(s.dim0, s.C, s.N, dir, ex != 0, g);
      if (!s.band_ok[dir][ex]) continue;
      g.hdr = ex ? kBandHdrExtra : kBandHdr;
      const uint64_t end = align_up_u64(at + band_words(g) * 2 * kBandWordBytes, 256);
      if (end > 0xffffffffull) { s.band_ok[dir][ex] = false; continue; }
      g.tag = (uint32_t)at;
      at = end;
    }
    if (at > s.part_bytes) s.part_bytes = at;
  }
  for (int dir = 0; dir < 2; ++dir)
    for (int ex = 0; ex < 2; ++ex) s.stream_ok[dir][ex] = s.masked_ok[dir][ex] = s.long_ok[dir][ex] = 0;
}

bool stream_geom_of(const FusedArgs &a, int dir, StreamGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  const ShapeInfo &s = shape_info(a.plan.dim0, a.plan.C, a.plan.N);
  uint8_t &ok = s.stream_ok[dir][extra];
  if (!ok) ok = stream_plan(s.dim0, s.C, s.N, dir, extra, s.stream[dir][extra]) ? 2 : 1;
  if (ok == 2) g = s.stream[dir][extra];
  return ok == 2;
}

bool masked_geom_of(const FusedArgs &a, int dir, StreamGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  if (a.mode != MODE_FUSED || a.world > 1) return false;
  const ShapeInfo &s = shape_info(a.plan.dim0, a.plan.C, a.plan.N);
  uint8_t &ok = s.masked_ok[dir][extra];
  if (!ok) ok = masked_plan(s.dim0, s.C, s.N, dir, extra, s.stream[dir][extra]) ? 2 : 1;
  if (ok == 2) g = s.stream[dir][extra];
  return ok == 2;
}

bool band_geom_of(const FusedArgs &a, int dir, BandGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  const ShapeInfo &s = shape_info(a.plan.dim0, a.plan.C, a.plan.N);
  if (!s.band_ok[dir][extra]) return false;
  g = s.band[dir][extra];
  return a.bands && a.ws_capacity >= g.tag + band_words(g) * 2 * kBandWordBytes;
}

bool long_geom_of(const FusedArgs &a, int dir, LongGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  if (a.mode != MODE_FUSED || a.world > 1) return false;
  const ShapeInfo &s = shape_info(a.plan.dim0, a.plan.C, a.plan.N);
  uint8_t &ok = s.long_ok[dir][extra];
  if (!ok) ok = long_plan(s.dim0, s.C, s.N, dir, extra, s.long_rows[dir][extra]) ? 2 : 1;
  if (ok == 2) g = s.long_rows[dir][extra];
  return ok == 2;
}

// Bytes of a part taken by the tile-plan kernels (plain, warp-specialised, cluster); the records of the
// slice-resident kernel follow behind them.
static uint64_t tiled_part_bytes(uint32_t dim0, uint32_t C, uint32_t N) { return shape_info(dim0, C, N).tiled_bytes; }

uint64_t workspace_part_bytes(uint32_t dim0, uint32_t C, uint32_t N) { return shape_info(dim0, C, N).part_bytes; }

// Bytes of a part behind which only the ragged and the residual plans of the tiled kernel keep their words.
uint64_t workspace_static_bytes(uint32_t dim0, uint32_t C, uint32_t N) { return shape_info(dim0, C, N).static_bytes; }

// Bytes at the start of a workspace that hold progress counters, flags and records, i.e. what has
// to be zero when a launch begins (the per-tile partials behind them are written before they are read).
uint64_t control_region_bytes(uint32_t dim0, uint32_t C, uint32_t N, bool aligned)
{
  uint64_t n = plan_for(dim0, C, N, aligned).off_part;
  for (int dir = 0; dir < 2; ++dir) {
    Plan rp; RingGeom g;
    if (ring_plan_for(dim0, C, N, aligned, dir, false, rp, g) && rp.off_part > n) n = rp.off_part;
  }
  // the slice-resident kernel's records validate themselves against the launch counter in the header,
  // which the clearing resets: they have to go too
  if (aligned && resident_ws_bytes(dim0, C, N)) { const uint64_t r = workspace_static_bytes(dim0, C, N); if (r > n) n = r; }
  return n;
}

// Which kernel launch_best takes for a prepared call: ANODE_KERNEL_* (never AUTO), or -1 when none can
// (a synchronized call in fused mode on a shape only the plain kernel takes: it has no exchange).
int pick_kernel_kind(const FusedArgs &a, int dir, bool aligned)
{
  const bool extra = a.res || a.ymask || a.dres;        // residual epilogue
  const bool plain_ok = !(a.mode == MODE_FUSED && a.world > 1);
  StreamGeom mg;
  const bool tiled_ok = ring_serves(a, dir, aligned) && (kernel_choice() != ANODE_KERNEL_AUTO || tiled_preferred(a, dir));
  switch (kernel_choice()) {
    case ANODE_KERNEL_TILED: if (tiled_ok) return ANODE_KERNEL_TILED; break;
    case ANODE_KERNEL_CLUSTER: if (segres_applies(a, dir, aligned)) return ANODE_KERNEL_CLUSTER; break;
    case ANODE_KERNEL_RESIDENT: if (resident_applies(a, dir, aligned)) return ANODE_KERNEL_RESIDENT; break;
    case ANODE_KERNEL_PLAIN: if (plain_ok) return ANODE_KERNEL_PLAIN; break;
    case ANODE_KERNEL_REGISTER: if (chan_applies(a, dir, aligned)) return ANODE_KERNEL_REGISTER; break;
    case ANODE_KERNEL_STREAM: if (stream_applies(a, dir, aligned) || (aligned && masked_geom_of(a, dir, mg))) return ANODE_KERNEL_STREAM; break;
    case ANODE_KERNEL_BAND: { BandGeom bg; if (stream_applies(a, dir, aligned) && band_geom_of(a, dir, bg)) return ANODE_KERNEL_STREAM; break; }
    default:
      if (chan_preferred(a, dir, aligned, tiled_ok)) return ANODE_KERNEL_REGISTER;
      if (stream_preferred(a, dir, aligned, tiled_ok)) return ANODE_KERNEL_STREAM;
      break;
  }
  if (extra) {
    // long rows: the tiled kernel on one GPU (forward / backward: [256,512,28,28] 263 / 452 us, cluster kernel 383 / too
    // large for it, plain kernel 315 / 618; [256,64,56,56] 136 / 188 us, plain kernel 152 / 303); short ones the cluster
    // kernel, and in synchronized calls what has the exchange inside
    if (tiled_ok) return ANODE_KERNEL_TILED;
    if (segres_applies(a, dir, aligned)) return ANODE_KERNEL_CLUSTER;
    if (plain_ok) return ANODE_KERNEL_PLAIN;
    return resident_applies(a, dir, aligned) ? ANODE_KERNEL_RESIDENT : -1;
  }
  // short rows, and in synchronized calls channels small enough to sit in a few blocks' shared memory: the cluster
  // kernel (on one GPU the register-resident kernel has those, and of large layers the tiled kernel is the faster one:
  // [128,512,28,28] forward 87 us, 105 us on the cluster kernel)
  if (segres_preferred(a, dir, aligned) && !(tiled_ok && a.world <= 1 && kernel_choice() == ANODE_KERNEL_AUTO)) return ANODE_KERNEL_CLUSTER;
  if (tiled_ok) return ANODE_KERNEL_TILED;
  if (segres_applies(a, dir, aligned)) return ANODE_KERNEL_CLUSTER;
  if (plain_ok) return ANODE_KERNEL_PLAIN;
  return resident_applies(a, dir, aligned) ? ANODE_KERNEL_RESIDENT : -1;
}

// Us of the kernels that the two below take calls from.  The tiled kernel: its launch and agreement, the layer's bytes, and of ragged rows a
// copy for each and tensor; seven per cent off over 968 passes of 0.2 to 46 M elements, from memory.  The plain kernel: its agreement, 1.75 to
// 2 TB/s, and what a row's ends cost; 15 per cent off over 438 passes of 0.4 to 150 M elements.  From 256 floats a row on it takes them one by
// one: 18 per cent off over 260 passes of 0.3 to 40 M elements.
static float takes_from_us(const FusedArgs &a, int dir, bool extra, int kind)
{
  const float rows = (float)a.plan.C * (float)a.plan.N, bytes = 4.0f * rows * (float)a.plan.dim0 * (dir == 0 ? (extra ? 3.0f : 2.0f) : extra ? 5.0f : 3.0f);
  if (kind == ANODE_KERNEL_PLAIN && a.plan.dim0 >= 256) return dir == 0 ? 21.0f + bytes * 3.6e-7f + rows * 1e-3f : 17.0f + bytes * 3.6e-7f + rows * 2e-3f;
  if (kind == ANODE_KERNEL_PLAIN) return dir == 0 ? 13.0f + bytes * 5.7e-7f + rows * 4e-5f : 10.0f + bytes * 5e-7f + rows * 4e-5f;
  return 11.0f + bytes * 1.35e-7f + (a.plan.dim0 % 4 == 0 ? 0.0f : rows * (dir == 1 ? 5e-4f : extra ? 4.3e-4f : 2.2e-4f));
}

// Odd rows, on one GPU: where the streaming kernel, or its masked form for rows without an aligned run of channels, is launched in the
// place of the kernel that pick_kernel_kind names.  Us there and here, forward, backward, residual forward and backward:
//  - the register-resident kernel, which loads such rows float by float, from these sizes and twenty samples on.  Masked: [270,490,49]
//    22.9, 34.9, 34.8, 61.1 and 15.8, 22.6, 19.6, 30.1, [356,2022,25] 59, 84, 85, 157 and 35, 56, 46, 80; but [67,706,37], 1.75 M, 5.2, 8.1, 7.6,
//    15.7 and 6.6, 8.9, 8.4, 10.2, [802,67,19], 1.0 M, 4.5, 5.5, 5.0, 7.2 and 6.6, 8.1, 7.8, 9.3, and few samples, [16,2017,151] 17.5, 22.2,
//    22.6, 39.7 and 22.4, 23.8, 25.1, 32.9.  Aligned runs: [188,356,39], 2.6 M, 11.5, 11.1, 14.8, 31.7 and 6.3, 9.1, 8.3, 12.0, [2604,86,14]
//    12.8, 16.3, 19.4, 36.0 and 11.0, 15.0, 13.2, 21.1, but [2311,68,14], 2.2 M, 6.7, 9.8, 10.6, 20.6 and 8.4, 10.1, 9.6,
//    13.2, and forward [30,298,258], 2.3 M, 7.3 and 7.9;
//  - the plain and the tiled kernel (which copies a row at a time), masked, where its estimate with these margins is below theirs
//    (takes_from_us): clusters of few channels leave the device empty and walk their samples for long.  Plain: figures at the head of
//    bn_stream.cu, but [97106,1,81] forward 57 and 144, [93078,1,146] backward 92 and 575, [130265,1,47] residual forward 61 and 254,
//    [154066,1,113] residual backward 151 and 972; of 452 such passes 326 are taken, 0.62 of the time, nine of them slower by more than a
//    twentieth (with margins of 1.3, 1.15, 1.1 and 1.1 [4096,3,7,7] backward was left out, 17.9 and 13.2; with a tenth less three are slower by
//    1.2 to 1.3), and what is left out would take 1.89 times as long here.  Tiled: [604,18,221] 16.4, 20.5, 18.5, 25.6 and 9.3, 11.7, 10.6, 14.8,
//    [1826,159,179] 128, 246, 213, - and 118, 186, 153, -, [1403,355,131] forward 191 and 143, [947,13,350] forward 19.5 and 13.3, residual forward 22.6
//    and 20.1; but [110600,1,165] forward 63 and 496, [2705,2,818] backward 21.9 and 96.9, residual forward 17.9 and 88.1.  On rows of 200 floats and
//    more only in small layers, where the tiled kernel's launch costs ten us: [1594,54,227] 54, 81, 77, 101 and 58, 80, 69, 107, [2147,15,254], 8.2 M, 27.5,
//    42.0, 39.0, 49.4 and 29.2, 46.1, 42.6, 63.5.
constexpr uint32_t kMaskedSamples = 20, kMaskedShortRow = 200;
constexpr uint64_t kMaskedChan[2][2] = {{2500000, 2100000}, {2300000, 1100000}};        // [direction][residual]
constexpr uint64_t kMaskedTiled[2][2] = {{8000000, 5000000}, {4500000, 2500000}};
constexpr float kMaskedMargin[2][2] = {{1.2f, 1.05f}, {1.05f, 1.05f}};
static bool masked_takes(const FusedArgs &a, int dir, int kind, StreamGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  const uint64_t elements = (uint64_t)a.plan.dim0 * a.plan.C * a.plan.N;
  if (a.plan.dim0 % 4 == 0) return false;
  if (kind == ANODE_KERNEL_REGISTER)
    return a.plan.N >= kMaskedSamples && elements >= kMaskedChan[dir][extra] && (stream_geom_of(a, dir, g) || masked_geom_of(a, dir, g));
  if (kind == ANODE_KERNEL_TILED && a.plan.dim0 >= kMaskedShortRow && (a.plan.N < kMaskedSamples || elements > kMaskedTiled[dir][extra])) return false;
  return masked_geom_of(a, dir, g) && g.cost * kMaskedMargin[dir][extra] < takes_from_us(a, dir, extra, kind);
}

// Rows of 250 floats and more, on one GPU: where the kernel for long rows (bn_long.cu) is launched in the place of the one that
// pick_kernel_kind names.  Us there and here, forward, backward, residual forward and backward:
//  - the tiled kernel where its time (takes_from_us), with what kLongAhead adds, is more than the estimate of the other: [1,3,64,64,64] 12.5,
//    12.4, -, - and 6.0, 7.9, -, -, [1,11,99716] -, 13.8, 13.2, 13.0 and -, 7.2, 6.7, 9.2; but [1,4,1630016], 6.5 M, 19.4, 25.2, 22.3, 31.8 and
//    28.6, 47.6, 47.3, 58.0, [392,12,1225] residual forward 19.7 and 27.7, [33,25,6426] backward 23.1 and 27.9.
//    kLongAhead is from forward and backward passes of a layer in turn on a stream, where a forward pass on the tiled kernel costs more than
//    the same pass over and over ([32,42,7480], forward and backward, 48.8 us, forward here 44.7; over the 351 of 8000 such pairs for which
//    these rules and those without estimates of the other kernels launch something else, 0.87 of the time, and 0.86 of that without this kernel);
//  - the register-resident kernel on ragged rows, which it loads float by float, from these sizes or channels on: [8,217,2678] 18.5, 29.8,
//    30.9, 52.6 and 12.7, 16.1, 14.5, 20.6, [2,5,19011] 3.8, 5.2, 5.2, 6.9 and 5.1, 4.1, 4.5, 4.6, [9,4,12887] forward 8.1 and 5.5, but
//    [10,119,1502], 1.8 M, 5.4, 8.5, 8.0 and 7.9, 10.0, 9.8, and where the clusters take a second wave, [71,25,577] backward 7.1 and 8.9,
//    [3,1023,366] residual backward 8.0 and 11.3; in three waves and more what each block walks has to make up for them (kLongManyWaves),
//    [4,2048,435] 12.4, 16.1, 16.4 and 27.4, 21.6, 24.8, [1,1024,8190] forward 24.6 and 26.4, but [1,923,8710] 28.3 and 25.9 (the lines are from
//    forward and backward in turn: [2,2048,1078] 38.7 and 49.9, [3,1926,1381] 61.4 and 61.1, [5,1173,999] 45.0 and 42.4, [3,1199,2091] 52.7 and 45.9);
//  - and the same on aligned ones in the residual epilogue, where one block or two hold a channel: [35,183,1292], 8.3 M, 28.3, 40.8 and
//    23.6, 35.8, [82,110,440], 4.0 M, 14.8, 21.1 and 13.6, 18.5, [7,331,1108], 2.6 M, backward 12.9 and 10.5; but forward [12,316,1032],
//    3.9 M, 13.2 and 15.2, [18,380,464], 3.2 M, 10.5 and 12.0, and more channels, [2,512,4096] 10.8, 16.0 and 11.4, 19.4, [11,1404,420]
//    15.6, 25.6 and 22.5, 28.7.
constexpr uint32_t kLongRow = 250, kLongFewChannels = 128, kLongOneWave = 20;
constexpr float kLongAhead[2][2][2] = {{{1.5f, 3.0f}, {1.0f, -1.0f}}, {{-1.5f, -0.5f}, {1.0f, 0.5f}}};      // us: [direction][residual][ragged]
constexpr uint64_t kLongManyWaves[2][2] = {{4250, 2850}, {2000, 0}};                   // floats of a channel: [direction][residual]
constexpr uint64_t kLongTiledMost = 12000000;
constexpr uint64_t kLongManyChannels = 2400000;
constexpr uint32_t kLongChannelsAligned = 450;
constexpr uint64_t kLongChan[2][2] = {{3300000, 1800000}, {1800000, 700000}};           // [direction][residual]
constexpr uint64_t kLongChannel[2][2] = {{64 << 10, 32 << 10}, {32 << 10, 24 << 10}};
constexpr uint64_t kLongChanAligned[2][2] = {{~0ull, 3950000}, {~0ull, 2400000}};
static bool long_takes(const FusedArgs &a, int dir, int kind, LongGeom &g)
{
  const bool extra = (dir == 0 ? a.res : a.ymask) != nullptr;
  const uint64_t channel = (uint64_t)a.plan.dim0 * a.plan.N, elements = channel * a.plan.C;
  if (a.plan.dim0 < kLongRow) return false;
  if (kind == ANODE_KERNEL_TILED)
    return elements <= kLongTiledMost && long_geom_of(a, dir, g) && g.cost < takes_from_us(a, dir, extra, kind) + kLongAhead[dir][extra][a.plan.dim0 % 4 != 0];
  if (kind != ANODE_KERNEL_REGISTER) return false;
  const uint32_t C = a.plan.C;
  if (a.plan.dim0 % 4 != 0 && C > 2 * kLongBlocks * sm_count() && channel < kLongManyWaves[dir][extra]) return false;
  return (a.plan.dim0 % 4 == 0 ? elements >= kLongChanAligned[dir][extra] && C <= kLongChannelsAligned
                               : (elements >= kLongChan[dir][extra] && (C <= kLongFewChannels || elements >= kLongManyChannels)) ||
                                     (channel >= kLongChannel[dir][extra] && C <= kLongOneWave)) && long_geom_of(a, dir, g);
}

// Which of those two takes the call from `kind`: STREAM, LONG (and its geometry), or -1.  Where both do, the one of the smaller estimate.
static int pick_instead(const FusedArgs &a, int dir, int kind, bool aligned, LongGeom &lg)
{
  if (!aligned || a.mode != MODE_FUSED || a.world > 1 ||
      (kind != ANODE_KERNEL_REGISTER && kind != ANODE_KERNEL_TILED && kind != ANODE_KERNEL_PLAIN)) return -1;
  const int choice = kernel_choice();
  if (choice != ANODE_KERNEL_AUTO) return choice == ANODE_KERNEL_LONG && long_geom_of(a, dir, lg) ? ANODE_KERNEL_LONG : -1;
  StreamGeom sg;
  const bool masked = masked_takes(a, dir, kind, sg), rows = long_takes(a, dir, kind, lg);
  if (masked && rows) return lg.cost < sg.cost ? ANODE_KERNEL_LONG : ANODE_KERNEL_STREAM;
  return masked ? ANODE_KERNEL_STREAM : rows ? ANODE_KERNEL_LONG : -1;
}

// Launches it; -1 where there is none, or the device refuses its clusters.
static int launch_instead(FusedArgs &a, int dir, int kind, bool aligned, cudaStream_t stream)
{
  LongGeom lg;
  const int k = pick_instead(a, dir, kind, aligned, lg);
  if (k == ANODE_KERNEL_STREAM && launch_stream(a, dir, stream) == ANODE_OK) return k;
  if (k == ANODE_KERNEL_LONG && launch_long(a, lg, dir, stream) == ANODE_OK) return k;
  return -1;
}

static thread_local int t_last_kernel = -1;

// Launches direction `dir` of a prepared call with the kernel pick_kernel_kind names.  A cluster launch
// the device refuses falls back to the next kernel that applies.
int launch_best(FusedArgs &a, int dir, bool aligned, cudaStream_t stream)
{
  int kind = pick_kernel_kind(a, dir, aligned);
  auto launched = [&](int k, int rc) { if (rc == ANODE_OK) t_last_kernel = k; return rc; };
  const int instead = launch_instead(a, dir, kind, aligned, stream);
  if (instead >= 0) return launched(instead, ANODE_OK);
  if (kind == ANODE_KERNEL_REGISTER) return launched(kind, launch_chan(a, dir, aligned, stream));
  if (kind == ANODE_KERNEL_STREAM) {
    BandGeom bg;
    if (kernel_choice() != ANODE_KERNEL_STREAM && band_geom_of(a, dir, bg) &&
        launched(ANODE_KERNEL_BAND, launch_band(a, bg, dir, stream)) == ANODE_OK) return ANODE_OK;
    if (launched(kind, launch_stream(a, dir, stream)) == ANODE_OK) return ANODE_OK;
    kind = segres_applies(a, dir, aligned) ? ANODE_KERNEL_CLUSTER : ANODE_KERNEL_PLAIN;
  }
  if (kind == ANODE_KERNEL_CLUSTER) {
    if (launched(kind, launch_segres(a, dir, stream)) == ANODE_OK) return ANODE_OK;
    Plan rp; RingGeom g;
    if (ring_plan_of(a, dir, aligned, rp, g)) kind = ANODE_KERNEL_TILED;
    else if (resident_applies(a, dir, aligned)) kind = ANODE_KERNEL_RESIDENT;
    else kind = (a.mode == MODE_FUSED && a.world > 1) ? -1 : ANODE_KERNEL_PLAIN;
  }
  if (kind == ANODE_KERNEL_TILED) {
    Plan rp; RingGeom g;
    if (!ring_plan_of(a, dir, aligned, rp, g)) return ANODE_E_LAUNCH;
    a.plan = rp;
    return launched(kind, launch_ring(a, g, dir, stream));
  }
  if (kind == ANODE_KERNEL_RESIDENT) return launched(kind, launch_resident(a, dir, tiled_part_bytes(a.plan.dim0, a.plan.C, a.plan.N), stream));
  if (kind == ANODE_KERNEL_PLAIN) return launched(kind, launch_pipeline(a, dir, stream));
  return ANODE_E_LAUNCH;
}

int check_dims(uint32_t dim0, uint32_t dim1, uint32_t dim2)
{
  if (dim0 == 0 || dim1 == 0 || dim2 == 0) return ANODE_E_DIMS;
  const unsigned __int128 len = (unsigned __int128)dim0 * dim1 * dim2;
  if (len >= ((unsigned __int128)1 << 32)) return ANODE_E_DIMS;
  return ANODE_OK;
}

typedef void (*PipelineKernel)(const FusedArgs);

static PipelineKernel pick_kernel(const Plan &p, int dir)
{
  if (p.regime == 1) return dir == 0 ? bn_pipeline_kernel<4, 0, 1> : bn_pipeline_kernel<4, 1, 1>;
  if (p.vec == 4) return dir == 0 ? bn_pipeline_kernel<4, 0, 0> : bn_pipeline_kernel<4, 1, 0>;
  return dir == 0 ? bn_pipeline_kernel<1, 0, 0> : bn_pipeline_kernel<1, 1, 0>;
}

// Blocks of `k` that fit on one SM (cached per kernel; same answer on every B200).
static uint32_t blocks_per_sm(PipelineKernel k)
{
  static std::mutex mu;
  static std::map<const void *, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  auto it = cache.find((const void *)k);
  if (it != cache.end()) return (uint32_t)it->second;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, (int)kThreads, 0) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
  cache[(const void *)k] = n;
  return (uint32_t)n;
}

int launch_pipeline(FusedArgs &a, int dir, cudaStream_t stream)
{
  PipelineKernel k = pick_kernel(a.plan, dir);
  const uint32_t fit = blocks_per_sm(k) * sm_count();
  if (fit == 0) return ANODE_E_LAUNCH;
  if (a.plan.grid > fit) {
    // fewer blocks are resident than planned: shrink the grid and re-derive the lookahead
    a.plan.grid = fit;
    a.plan.lookahead_steps = ceil_div_u32(a.plan.tiles_per_unit, a.plan.grid) + 1;
  }
  void *params[] = {(void *)&a};
  cudaError_t e;
  if (a.mode == MODE_FUSED) {
    // Blocks wait on one another's results, so all of them must be resident: a cooperative
    // launch fails instead of deadlocking when they would not be.
    e = cudaLaunchCooperativeKernel((const void *)k, dim3(a.plan.grid), dim3(kThreads), params, 0, stream);
  } else {
    e = cudaLaunchKernel((const void *)k, dim3(a.plan.grid), dim3(kThreads), params, 0, stream);
  }
  if (e != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
bool aligned4(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 3u) == 0; }

int prepare_fwd(FusedArgs &a, uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate,
                int relu, const float *x, const float *gamma, const float *beta, float *y, float *mean,
                float *var, float *run_mean, float *run_var, void *ws, size_t ws_bytes)
{
  const int rc = check_dims(dim0, dim1, dim2);
  if (rc) return rc;
  if (!x || !y || !mean || !var) return ANODE_E_NULL;
  if (!aligned4(x) || !aligned4(y)) return ANODE_E_ALIGN;
  if (!ws || !aligned16(ws)) return ANODE_E_WORKSPACE;
  a = FusedArgs{};
  const ShapeInfo &shape = shape_info(dim0, dim1, dim2);
  a.plan = shape.plan[aligned16(x) && aligned16(y) ? 1 : 0];
  const uint64_t part = shape.part_bytes;
  if (ws_bytes < part) return ANODE_E_WORKSPACE;              // forward uses the first part only
  a.ws_capacity = part;
  a.status = static_cast<uint32_t *>(ws);
  a.x = x; a.gamma = gamma; a.beta = beta; a.out = y;
  a.mean = mean; a.var = var; a.run_mean = run_mean; a.run_var = run_var;
  a.ws = static_cast<unsigned char *>(ws);
  a.epsilon = epsilon; a.avg_rate = avg_rate; a.relu = relu ? 1u : 0u; a.neg_slope = relu ? 0.0f : 1.0f;
  a.mode = MODE_FUSED;
  a.count_total = (double)dim0 * (double)dim2;
  a.wait_cycles = wait_limit_cycles();
  a.bands = 1u;
  return ANODE_OK;
}

int prepare_bwd(FusedArgs &a, uint32_t dim0, uint32_t dim1, uint32_t dim2, int relu, int accumulate,
                const float *dy, const float *x, const float *mean, const float *var, const float *gamma,
                const float *beta, float *dx, float *dgamma, float *dbeta, void *ws, size_t ws_bytes)
{
  const int rc = check_dims(dim0, dim1, dim2);
  if (rc) return rc;
  if (!x || !dy || !dx || !mean || !var) return ANODE_E_NULL;
  if (!aligned4(x) || !aligned4(dy) || !aligned4(dx)) return ANODE_E_ALIGN;
  if (!ws || !aligned16(ws)) return ANODE_E_WORKSPACE;
  a = FusedArgs{};
  const ShapeInfo &shape = shape_info(dim0, dim1, dim2);
  a.plan = shape.plan[aligned16(x) && aligned16(dy) && aligned16(dx) ? 1 : 0];
  const uint64_t part = shape.part_bytes;
  if (ws_bytes < 2 * part) return ANODE_E_WORKSPACE;
  a.ws_capacity = part;
  a.status = static_cast<uint32_t *>(ws);
  a.x = x; a.dy = dy; a.gamma = gamma; a.beta = beta; a.mean_in = mean; a.var_in = var;
  a.out = dx; a.dgamma = dgamma; a.dbeta = dbeta;
  a.ws = static_cast<unsigned char *>(ws) + part;              // the backward part
  a.relu = relu ? 1u : 0u; a.neg_slope = relu ? 0.0f : 1.0f; a.accumulate = accumulate ? 1u : 0u;
  a.mode = MODE_FUSED;
  a.count_total = (double)dim0 * (double)dim2;
  a.wait_cycles = wait_limit_cycles();
  a.bands = 1u;
  return ANODE_OK;
}

__global__ void online_average_kernel(uint32_t len, float rate, const float *x, float *y)
{
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < len; i += gridDim.x * blockDim.x) {
    const float o = y[i];
    y[i] = o + rate * (x[i] - o);
  }
}

}  // namespace anode_b200

using namespace anode_b200;

extern "C" size_t anode_gpu_batch_norm_fused_workspace_bytes(uint32_t dim0, uint32_t dim1, uint32_t dim2)
{
  if (check_dims(dim0, dim1, dim2)) return 0;
  return (size_t)(2 * workspace_part_bytes(dim0, dim1, dim2));
}

extern "C" int anode_gpu_batch_norm_fused_workspace_init(void *workspace, size_t bytes, struct CUstream_st *stream)
{
  if (!workspace) return ANODE_E_NULL;
  if (cudaMemsetAsync(workspace, 0, bytes, stream) != cudaSuccess) { (void)cudaGetLastError(); return ANODE_E_LAUNCH; }
  return ANODE_OK;
}

extern "C" int anode_gpu_batch_norm_fused_status(const void *workspace, struct CUstream_st *stream, uint32_t *status)
{
  if (!workspace || !status) return ANODE_E_NULL;
  if (cudaMemcpyAsync(status, workspace, sizeof(uint32_t), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess) {
    (void)cudaGetLastError();
    return ANODE_E_LAUNCH;
  }
  return ANODE_OK;
}

extern "C" int anode_gpu_batch_norm_relu_fused_fwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate, int relu,
    const float *x, const float *gamma, const float *beta,
    float *y, float *mean, float *var, float *run_mean, float *run_var,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  FusedArgs a;
  const int rc = prepare_fwd(a, dim0, dim1, dim2, epsilon, avg_rate, relu, x, gamma, beta, y, mean, var,
                             run_mean, run_var, workspace, workspace_bytes);
  if (rc) return rc;
  if (workspace_bytes < 2 * a.ws_capacity) return ANODE_E_WORKSPACE;
  return launch_best(a, 0, aligned16(x) && aligned16(y), stream);
}

extern "C" int anode_gpu_batch_norm_relu_fused_bwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, int relu, int accumulate,
    const float *dy, const float *x, const float *mean, const float *var,
    const float *gamma, const float *beta, float *dx, float *dgamma, float *dbeta,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  FusedArgs a;
  const int rc = prepare_bwd(a, dim0, dim1, dim2, relu, accumulate, dy, x, mean, var, gamma, beta, dx,
                             dgamma, dbeta, workspace, workspace_bytes);
  if (rc) return rc;
  return launch_best(a, 1, aligned16(x) && aligned16(dy) && aligned16(dx), stream);
}

// The two calls above with a general activation t*(t > 0 ? 1 : neg_slope) instead of the ReLU switch.
extern "C" int anode_gpu_batch_norm_act_fused_fwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate, float neg_slope,
    const float *x, const float *gamma, const float *beta,
    float *y, float *mean, float *var, float *run_mean, float *run_var,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  FusedArgs a;
  const int rc = prepare_fwd(a, dim0, dim1, dim2, epsilon, avg_rate, 1, x, gamma, beta, y, mean, var,
                             run_mean, run_var, workspace, workspace_bytes);
  if (rc) return rc;
  if (workspace_bytes < 2 * a.ws_capacity) return ANODE_E_WORKSPACE;
  a.neg_slope = neg_slope;
  return launch_best(a, 0, aligned16(x) && aligned16(y), stream);
}

extern "C" int anode_gpu_batch_norm_act_fused_bwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float neg_slope, int accumulate,
    const float *dy, const float *x, const float *mean, const float *var,
    const float *gamma, const float *beta, float *dx, float *dgamma, float *dbeta,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  FusedArgs a;
  const int rc = prepare_bwd(a, dim0, dim1, dim2, 1, accumulate, dy, x, mean, var, gamma, beta, dx,
                             dgamma, dbeta, workspace, workspace_bytes);
  if (rc) return rc;
  a.neg_slope = neg_slope;
  return launch_best(a, 1, aligned16(x) && aligned16(dy) && aligned16(dx), stream);
}

// Residual block epilogue: y = act(bn(x) + residual), the step after batch-norm in every residual
// block (examples/run_imagenet_mpi.rs:191-195, 224-226: sum of the shortcut and the normalized
// branch, then positive_clip).  Backward: the mask comes from the saved output y (as the reference's
// positive_clip adjoint takes it, flat_map.cu:187-194), dresidual = dy*mask is the gradient of the
// shortcut (the sum's adjoint fans dz out to both inputs), dx / dgamma / dbeta as before.
extern "C" int anode_gpu_batch_norm_add_act_fused_fwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float epsilon, float avg_rate, float neg_slope,
    const float *x, const float *residual, const float *gamma, const float *beta,
    float *y, float *mean, float *var, float *run_mean, float *run_var,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  if (!residual) return ANODE_E_NULL;
  if (!aligned4(residual)) return ANODE_E_ALIGN;
  FusedArgs a;
  const int rc = prepare_fwd(a, dim0, dim1, dim2, epsilon, avg_rate, 1, x, gamma, beta, y, mean, var,
                             run_mean, run_var, workspace, workspace_bytes);
  if (rc) return rc;
  if (workspace_bytes < 2 * a.ws_capacity) return ANODE_E_WORKSPACE;
  a.neg_slope = neg_slope;
  a.res = residual;
  if (!aligned16(residual)) a.plan = plan_for(dim0, dim1, dim2, false);      // scalar path
  return launch_best(a, 0, aligned16(x) && aligned16(y) && aligned16(residual), stream);
}

extern "C" int anode_gpu_batch_norm_add_act_fused_bwd_3d1_packed_f32(
    uint32_t dim0, uint32_t dim1, uint32_t dim2, float neg_slope, int accumulate,
    const float *dy, const float *x, const float *y, const float *mean, const float *var,
    const float *gamma, const float *beta, float *dx, float *dresidual, float *dgamma, float *dbeta,
    void *workspace, size_t workspace_bytes, const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  if (!y) return ANODE_E_NULL;
  if (!aligned4(y) || (dresidual && !aligned4(dresidual))) return ANODE_E_ALIGN;
  FusedArgs a;
  const int rc = prepare_bwd(a, dim0, dim1, dim2, 1, accumulate, dy, x, mean, var, gamma, beta, dx,
                             dgamma, dbeta, workspace, workspace_bytes);
  if (rc) return rc;
  a.neg_slope = neg_slope;
  a.ymask = y; a.dres = dresidual;
  const bool al = aligned16(x) && aligned16(dy) && aligned16(dx) && aligned16(y) && (!dresidual || aligned16(dresidual));
  if (!al) a.plan = plan_for(dim0, dim1, dim2, false);
  return launch_best(a, 1, al, stream);
}

extern "C" int anode_gpu_online_average_f32(uint32_t len, float rate, const float *x, float *y,
                                            const struct KernelConfig *cfg, struct CUstream_st *stream)
{
  (void)cfg;
  if (!x || !y) return ANODE_E_NULL;
  if (len == 0) return ANODE_OK;
  const uint32_t blocks = (len + 255) / 256 < 1184 ? (len + 255) / 256 : 1184;
  online_average_kernel<<<blocks, 256, 0, stream>>>(len, rate, x, y);
  if (cudaGetLastError() != cudaSuccess) return ANODE_E_LAUNCH;
  return ANODE_OK;
}

// A call of this form with a workspace of the full size, as far as the choice of the kernel looks at it.
static FusedArgs probe_call(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool residual, bool aligned, int world)
{
  static const float dummy = 0.f;
  FusedArgs a{};
  a.plan = plan_for(dim0, C, N, aligned);
  a.mode = MODE_FUSED;
  a.world = world > 1 ? (uint32_t)world : 0u;
  a.ws_capacity = workspace_part_bytes(dim0, C, N);
  a.bands = 1u;
  if (residual) (dir == 0 ? a.res : a.ymask) = &dummy;       // only their presence matters here
  return a;
}

extern "C" int anode_gpu_batch_norm_fused_serving_kernel(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual,
                                                         int aligned, int world)
{
  if (check_dims(dim0, dim1, dim2) || (dir != 0 && dir != 1)) return ANODE_E_DIMS;
  const int k = pick_kernel_kind(probe_call(dim0, dim1, dim2, dir, residual != 0, aligned != 0, world), dir, aligned != 0);
  return k < 0 ? ANODE_KERNEL_AUTO : k;
}

extern "C" int anode_gpu_batch_norm_fused_launched_kernel(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, int aligned)
{
  if (check_dims(dim0, dim1, dim2) || (dir != 0 && dir != 1)) return ANODE_E_DIMS;
  const FusedArgs a = probe_call(dim0, dim1, dim2, dir, residual != 0, aligned != 0, 1);
  const int kind = pick_kernel_kind(a, dir, aligned != 0);
  LongGeom lg; BandGeom bg;
  const int instead = pick_instead(a, dir, kind, aligned != 0, lg);
  if (instead >= 0) return instead;
  return kind == ANODE_KERNEL_STREAM && kernel_choice() != ANODE_KERNEL_STREAM && band_geom_of(a, dir, bg) ? ANODE_KERNEL_BAND : kind;
}

extern "C" int anode_gpu_batch_norm_fused_last_kernel(void) { return t_last_kernel; }

// The family, among the first four kernels, of the shape of a one-GPU call on aligned tensors.
static int family(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool residual)
{
  if (check_dims(dim0, C, N)) return ANODE_E_DIMS;
  const FusedArgs a = probe_call(dim0, C, N, dir, residual, true, 1);
  const int k = pick_kernel_kind(a, dir, true);
  if (k == ANODE_KERNEL_TILED && dim0 % 4 != 0) return ANODE_KERNEL_PLAIN;
  if (k != ANODE_KERNEL_REGISTER && k != ANODE_KERNEL_STREAM) return k;
  if (segres_preferred(a, dir, true)) return ANODE_KERNEL_CLUSTER;
  Plan p; RingGeom g;
  if (dim0 % 4 == 0 && ring_plan_of(a, dir, true, p, g)) return ANODE_KERNEL_TILED;
  return segres_applies(a, dir, true) ? ANODE_KERNEL_CLUSTER : ANODE_KERNEL_PLAIN;
}

extern "C" int anode_gpu_batch_norm_fused_kernel_kind(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir)
{
  return family(dim0, dim1, dim2, dir, false);
}

// The same for the residual-epilogue calls (anode_gpu_batch_norm_add_act_fused_*).
extern "C" int anode_gpu_batch_norm_add_act_fused_kernel_kind(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir)
{
  return family(dim0, dim1, dim2, dir, true);
}

extern "C" int anode_gpu_batch_norm_fused_set_kernel(int kernel)
{
  if (kernel < ANODE_KERNEL_AUTO || kernel > ANODE_KERNEL_LONG) return ANODE_E_DIMS;
  g_kernel_choice.store(kernel, std::memory_order_relaxed);
  return ANODE_OK;
}

// ---- diagnostics: geometry of the tiled kernel for a shape (no GPU needed) ----------------------
// out (12 values): applies, rows per tile, floats per row piece, tiles per unit, slots, bytes per slot, dynamic
// shared memory bytes, KiB between a tile's two visits, the fraction (in 1/1000) of such a window that L2 keeps by
// itself, blocks, steps between a tile's two visits, tiles
extern "C" int anode_gpu_batch_norm_tiled_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  Plan p; RingGeom g;
  for (int i = 0; i < 12; ++i) out[i] = 0;
  if (!ring_plan_for(dim0, dim1, dim2, true, dir, false, p, g)) return ANODE_OK;
  const uint64_t window = ring_window_bytes(p, dir);
  out[0] = 1; out[1] = p.rows_per_tile; out[2] = p.piece_len; out[3] = p.tiles_per_unit; out[4] = g.slots;
  out[5] = g.slot_stride; out[6] = g.smem_bytes; out[7] = (uint32_t)(window >> 10);
  out[8] = window > kRingLargeWindowMax ? (uint32_t)(1000.0 * (double)kRingLargeWindowMax / (double)window) : 1000u;
  out[9] = p.grid; out[10] = p.lookahead_steps; out[11] = p.total_tiles;
  return ANODE_OK;
}

// ---- diagnostics: what of a block's tiles stays in tensor memory (no GPU needed) ------------------
// out (10 values): kept at all, tile number `tile` of a block kept, place, the dealt number of consumer warp `warp`, its first
// column, kept tiles before, vectors of the largest tile, consumer warps, columns per set, steps between a tile's two visits
extern "C" int anode_gpu_batch_norm_tiled_keep(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual,
                                               uint32_t tile, uint32_t warp, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2) || warp >= ring_warps(dir)) return ANODE_E_DIMS;
  Plan p; RingGeom g;
  for (int i = 0; i < 10; ++i) out[i] = 0;
  if (!ring_plan_for(dim0, dim1, dim2, true, dir, residual != 0, p, g)) return ANODE_OK;
  ring_keep(p, dir, residual != 0, g);
  const Keep k = keep_at(g, tile);
  out[0] = g.keep_slots; out[1] = k.kept ? 1u : 0u; out[2] = k.slot;
  keep_place(g, k.slot, warp, ring_warps(dir), out[3], out[4]);
  out[5] = kept_before(g, tile); out[6] = ring_tile_vecs(p); out[7] = ring_warps(dir); out[8] = g.keep_set; out[9] = p.lookahead_steps;
  return ANODE_OK;
}

// ---- diagnostics: floats of a row's last piece in the tiled kernel, 0 where it does not apply (no GPU needed) ----
extern "C" uint32_t anode_gpu_batch_norm_tiled_last_piece(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual)
{
  using namespace anode_b200;
  Plan p; RingGeom g;
  if ((dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2) || !ring_plan_for(dim0, dim1, dim2, true, dir, residual != 0, p, g)) return 0;
  return dim0 - (p.pieces - 1) * p.piece_len;
}

// ---- diagnostics: geometry of the band kernel (no GPU needed) --------------------------------------
extern "C" int anode_gpu_batch_norm_band_geometry(uint32_t dim0, uint32_t dim1, uint32_t dim2, int dir, int residual, uint32_t *out)
{
  using namespace anode_b200;
  if (!out || (dir != 0 && dir != 1) || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  BandGeom g{};
  const bool taken = band_geom_of(probe_call(dim0, dim1, dim2, dir, residual != 0, true, 1), dir, g);
  if (!taken && !band_geom(dim0, dim1, dim2, dir, residual != 0, sm_count(), g)) g = BandGeom{};
  const uint32_t v[16] = {taken ? 1u : 0u, g.cb, g.units, g.groups, g.vpt, g.rows, g.tiles, g.grid, g.look, g.boxes, g.box4, g.box_bytes,
                          g.slots, g.slot_stride, g.smem_bytes, g.lane_shift};
  for (int i = 0; i < 16; ++i) out[i] = v[i];
  return ANODE_OK;
}

// ---- diagnostics: the tile plan, for tests of the index arithmetic (no GPU needed) ----------
extern "C" int anode_gpu_batch_norm_fused_plan(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                               uint32_t resident_blocks, uint32_t tile_floats,
                                               uint32_t slack_steps, uint32_t *out, uint32_t out_len)
{
  if (!out || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  const Tunables &t = tunables();
  const Plan p = make_plan(dim0, dim1, dim2, aligned != 0,
                           resident_blocks ? resident_blocks : sm_count() * t.blocks_per_sm,
                           tile_floats ? tile_floats : t.tile_floats, slack_steps ? slack_steps : t.slack_steps);
  const uint32_t v[] = {p.regime, p.vec, p.cb, p.units, p.rows_per_tile, p.piece_len, p.pieces,
                        p.sample_blocks, p.tiles_per_unit, p.total_tiles, p.grid, p.lookahead_steps,
                        p.div_mul, (uint32_t)(p.ws_bytes & 0xffffffffu), (uint32_t)(p.ws_bytes >> 32)};
  for (uint32_t i = 0; i < out_len && i < sizeof(v) / sizeof(v[0]); ++i) out[i] = v[i];
  return ANODE_OK;
}

extern "C" int anode_gpu_batch_norm_fused_plan_tile(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                                    uint32_t resident_blocks, uint32_t tile_floats,
                                                    uint32_t tile, uint64_t *out)
{
  if (!out || check_dims(dim0, dim1, dim2)) return ANODE_E_DIMS;
  const Tunables &t = tunables();
  const Plan p = make_plan(dim0, dim1, dim2, aligned != 0,
                           resident_blocks ? resident_blocks : sm_count() * t.blocks_per_sm,
                           tile_floats ? tile_floats : t.tile_floats, t.slack_steps);
  if (tile >= p.total_tiles) return ANODE_E_DIMS;
  const TileRange r = tile_range(p, tile);
  out[0] = r.unit; out[1] = r.c0; out[2] = r.cw; out[3] = r.n0; out[4] = r.rows; out[5] = r.col0;
  out[6] = r.len; out[7] = r.base;
  return ANODE_OK;
}

// Walks `count` tiles first, first+stride, ... with the division-free iterator the kernels use.
// out: 8 values per tile as in anode_gpu_batch_norm_fused_plan_tile.
extern "C" int anode_gpu_batch_norm_fused_plan_walk(uint32_t dim0, uint32_t dim1, uint32_t dim2, int aligned,
                                                    uint32_t resident_blocks, uint32_t tile_floats,
                                                    uint32_t first, uint32_t stride, uint32_t count, uint64_t *out)
{
  if (!out || check_dims(dim0, dim1, dim2) || stride == 0) return ANODE_E_DIMS;
  const Tunables &t = tunables();
  const Plan p = make_plan(dim0, dim1, dim2, aligned != 0,
                           resident_blocks ? resident_blocks : sm_count() * t.blocks_per_sm,
                           tile_floats ? tile_floats : t.tile_floats, t.slack_steps);
  TileIter it; it.init(p, first, stride);
  for (uint32_t i = 0; i < count; ++i) {
    if (it.tile() >= p.total_tiles) return ANODE_E_DIMS;
    const TileRange r = it.range(p);
    uint64_t *o = out + 8 * (size_t)i;
    o[0] = r.unit; o[1] = r.c0; o[2] = r.cw; o[3] = r.n0; o[4] = r.rows; o[5] = r.col0; o[6] = r.len; o[7] = r.base;
    it.advance(p);
  }
  return ANODE_OK;
}
