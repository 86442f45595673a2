// Geometry of the band kernel (bn_band.cu): plain C++, also for the CPU tests of its index arithmetic.
//
//   band   the cb*dim0 contiguous floats that a unit (cb adjacent channels) has in one sample, a multiple of four
//   tile   `rows` bands, one below the other: sample group i of a tile is its samples i, i + groups, ...; a consumer thread owns
//          one 16-byte column of the band and one group
//   box    a band's part of at most 64 vectors: what a tensor copy fetches of all the tile's samples, packed in shared memory
#pragma once
#include "bn_plan.h"

namespace anode_b200 {

constexpr uint32_t kBandWarps = 8, kBandConsumers = 32 * kBandWarps;      // consumer warps and threads
constexpr uint32_t kBandThreads = kBandConsumers + 96;                     // + producer, delivery and coefficient warps
constexpr uint32_t kBandChannels = 32;      // most channels of a unit
constexpr uint32_t kBandVecs = 64;          // vectors of tensor memory per consumer thread (512 columns for four warps)
constexpr double kBandWordCost = 3.5, kBandRunCost = 140.0;      // band_geom: vectors that a word costs, bytes that a run's ends cost
constexpr uint32_t kBandWords = 512;        // most words of a unit
constexpr uint32_t kBandBox = 64;           // most vectors of a box (256 floats, the most a tensor map takes)
constexpr uint32_t kBandMaxSlots = 8, kBandQ = 3;
constexpr uint32_t kBandCtlBytes = 1024;
constexpr uint32_t kBandWordBytes = 16;     // a tile's pair of doubles for a channel
constexpr uint32_t kBandSmem = 227u * 1024u;

struct BandGeom {
  uint32_t cb, units, L4;              // channels of a unit, units, vectors of a unit's run in one sample (its band)
  uint32_t groups, vpt, rows;          // a tile: `groups` samples side by side, vpt samples per thread, rows = groups * vpt
  uint32_t tiles, total, grid, look;   // tiles of a unit, of the layer; blocks; steps between a tile's two visits
  uint32_t boxes, box4, box_bytes;     // boxes of a band, vectors of a box's row, bytes of a box in a slot
  uint32_t slots, plane_bytes, slot_stride, off_side, off_res, off_coef, off_slots, smem_bytes;
  uint32_t off_second, res_bytes;      // of an entry of the threads' sums (BandSums)
  uint32_t lane_shift;                 // log2 of the lanes that work on one channel in the service warps
  uint32_t whole;                      // loads: 1 the lines are dead once read, 0 neighbouring units' blocks read parts of them, too
  uint32_t tag, hdr;                   // workspace: tagged words, exit counter and parity word (byte offsets)
  double inv_count;                    // reciprocal of a channel's elements in the layer
};

// Tagged words of one of the two buffers.
ANODE_HD uint64_t band_words(const BandGeom &g) { return (uint64_t)g.total * g.cb; }

// Tensors of a slot: what the reduce visits read.
ANODE_HD uint32_t band_planes(int dir, bool extra) { return dir == 0 ? 1u : extra ? 3u : 2u; }

// The layer's geometry for `sms` blocks; false where the kernel cannot take it.
inline bool band_geom(uint32_t dim0, uint32_t C, uint32_t N, int dir, bool extra, uint32_t sms, BandGeom &g)
{
  if (dim0 < 4 || (uint64_t)C * dim0 % 4 != 0) return false;
  uint32_t q = 4; if (dim0 % 2 == 0) q = 2; if (dim0 % 4 == 0) q = 1;      // cb*dim0 must be a multiple of 4
  const uint32_t kept = dir == 0 ? 1u : 2u, most = kBandVecs / 4 / kept;      // tensors kept; most samples per thread, for four tiles
  // Channels of a unit and samples per thread: the least (steps + 3) * (cost of a step) * (cost of the runs), fitted to measurements
  // of the form with f32 words.  (Twice the cost per word with today's, us: [256,2048,7,7] forward 45.8 -> 51.3, [256,1024,14,14] backward 106 -> 113,
  // [4000,100,12,12] backward 139 -> 131.)
  //   A step: a fixed part (merge, barriers, parameters), the tile's vectors, the unit's words.  [1024,2048,7,7] forward / backward with
  //   tiles of 16 / 8, 12 / 6, 8 / 4 samples per thread 143 / 202, 145 / 231, 169 / 300 us; [200,2048,8,8] backward with units of 16
  //   channels and 400 words 64 us, of 2 and 22 words 60; [400,2048,8,8] forward with 400 words 82 us, with 15 76.
  //   The runs: short ones cost HBM and the copies more (a run that ends within a 32-byte sector shares it with another block's).
  //   [256,1024,14,14] forward with runs of 784, 1568, 3136, 3920 bytes 92, 84, 80, 80 us; [100,2048,12,12] of 576 and 4032 bytes 59 and 49.
  // Runs of 512 bytes at least where the channels make them.
  const double fixed = dir == 0 ? 1000.0 : 1900.0;
  double best = 0.0;
  for (uint32_t cb = q; cb <= C && cb <= kBandChannels && (uint64_t)cb * dim0 <= 4 * kBandConsumers; cb += q) {
    const uint32_t L4 = cb * dim0 / 4;
    if (L4 < 32 && cb + q <= C && cb + q <= kBandChannels) continue;
    const uint32_t units = ceil_div_u32(C, cb), groups = kBandConsumers / L4 < N ? kBandConsumers / L4 : N;
    for (uint32_t vpt = most; vpt >= most / 4; --vpt) {
      if (vpt * groups > 256) continue;                                         // (rows of a box)
      const uint32_t per = ceil_div_u32(ceil_div_u32(N, ceil_div_u32(N, groups * vpt)), groups), rows = groups * per;      // equal tiles
      const uint32_t tiles = ceil_div_u32(N, rows);
      // A unit's tiles make one step of the grid at most, and every block merges a unit's words: sixteen per lane at most where the channels
      // are a power of two, thirty where a lane has a channel of 17 to itself.  (Forward, streaming kernel and this one with more of them: [8000,20,11,11] 66 and 103 us, [20000,12,7,9] 72 and 109.)
      if (tiles > sms || tiles * cb > kBandWords || 4ull * rows * C * dim0 >> 32) continue;      // (a thread's places within a tile: 32 bits)
      const uint32_t total = units * tiles;
      if (total < sms) continue;
      const double cost = (double)(ceil_div_u32(total, sms) + 3) * (fixed + (double)(rows * L4) + kBandWordCost * (double)(tiles * cb)) * (1.0 + kBandRunCost / (16.0 * L4));
      if (best != 0.0 && cost > 0.98 * best) continue;
      best = cost;
      g.cb = cb; g.L4 = L4; g.units = units; g.groups = groups; g.vpt = per; g.rows = rows; g.tiles = tiles; g.total = total;
    }
  }
  if (best == 0.0) return false;
  g.grid = sms; g.look = 3;
  g.boxes = ceil_div_u32(g.L4, kBandBox); g.box4 = ceil_div_u32(g.L4, g.boxes);
  g.box_bytes = (g.rows * g.box4 * 16 + 127) / 128 * 128;
  g.plane_bytes = g.boxes * g.box_bytes;
  g.lane_shift = 5;
  while (g.lane_shift && (32u >> g.lane_shift) < g.cb) --g.lane_shift;
  uint32_t off = kBandCtlBytes;
  g.off_side = off; off += kBandMaxSlots * kBandChannels * 16;                          // per slot (mean, scale, beta) of the channels
  // per entry: the threads' sums for their first channels, and for their second ones (a channel has one such vector per group)
  g.off_second = kBandConsumers * 16; g.res_bytes = g.off_second + (dim0 % 4 ? g.groups * g.cb * 16 : 0);
  g.off_res = off; off += kBandQ * g.res_bytes;
  g.off_coef = off; off += kBandQ * 2 * kBandChannels * 16;                             // per entry: the channels' coefficients
  g.off_slots = off = (off + 127) / 128 * 128;
  g.slot_stride = g.plane_bytes * band_planes(dir, extra);
  g.slots = (kBandSmem - off) / g.slot_stride;
  if (g.slots < 2) return false;
  if (g.slots > kBandMaxSlots) g.slots = kBandMaxSlots;
  g.smem_bytes = off + g.slots * g.slot_stride;
  g.inv_count = 1.0 / ((double)dim0 * (double)N);
  return true;
}

}  // namespace anode_b200
