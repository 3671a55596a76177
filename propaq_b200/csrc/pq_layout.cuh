// pq_layout.cuh -- how the rows of a binned sweep are laid out in a buffer
// (pq_bins.cuh): plain arithmetic, the same on the device and on the host,
// which sizes the buffers by it.
#pragma once
#include "pq_device.cuh"

namespace pq {

constexpr u32 BIN_THREADS = 256;   // of a block
constexpr u32 SOLO_ROWS = 2048;    // of a block alone; a rotation runs while it may double its rows
constexpr u32 BIN_MAX = 1u << 18;  // bins of one buffer
constexpr u32 COUNT_WORDS = BIN_MAX;  // words of one counter set (fewer bins, wider stride: choose_layout)

// Bin b holds rows [b * cap, b * cap + count[b]) of its buffer, and rows past
// a full bin go to the buffer's spill area, tagged with their bin.
constexpr u64 SPILL_SHARE = 16;  // of a buffer, at least; more spills than there is room for and the host grows it
struct Layout {
  u32 bins, stride;  // counters are `stride` words apart (few bins: a sector or line each)
  u32 cap;
};

// Spill tags a buffer of `room` rows holds.
__host__ __device__ __forceinline__ u64 spill_tags(u64 room) { return room / 8; }
// Rows that may spill: what the bins leave of the buffer, as far as there are
// tags.  The bins leave room / SPILL_SHARE and up to bins - 1 rows more, which
// is more than the tags when a small buffer gets very many bins.
__host__ __device__ __forceinline__ u64 spill_room(const Layout& l, u64 room) {
  const u64 rest = room - (u64)l.bins * l.cap, tags = spill_tags(room);
  return rest < tags ? rest : tags;
}
// Every bin that spilled reads all the tags, so a buffer that more rows than
// this spill in is grown although it holds them, as long as the device has room
// for a larger one (2^22 rows in a buffer of 2^22, 260,000 of them spilled: a call
// that ends in two rotations on them took 5.5 ms, and 1.3 with a larger one).
__host__ __device__ __forceinline__ u64 spill_limit(u64 room) { return room / 32; }

// Bins for about n rows that a window lets grow by a factor `grow`, grown bins
// `fill` full.  While a bin of every warp holds at most WARP_ROWS rows when
// grown, that many (a warp alone runs 32 branching rows at a time, a block
// 256: bins that grew to 62 rows a warp ran a window of 50 rotations in 79 us
// (kicked Ising 10x10) against 72 us by blocks, bins of 22 one of 40 in 43
// against 51 us; where one family fills a bin, as in a TFIM chain's RX layer,
// the line is lower); else bins of blocks, one each or, up to four, a whole
// number each (340 bins on 296 blocks cost two rounds).  All the room there
// is, less the spill area.
constexpr float WARP_ROWS = 12.0f;
__host__ __device__ __forceinline__ Layout choose_layout(float n, float grow, float fill, u32 blocks, u32 warps,
                                                         u32 rows, u64 room) {
  Layout l;
  u64 b = (u64)(n * grow / (fill * (float)rows)) + 1;
  if (n * grow <= WARP_ROWS * (float)(blocks * warps)) b = (u64)blocks * warps;
  else if (b < 4ull * blocks) b = (b + blocks - 1) / blocks * blocks;
  else if (b == (u64)blocks * warps) ++b;  // that number means bins of warps
  if (b > BIN_MAX) b = BIN_MAX;
  l.bins = (u32)b;
  l.stride = b <= 4096 ? 32u : (b <= 16384 ? 8u : 1u);
  const u64 c = (room - room / SPILL_SHARE) / b;
  l.cap = c > 0x7fffffffull ? 0x7fffffffu : (u32)c;
  return l;
}

}  // namespace pq
