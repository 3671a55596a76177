// The layout rule of the binned sweep (propaq_b200/csrc/pq_layout.cuh)
// compiled for the host with g++; built by test_bin_layout_cpu.py.
#define __host__
#define __device__
#define __forceinline__ inline
static inline int __popcll(unsigned long long x) { return __builtin_popcountll(x); }

#include "../propaq_b200/csrc/pq_layout.cuh"

// out: bins, stride, cap, rows that may spill, tags allocated, words of a counter set
extern "C" void bl_layout(float n, float grow, float fill, unsigned blocks, unsigned warps, unsigned rows,
                          unsigned long long room, unsigned long long* out) {
  const pq::Layout l = pq::choose_layout(n, grow, fill, blocks, warps, rows, room);
  out[0] = l.bins;
  out[1] = l.stride;
  out[2] = l.cap;
  out[3] = pq::spill_room(l, room);
  out[4] = pq::spill_tags(room);
  out[5] = pq::COUNT_WORDS;
}
