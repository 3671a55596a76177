// pq_bins.cuh -- the binned sweep: whole runs of rotations on rows held in
// shared memory.
//
// Included by pq_kernels.cu inside its anonymous namespace (it uses that
// file's barrier and algebra helpers).
//
// A *window* is a run of rotations together with a function of the key, the
// group hash, that none of its rotations changes: a term and every term the
// window can ever pair it with or branch it into have the same group hash.
// So the rows can be dealt into *bins* by that hash, and a block can take one
// bin into shared memory and run the whole window on it -- the reference's
// pair rule (crates/core/src/engine/termsum.rs:604-751) rotation by rotation,
// in order, with every partner found in a shared-memory hash table -- without
// looking at any other bin.  Every coefficient is the same two-operand result
// as in a pass over all rows per rotation, and the per-rotation live counts
// are the sums over the bins; only where a row is stored differs.  When the
// window is done the block applies the reclaim that follows it, if any
// (engine.rs:117-161), and deals its rows straight into the bins of the next
// window.  A window therefore costs one grid barrier and one read and one
// write of each row, where the row sweep (sweep_body) pays a barrier and
// several dependent L2 or DRAM round trips per rotation.
//
// Group hashes (host: plan_windows).  Keys are hashed by a GF(2)-linear map h
// (lin_hash), so h(K ^ G) = h(K) ^ h(G) and a child's hash costs one xor.
//   * span windows: the hash of K reduced by a row-echelon basis of the span
//     of the window's generators, of rank at most BIN_RANK: a group has at
//     most 2^rank keys, so one always fits in shared memory;
//   * disjoint windows: Pauli generators on pairwise disjoint qubits (they
//     commute).  K is reduced only by the generators it anticommutes with --
//     the set no rotation of the window changes -- so their number is not
//     limited: a weight cut of at most BIN_RANK bounds that set's size, and
//     with it the group's, for every row.
//
// A bin that does not fit (its rows, or the rows it grows to) is run again in
// halves by further bits of the group hash, as often as it takes; nothing of
// a bin is written before all of it has fitted.
//
// Small live sets run in one block with no grid barrier at all (solo_body):
// all rows in shared memory, every op a step between two block barriers.
//
// What bounds it: the dependent shared-memory round trips of a rotation's
// step (about 1 us on small bins; 2-3 us where a block's 1,500-3,000 rows
// branch often), no longer the grid barrier or DRAM.  Whole calls, row sweep
// -> binned sweep, on one box: 4-qubit circuit, 40 noisy rotations 0.66 ->
// 0.29 ms; 20-qubit TFIM (to 57k rows) 2.05 -> 0.83 ms; kicked Ising 10x10 x
// 20 steps (4-word keys, to 477k rows) 23.3 -> 8.8 ms, 6x6 x 8 (2 words, to
// 1.2M) 9.2 -> 3.0 ms, 12x15 x 8 (8 words) 31.5 -> 12.3 ms; Givens circuits
// of 24 sites (16M rows) 54 -> 15.6 ms and 32 sites (80M rows) 453 -> 119 ms.
#pragma once

constexpr u32 TAB_EMPTY = 0xffffffffu;
constexpr u32 IDX_BITS = 13;  // row index bits of a shared-memory table slot, the rest is fingerprint
constexpr u32 IDX_MASK = (1u << IDX_BITS) - 1u;

template <int W, int T_, int R_, int SLOTS_>
struct BinSmem {
  static constexpr int T = T_, R = R_, SLOTS = SLOTS_;
  static_assert(R < (int)IDX_MASK && R <= 32 * T, "a table slot holds a row index, a thread 32 row bits");
  double coef[R];
  u64 key[W][R];  // by word: lanes of consecutive rows read consecutive addresses
  u32 h[R];
  u32 tab[SLOTS];
  GateDesc<W> gate[4];  // ring: the running rotation and the next two
  u64 pm[W];  // pivot bits of the next window's grouping
  u32 hv[64 * W];  // per pivot bit: hash of its basis vector
  u32 born[WIN_MAX], anti[WIN_MAX];    // this bin, per rotation
  u32 born_all[WIN_MAX], anti_all[WIN_MAX];  // this block's bins of the window
  OpDesc op[4];  // ring (solo)
  unsigned short list[R];  // the running rotation's anticommuting rows
  u32 n_list[2];           // their number; the other one is zero for the next rotation
  unsigned char gate_of[64 * W];  // per pivot bit: the window's rotation it belongs to (disjoint windows)
  u32 n, kept, tick;
  u32 x[8];  // words read after a grid barrier
  u64 y[4];
};

// ------------------------------------------------------------ linear hash
__device__ __forceinline__ u32 rotl32(u32 v, int r) { return r ? (v << r) | (v >> (32 - r)) : v; }
template <int W>
__device__ u32 lin_hash(const u64* k, const u32* lin) {
  u32 h = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    if (!k[w]) continue;
    u32 t = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) t ^= __ldg(lin + 256 * b + ((k[w] >> (8 * b)) & 255u));
    h ^= rotl32(t, (5 * w) & 31);
  }
  return h;
}

// Does K anticommute with the generator: the parity of K against one mask
// (Pauli: the pair-swapped generator; Majorana: the generator, or its
// complement when its length is odd -- overlap plus K's length).
template <int W, int ALG>
__device__ __forceinline__ u64 anti_word(const GateDesc<W>& d, int w) {
  if constexpr (ALG == 0) return d.g.fold[w];
  return (d.g.aux & 1) ? ~d.g.gen[w] : d.g.gen[w];
}

// ------------------------------------------------------------ rotation
struct BinRules {
  u32 wcut, n_units;
  bool ccut;
  double minc;
};

// The table: pairs of slots (8 bytes, one load), probed pair by pair from the
// key's; a pair fills its first slot first.  A slot is the hash's upper bits
// over the row; 0xffffffff (row 8191) cannot occur since rows stop below it.
template <class S>
__device__ __forceinline__ u32 tab_start(u32 h) {
  constexpr int SHIFT = 33 - (S::SLOTS == 4096 ? 12 : (S::SLOTS == 8192 ? 13 : 14));
  static_assert(S::SLOTS / 2 == 1 << (32 - SHIFT), "table size");
  return (h * 0xC2B2AE35u) >> SHIFT;
}
template <class S>
__device__ __forceinline__ void tab_insert(S& s, u32 h, u32 row, u32 pair) {
  const u32 v = (h & ~IDX_MASK) | row;
  for (;;) {
    if (atomicCAS(&s.tab[2 * pair], TAB_EMPTY, v) == TAB_EMPTY) return;
    if (atomicCAS(&s.tab[2 * pair + 1], TAB_EMPTY, v) == TAB_EMPTY) return;
    pair = (pair + 1) & (S::SLOTS / 2 - 1);
  }
}

__device__ __forceinline__ double flip(double v, bool neg) {  // v * -1.0 or v * 1.0
  return __longlong_as_double(__double_as_longlong(v) ^ ((long long)neg << 63));
}

// One rotation on the n rows in shared memory, in two parts.  First every
// thread tests its rows for anticommutation (all loads independent) and the
// block gathers the anticommuting ones into one list; then the warps take 32
// of them at a time through the long path -- partner lookup, pair rule, child
// -- so that it runs with full warps, evenly over the block, however few rows
// anticommute and wherever they lie.  The lower row of a pair owns both
// coefficients; children are appended from row n on (born counts them) and
// inserted into the table, where no lookup of this rotation can match them
// (their row is >= n).  Rows past the capacity are counted but not stored;
// the caller sees n grow past R.  Block-wide; the caller's barrier ends it.
//
// Every row in a run without a TermBudget floor is within the weight cut (the
// admission, each branch and each reclaim keep to it), so in a pair only the
// coefficient check can hold a branch back: S_DROP arises for a lone row's
// child alone.
template <int W, int ALG, class S>
__device__ __forceinline__ void rotate_rows(S& s, const GateDesc<W>& d, const BinRules& R, u32 n, u32 flip_flop,
                                            u32* born, u32* anti) {
  using Ops = typename Alg<ALG>::T;
  constexpr int T = S::T, U = 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if ((u32)warp * 32u < n) {
    u32 bits = 0;
    for (u32 i = 0; i * T < n; i += U) {
      u64 acc[U];
#pragma unroll
      for (int u = 0; u < U; ++u) acc[u] = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        const u64 am = anti_word<W, ALG>(d, w);
        if (am) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const u32 r = (i + u) * T + tid;
            if (r < n) acc[u] ^= s.key[w][r] & am;
          }
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) bits |= (u32)(popc(acc[u]) & 1) << (i + u);
    }
    if (__any_sync(FULL, bits != 0)) {
      const u32 mine = __popc(bits);
      u32 at = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 y = __shfl_up_sync(FULL, at, o);
        if (lane >= o) at += y;
      }
      u32 base = 0;
      if (lane == 31) base = atomicAdd(&s.n_list[flip_flop], at);
      at += __shfl_sync(FULL, base, 31) - mine;
      for (; bits; bits &= bits - 1) s.list[at++] = (unsigned short)((__ffs(bits) - 1) * T + tid);
    }
  }
  __syncthreads();
  const u32 total = s.n_list[flip_flop];
  if (tid == 0) {
    s.n_list[flip_flop ^ 1] = 0;
    *anti = total;
  }
  if (fabs(d.sn) < 1e-9) {  // OP_PHASE
    for (u32 i = tid; i < total; i += T) s.coef[s.list[i]] = __dmul_rn(s.coef[s.list[i]], d.cs);
    return;
  }
  const unsigned lt = (1u << lane) - 1u;
  for (u32 i = (u32)warp * 32u; i < total; i += T) {
    const bool act = i + lane < total;
    const u32 r = act ? s.list[i + lane] : 0u;
    bool emit = false;
    u64 k[W], q[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      k[w] = s.key[w][r];
      q[w] = k[w] ^ d.g.gen[w];
    }
    const u32 hq = s.h[r] ^ d.hash;
    u32 pair = tab_start<S>(hq);
    uint2 e = reinterpret_cast<const uint2*>(s.tab)[pair];
    // beside the lookup: phase of G K = i^p, p odd; the sin branch's sign is - for p = 1
    const bool neg = (Ops::template product_exp<W>(d.g, k) == 1) != (d.g.sign < 0.0);
    const double c = s.coef[r], m = __dmul_rn(c, d.sn);
    const double b = flip(m, neg);
    const bool held = R.ccut && fabs(m) < R.minc;
    if (act) {
      u32 j = TAB_EMPTY;
      for (;;) {
        auto hit = [&](u32 v) {
          const u32 row = v & IDX_MASK;
          if (((v ^ hq) & ~IDX_MASK) != 0 || row >= n) return false;
          u64 df = 0;
#pragma unroll
          for (int w = 0; w < W; ++w) df |= s.key[w][row] ^ q[w];
          if (!df) j = row;
          return !df;
        };
        if (e.x == TAB_EMPTY || hit(e.x) || e.y == TAB_EMPTY || hit(e.y)) break;
        pair = (pair + 1) & (S::SLOTS / 2 - 1);
        e = reinterpret_cast<const uint2*>(s.tab)[pair];
      }
      if (j > r) {  // lone (j empty), or the pair's owner
        double nc = __dmul_rn(c, d.cs);
        if (j == TAB_EMPTY) {
          emit = !held && (R.wcut == NO_WEIGHT_CUT || Ops::template weight<W>(q, R.n_units) <= R.wcut);
        } else {
          // G (G K) = K: the partner's phase is the inverse, its sign the opposite
          const double cj = s.coef[j], mj = __dmul_rn(cj, d.sn);
          double nj = __dmul_rn(cj, d.cs);
          if (!(held && fabs(mj) < R.minc)) {
            nc = __dadd_rn(nc, flip(mj, !neg));
            nj = __dadd_rn(nj, b);
          }
          s.coef[j] = nj;
        }
        s.coef[r] = nc;
      }
    }
    __syncwarp();
    const unsigned em = __ballot_sync(FULL, emit);
    if (em) {
      u32 row = 0;
      if (lane == 0) row = atomicAdd(born, (u32)__popc(em));
      row = n + __shfl_sync(FULL, row, 0) + __popc(em & lt);
      if (emit && row < (u32)S::R) {
#pragma unroll
        for (int w = 0; w < W; ++w) s.key[w][row] = q[w];
        s.coef[row] = b;
        s.h[row] = hq;
        tab_insert(s, hq, row, pair);
      }
    }
  }
}

// Descriptors on their way into the ring (cp.async), by the block's last
// warp, which has rows of its own only when the block is nearly full: its
// waits overlap the other warps' work.
template <int W>
__device__ __forceinline__ void fetch_gate(GateDesc<W>* dst, const GateDesc<W>* src) {
  constexpr u32 WORDS = sizeof(GateDesc<W>) / 8;
  for (u32 w = threadIdx.x & 31; w < WORDS; w += 32)
    cp_async8(reinterpret_cast<u64*>(dst) + w, reinterpret_cast<const u64*>(src) + w);
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All groups but the latest are complete.
__device__ __forceinline__ void cp_async_wait_1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ void stamp_op(u64* stamps, u32 op) {
  u64 t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  stamps[op] = t;
}

// ------------------------------------------------------------ solo
// One block runs ops from a.op_begin on while the rows fit its shared memory
// (a gate may double them), then writes the rows out dense and leaves the op
// it stopped before in st->end_op and the live count in st->n[0].
template <int W, int ALG, class S>
__device__ __forceinline__ void solo_body(const BinArgs& a, S& s) {
  using Ops = typename Alg<ALG>::T;
  constexpr int T = S::T;
  const int tid = threadIdx.x, lane = tid & 31;
  SweepState* st = a.st;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  u32 op = a.op_begin;
  const u64 n_in = a.n0;
  if (n_in > (u64)S::R / 2) {
    if (tid == 0) {
      st->n[0] = n_in;
      st->end_op = op;
    }
    return;
  }
  u32 n = (u32)n_in;
  auto clear_table = [&] {
    for (int i = tid; i < S::SLOTS / 4; i += T)
      reinterpret_cast<uint4*>(s.tab)[i] = make_uint4(TAB_EMPTY, TAB_EMPTY, TAB_EMPTY, TAB_EMPTY);
  };
  clear_table();
  if (tid < 4) s.born[tid] = s.anti[tid] = 0;
  if (tid < 2) s.n_list[tid] = 0;
  __syncthreads();
  for (u32 r = tid; r < n; r += T) {
    u64 k[W];
    load_key<W>(a.keys, r, k);
    const u32 h = lin_hash<W>(k, a.lin);
#pragma unroll
    for (int w = 0; w < W; ++w) s.key[w][r] = k[w];
    s.coef[r] = a.coeffs[r];
    s.h[r] = h;
    tab_insert(s, h, r, tab_start<S>(h));
  }
  BinRules R;
  R.n_units = a.n_units;
  R.minc = a.min_coeff;
  u32 step = 0;  // rotations run: their counters are born / anti [step & 3]
  u32 last = 0xffffffffu;   // op whose counters are in born[(step - 1) & 3], not yet taken
  const bool fetcher = tid >= T - 32;
  // The live count after the last rotation; thread 0 records its counters.
  auto take = [&] {
    if (last == 0xffffffffu) return;
    const u32 b = s.born[(step - 1) & 3];
    n += b;
    if (tid == 0) {
      a.born[last] = b;
      a.anti[last] = s.anti[(step - 1) & 3];
    }
    last = 0xffffffffu;
  };
  // Rings: ops op, op + 1 (and, while op runs, op + 2); the next rotation's
  // descriptor (gate index gi), the one after, and gi + 2 while gi runs.
  u32 gi = a.first_gate;
  if (fetcher) {
    if (lane < 2 && op + lane < a.op_end) cp_async8(&s.op[(op + lane) & 3], a.ops + op + lane);
    for (u32 g = gi; g < gi + 2 && g < a.n_gdesc; ++g) fetch_gate<W>(&s.gate[g & 3], gates + g);
    cp_async_wait();
  }
  while (op < a.op_end) {
    if (fetcher) cp_async_wait_1();
    __syncthreads();  // the step before is done; this op's descriptors are here
    take();
    const OpDesc od = s.op[op & 3];
    const bool rot = od.kind == OP_GATE || od.kind == OP_PHASE;
    if (od.kind == OP_GATE && 2 * n > (u32)S::R) break;
    if (fetcher) {
      if (lane == 0 && op + 2 < a.op_end) cp_async8(&s.op[(op + 2) & 3], a.ops + op + 2);
      if (rot && gi + 2 < a.n_gdesc) fetch_gate<W>(&s.gate[(gi + 2) & 3], gates + gi + 2);
      cp_async_commit();
    }
    if (rot) {
      if (tid == 0) s.born[(step + 2) & 3] = 0;
      R.wcut = a.max_weight;
      R.ccut = a.has_min_coeff != 0;
      rotate_rows<W, ALG>(s, s.gate[gi & 3], R, n, step & 1, &s.born[step & 3], &s.anti[step & 3]);
      last = op;
      ++step;
      ++gi;
    } else {
      const double* factors = a.tables + (u64)od.idx * a.table_len;
      const u32 lastw = a.table_len - 1;
      const bool reclaim = od.kind == OP_NOISE_COMPACT;
      if (reclaim) {
        if (tid == 0) s.n = 0;
        clear_table();
      }
      // T rows a round: all of a round are in registers before any is written
      // back, and the survivors of the first i rounds never reach row i T.
      for (u32 r0 = 0; r0 < n; r0 += T) {
        const u32 r = r0 + tid;
        u64 k[W];
        double c = 0.0;
        u32 h = 0;
        bool kp = false;
        if (r < n) {
#pragma unroll
          for (int w = 0; w < W; ++w) k[w] = s.key[w][r];
          h = s.h[r];
          const u32 wt = Ops::template weight<W>(k, a.n_units);
          c = __dmul_rn(s.coef[r], __ldg(factors + (wt < lastw ? wt : lastw)));
          if (!reclaim)
            s.coef[r] = c;
          else
            kp = (a.max_weight == NO_WEIGHT_CUT || wt <= a.max_weight) &&
                 (!a.has_min_coeff || fabs(c) >= a.min_coeff);
        }
        if (!reclaim) continue;
        __syncthreads();
        const unsigned m = __ballot_sync(FULL, kp);
        if (!m) continue;
        u32 at = 0;
        if (lane == 0) at = atomicAdd(&s.n, (u32)__popc(m));
        at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (!kp) continue;
#pragma unroll
        for (int w = 0; w < W; ++w) s.key[w][at] = k[w];
        s.coef[at] = c;
        s.h[at] = h;
        tab_insert(s, h, at, tab_start<S>(h));
      }
      if (reclaim) {
        __syncthreads();
        n = s.n;
      }
      if (tid == 0) a.hist[op] = n;
    }
    if (tid == T - 1 && (op + 1 == a.op_end || (s.op[(op + 1) & 3].kind == OP_NOISE_COMPACT) !=
                                                   (od.kind == OP_NOISE_COMPACT)))
      stamp_op(a.stamps, op);
    ++op;
  }
  __syncthreads();
  take();
  if (fetcher) cp_async_wait();
  for (u32 r = tid; r < n; r += T) {
    u64 k[W];
#pragma unroll
    for (int w = 0; w < W; ++w) k[w] = s.key[w][r];
    store_key<W>(a.keys, r, k);
    a.coeffs[r] = s.coef[r];
  }
  if (tid == 0) {
    st->n[0] = n;
    st->end_op = op;
  }
}

// ------------------------------------------------------------ binned windows
// The bins the rows are dealt into: bin b holds rows [b * cap, b * cap +
// count[b]) of its buffer, and rows past a full bin go to the buffer's spill
// area, tagged with their bin.  to == 0xffffffff: dense, no bins (the end of
// the sweep).
constexpr u64 SPILL_SHARE = 16;  // of a buffer; more spills than that and the host grows it
struct Layout {
  u32 bins, stride;  // counters are `stride` words apart (few bins: a sector or line each)
  u32 cap;
};

// Bins for about n rows, m of them each, in a buffer of `room` rows: never
// fewer than the blocks, all the room there is (less an eighth for spills).
__device__ __forceinline__ Layout choose_layout(u64 n, u32 m, u32 blocks, u64 room) {
  Layout l;
  u64 b = (n + m - 1) / m;
  if (b < blocks) b = blocks;
  if (b > BIN_MAX) b = BIN_MAX;
  l.bins = (u32)b;
  l.stride = b <= 2048 ? 32u : (b <= 16384 ? 4u : 1u);
  const u64 c = (room - room / SPILL_SHARE) / b;
  l.cap = c > 0x7fffffffull ? 0x7fffffffu : (u32)c;
  return l;
}

__device__ __forceinline__ u32 bin_of(u32 g, u32 bins) { return __umulhi(g * 0x9E3779B1u, bins); }
// The bits a bin is split by when it does not fit.
__device__ __forceinline__ u32 split_bits(u32 g) { return (g ^ (g >> 15)) * 0x85EBCA6Bu; }

// Group hash from the basis list itself (the slow way: splits only).
template <int W, int ALG>
__device__ u32 group_hash_list(const u64* k, u32 h, const BinArgs& a, const WinDesc& w) {
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  for (u32 i = 0; i < w.n_basis; ++i) {
    const BasisDesc b = a.basis[w.basis + i];
    if (!key_bit(k, b.bit)) continue;
    if (w.disjoint) {
      u64 acc = 0;
#pragma unroll
      for (int x = 0; x < W; ++x) acc ^= k[x] & anti_word<W, ALG>(gates[w.gate + b.gate], x);
      if (!(popc(acc) & 1)) continue;
    }
    h ^= b.hash;
  }
  return h;
}

template <int W, int ALG, class S>
__device__ __forceinline__ u32 group_hash(const S& s, const u64* k, u32 h, const GateDesc<W>* gates, const WinDesc& w) {
#pragma unroll
  for (int x = 0; x < W; ++x)
    for (u64 m = k[x] & s.pm[x]; m; m &= m - 1) {
      const int bit = 64 * x + __ffsll((long long)m) - 1;
      if (w.disjoint) {
        const GateDesc<W>& d = gates[w.gate + s.gate_of[bit]];
        u64 acc = 0;
#pragma unroll
        for (int y = 0; y < W; ++y) acc ^= k[y] & __ldg(&d.g.fold[y]);
        if (!(popc(acc) & 1)) continue;
      }
      h ^= s.hv[bit];
    }
  return h;
}

// Loads the grouping of window w into shared memory.
template <int W, class S>
__device__ __forceinline__ void load_grouping(S& s, const BinArgs& a, const WinDesc& w) {
  if (threadIdx.x < W) s.pm[threadIdx.x] = 0;
  __syncthreads();
  for (u32 i = threadIdx.x; i < w.n_basis; i += S::T) {
    const BasisDesc b = a.basis[w.basis + i];
    s.hv[b.bit] = b.hash;
    s.gate_of[b.bit] = (unsigned char)b.gate;
    atomicOr(&s.pm[b.bit >> 6], 1ull << (b.bit & 63));
  }
  __syncthreads();
}

// Where finished rows go: into the bins of window `w` (layout `l`, buffer
// `buf`, counters `cnt`), or dense.
template <int W>
struct Dest {
  bool dense;
  Layout l;
  u64* keys;
  double* coeffs;
  u32* h;
  u32* cnt;
  u32* spill_bin;
  u64 room;        // rows of the buffer (bins, then spills)
  u32* n_spill;    // spilled rows
  u64* n_dense;    // dense: rows written
  u32* fail;       // set when the buffer is full
};

template <int W, int ALG, class S>
__device__ __forceinline__ void put_row(const S& s, const Dest<W>& d, const u64* k, double c, u32 h, bool act,
                                        const GateDesc<W>* gates, const WinDesc& w) {
  u64 at;
  if (d.dense) {
    const unsigned m = __ballot_sync(FULL, act);
    if (!m) return;
    const int lane = threadIdx.x & 31;
    u64 base = 0;
    if (lane == 0) base = atomicAdd(d.n_dense, (u64)__popc(m));
    at = __shfl_sync(FULL, base, 0) + __popc(m & ((1u << lane) - 1u));
    if (!act) return;
    if (at >= d.room) {
      *d.fail = 1;
      return;
    }
  } else {
    if (!act) return;
    const u32 bin = bin_of(group_hash<W, ALG>(s, k, h, gates, w), d.l.bins);
    const u32 pos = atomicAdd(d.cnt + (u64)bin * d.l.stride, 1u);
    if (pos < d.l.cap) {
      at = (u64)bin * d.l.cap + pos;
    } else {
      const u64 first = (u64)d.l.bins * d.l.cap;
      const u32 sp = atomicAdd(d.n_spill, 1u);
      at = first + sp;
      if (at >= d.room) {
        *d.fail = 1;
        return;
      }
      d.spill_bin[sp] = bin;
    }
    d.h[at] = h;
  }
  store_key<W>(d.keys, at, k);
  d.coeffs[at] = c;
}

template <int W, int ALG, class S>
__device__ __forceinline__ void bins_body(const BinArgs& a, const Grp grp, S& s) {
  using Ops = typename Alg<ALG>::T;
  constexpr int T = S::T;
  const int tid = threadIdx.x, lane = tid & 31;
  const bool fetcher = tid >= T - 32;
  SweepState* st = a.st;
  BinState* bs = a.bs;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  u32 gen = *(volatile u32*)&st->bar_gen;
  if (a.hold_us && grp.bid == a.hold_block && tid == 0) hold(a.hold_us);

  // Position: the window, the first rotation of it still to run, the buffer
  // and counter set holding the rows (ph), or the dense rows at entry.
  const bool resumed = a.resume != 0;
  const u32 op_start = resumed ? bs->op : *(volatile u32*)&st->end_op;
  u64 N = resumed ? bs->rows : ld_volatile(&st->n[0]);
  u32 win = a.n_windows, first = 0;
  {  // the window op_start lies in (windows cover every op in order)
    u32 lo = 0, hi = a.n_windows;
    while (lo < hi) {
      const u32 mid = (lo + hi) / 2;
      if (a.windows[mid].op_end <= op_start) lo = mid + 1;
      else hi = mid;
    }
    win = lo;
  }
  if (win >= a.n_windows) return;  // nothing left (the dense rows are the result)
  {
    const WinDesc& w0 = a.windows[win];
    first = op_start > w0.op ? op_start - w0.op : 0;
  }
  u32 ph = resumed ? bs->phase : 0;
  Layout lay = resumed ? Layout{bs->bins, bs->stride, bs->cap} : Layout{0, 0, 0};
  float rho = resumed ? bs->rho : 1.5f;  // growth of the live count inside recent windows

  auto dest_bins = [&](u32 set, const Layout& l) {
    Dest<W> d;
    d.dense = false;
    d.l = l;
    d.keys = a.bin_keys[set & 1];
    d.coeffs = a.bin_coeffs[set & 1];
    d.h = a.bin_hash[set & 1];
    d.cnt = a.counts + (u64)(set % 3) * a.count_words;
    d.spill_bin = a.spill_bin[set & 1];
    d.room = a.room[set & 1];
    d.n_spill = &bs->n_spill[set % 3];
    d.n_dense = nullptr;
    d.fail = &bs->fail[set % 3];
    return d;
  };
  auto rows_per_bin = [&] {
    return (u32)((float)S::R / fminf(fmaxf(1.5f, 1.15f * rho), 3.0f));
  };
  // `ph` counts buffer fills: set ph lives in buffer ph & 1, counters ph % 3.
  if (!resumed) {
    // Deal the dense rows into the bins of the first window.
    const WinDesc w = a.windows[win];
    lay = choose_layout(N, rows_per_bin(), grp.nblk, a.room[0]);
    load_grouping<W>(s, a, w);
    const Dest<W> d = dest_bins(0, lay);
    for (u64 r0 = (u64)grp.bid * T; r0 < N; r0 += (u64)grp.nblk * T) {
      const u64 r = r0 + tid;
      u64 k[W];
      double c = 0.0;
      u32 h = 0;
      if (r < N) {
        load_key<W>(a.keys, r, k);
        c = __ldcg(a.coeffs + r);
        h = lin_hash<W>(k, a.lin);
      }
      put_row<W, ALG>(s, d, k, c, h, r < N, gates, w);
    }
    grid_barrier(st, gen, grp);
    if (*(volatile u32*)&st->error) return;
    if (*(volatile u32*)&bs->fail[0]) {  // the first buffer is too small: the dense rows are untouched
      if (grp.bid == 0 && tid == 0) {
        bs->stopped = 1;
        bs->dense_start = 1;
        bs->op = op_start;
        bs->rows = N;
      }
      return;
    }
  }

  for (;;) {
    const WinDesc w = a.windows[win];
    const bool last = win + 1 >= a.n_windows;
    const WinDesc wn = last ? WinDesc{} : a.windows[win + 1];
    const u32 set = ph, nset = ph + 1;
    const u32* cnt = a.counts + (u64)(set % 3) * a.count_words;
    const u64* bk = a.bin_keys[set & 1];
    const double* bc = a.bin_coeffs[set & 1];
    const u32* bh = a.bin_hash[set & 1];
    const u32* bsp = a.spill_bin[set & 1];
    const u64 spill0 = (u64)lay.bins * lay.cap;
    Dest<W> d;
    Layout nlay = lay;
    if (last) {
      d = Dest<W>{};
      d.dense = true;
      d.keys = a.keys;
      d.coeffs = a.coeffs;
      d.room = a.dense_room;
      d.n_dense = &bs->n_dense;
      d.fail = &bs->fail[nset % 3];
    } else {
      nlay = choose_layout(w.noise == 2 ? N : N + N / 2, rows_per_bin(), grp.nblk, a.room[nset & 1]);
      d = dest_bins(nset, nlay);
      load_grouping<W>(s, a, wn);
    }
    const u32 G = w.n_gates;
    for (u32 i = tid; i < WIN_MAX; i += T) s.born_all[i] = s.anti_all[i] = 0;
    if (tid == 0) s.kept = 0;
    const u32 spilled = *(volatile u32*)&bs->n_spill[set % 3];
    const double* factors = a.tables + (u64)w.table * a.table_len;
    const u32 lastw = a.table_len ? a.table_len - 1 : 0;
    BinRules R;
    R.n_units = a.n_units;
    R.minc = a.min_coeff;
    R.wcut = a.max_weight;
    R.ccut = a.has_min_coeff != 0;

    // A finished row: the reclaim after the window, then its next bin.
    u32 kept = 0;
    auto finish_row = [&](u64* k, double c, u32 h, bool act) {
      if (act && w.noise) {
        const u32 wt = Ops::template weight<W>(k, a.n_units);
        c = __dmul_rn(c, __ldg(factors + (wt < lastw ? wt : lastw)));
        if (w.noise == 2)
          act = (a.max_weight == NO_WEIGHT_CUT || wt <= a.max_weight) && (!a.has_min_coeff || fabs(c) >= a.min_coeff);
      }
      kept += act;
      put_row<W, ALG>(s, d, k, c, h, act, gates, wn);
    };

    const bool dynamic = lay.bins > grp.nblk;
    u32 bin = grp.bid, depth0 = 0;
    __syncthreads();
    for (;;) {
      if (dynamic) {
        if (tid == 0) s.tick = atomicAdd(&bs->ticket[set % 3], 1u);
        __syncthreads();
        bin = s.tick;
        __syncthreads();
      }
      if (bin >= lay.bins) break;
      const u32 n_all = __ldcg(cnt + (u64)bin * lay.stride);
      const u32 n_bin = n_all < lay.cap ? n_all : lay.cap;
      const bool has_spill = n_all > lay.cap;
      const u64 row0 = (u64)bin * lay.cap;
      if (G == 0 || first >= G) {
        // no rotation: straight through
        for (u32 r0 = 0; r0 < n_bin; r0 += T) {
          const u32 r = r0 + tid;
          u64 k[W];
          double c = 0.0;
          u32 h = 0;
          if (r < n_bin) {
            load_key<W>(bk, row0 + r, k);
            c = __ldcg(bc + row0 + r);
            h = __ldcg(bh + row0 + r);
          }
          finish_row(k, c, h, r < n_bin);
        }
        for (u32 r0 = 0; has_spill && r0 < spilled; r0 += T) {
          const u32 r = r0 + tid;
          const bool mine = r < spilled && __ldcg(bsp + r) == bin;
          u64 k[W];
          double c = 0.0;
          u32 h = 0;
          if (mine) {
            load_key<W>(bk, spill0 + r, k);
            c = __ldcg(bc + spill0 + r);
            h = __ldcg(bh + spill0 + r);
          }
          finish_row(k, c, h, mine);
        }
      } else if (n_all) {
        // Parts of the bin: `part` of 2^depth by split_bits, in order.
        u32 depth = depth0, part = 0;
        while (depth < 24 && (n_all >> depth) > (u32)S::R * 7 / 8) ++depth;
        const u32 base = depth;
        for (;;) {
          for (u32 i = tid; i < G; i += T) s.born[i] = s.anti[i] = 0;
          for (int i = tid; i < S::SLOTS / 4; i += T)
            reinterpret_cast<uint4*>(s.tab)[i] = make_uint4(TAB_EMPTY, TAB_EMPTY, TAB_EMPTY, TAB_EMPTY);
          if (tid == 0) s.n = s.n_list[0] = s.n_list[1] = 0;
          if (fetcher) {
            for (u32 g = first; g < first + 2 && g < G; ++g) fetch_gate<W>(&s.gate[g & 3], gates + w.gate + g);
            cp_async_wait();
          }
          __syncthreads();
          u32 n = n_all;
          const bool whole = depth == 0 && !has_spill;
          if (whole) {
            for (u32 r = tid; r < n_bin; r += T) {
              u64 k[W];
              load_key<W>(bk, row0 + r, k);
              const double c = __ldcg(bc + row0 + r);
              const u32 h = __ldcg(bh + row0 + r);
#pragma unroll
              for (int x = 0; x < W; ++x) s.key[x][r] = k[x];
              s.coef[r] = c;
              s.h[r] = h;
              tab_insert(s, h, r, tab_start<S>(h));
            }
          } else {
            auto take = [&](u64 src) {
              u64 k[W];
              load_key<W>(bk, src, k);
              const u32 h = __ldcg(bh + src);
              if (depth && (split_bits(group_hash_list<W, ALG>(k, h, a, w)) >> (32 - depth)) != part) return;
              const u32 r = atomicAdd(&s.n, 1u);
              if (r >= (u32)S::R) return;
#pragma unroll
              for (int x = 0; x < W; ++x) s.key[x][r] = k[x];
              s.coef[r] = __ldcg(bc + src);
              s.h[r] = h;
              tab_insert(s, h, r, tab_start<S>(h));
            };
            for (u32 r = tid; r < n_bin; r += T) take(row0 + r);
            if (has_spill)
              for (u32 r = tid; r < spilled; r += T)
                if (__ldcg(bsp + r) == bin) take(spill0 + r);
            __syncthreads();
            n = s.n;
          }
          bool fits = n <= (u32)S::R;
          for (u32 g = first; fits && g < G; ++g) {
            if (fetcher) cp_async_wait_1();
            __syncthreads();
            if (g > first) {
              n += s.born[g - 1];
              if (n > (u32)S::R) {
                fits = false;
                break;
              }
            }
            if (fetcher) {
              if (g + 2 < G) fetch_gate<W>(&s.gate[(g + 2) & 3], gates + w.gate + g + 2);
              cp_async_commit();
            }
            rotate_rows<W, ALG>(s, s.gate[g & 3], R, n, g & 1, &s.born[g], &s.anti[g]);
          }
          if (fetcher) cp_async_wait();
          __syncthreads();
          if (fits) {
            n += s.born[G - 1];
            fits = n <= (u32)S::R;
          }
          if (!fits) {  // run the part again in halves
            ++depth;
            part <<= 1;
            if (depth0 < depth && depth0 < 8) depth0 = depth;
            if (depth > 24) {
              if (tid == 0) atomicOr(&st->error, ERR_CAPACITY);
              break;
            }
            __syncthreads();
            continue;
          }
          for (u32 i = tid; i < G; i += T) {
            s.born_all[i] += s.born[i];
            s.anti_all[i] += s.anti[i];
          }
          for (u32 r0 = 0; r0 < n; r0 += T) {
            const u32 r = r0 + tid;
            u64 k[W];
            double c = 0.0;
            u32 h = 0;
            if (r < n) {
#pragma unroll
              for (int x = 0; x < W; ++x) k[x] = s.key[x][r];
              c = s.coef[r];
              h = s.h[r];
            }
            finish_row(k, c, h, r < n);
          }
          __syncthreads();
          while (depth && (part & 1u)) {
            part >>= 1;
            --depth;
          }
          if (!depth) break;
          ++part;
          while (depth < base) {
            ++depth;
            part <<= 1;
          }
        }
      }
      if (!dynamic) break;
    }
    // Block totals: rows kept, rows created and rows branching per rotation.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) kept += __shfl_xor_sync(FULL, kept, o);
    if (lane == 0 && kept) atomicAdd(&s.kept, kept);
    __syncthreads();
    if (tid == 0 && s.kept) atomicAdd(&bs->n[nset % 3], (u64)s.kept);
    for (u32 i = tid; i < G; i += T) {
      if (s.born_all[i]) {
        atomicAdd(a.born + w.op + i, s.born_all[i]);
        atomicAdd(&bs->grown[nset % 3], (u64)s.born_all[i]);
      }
      if (s.anti_all[i]) atomicAdd(a.anti + w.op + i, (u64)s.anti_all[i]);
    }
    // The counter set after next: its last readers ran the window before this one.
    if (ph > a.phase0) {
      u32* z = a.counts + (u64)((ph + 2) % 3) * a.count_words;
      const Layout pl{s.x[6], s.x[7], 0};
      for (u32 b = grp.bid * T + tid; b < pl.bins; b += grp.nblk * T) z[(u64)b * pl.stride] = 0;
      if (grp.bid == 0 && tid == 0) {
        bs->n[(ph + 2) % 3] = 0;
        bs->grown[(ph + 2) % 3] = 0;
        bs->n_spill[(ph + 2) % 3] = 0;
        bs->ticket[(ph + 2) % 3] = 0;
      }
    }
    __syncthreads();
    if (tid == 0) {
      if (barrier_arrive(st, grp)) barrier_release(st, gen);
      else barrier_wait(st, gen);
      ++gen;
      const u64 nn = ld_volatile(&bs->n[nset % 3]), gr = ld_volatile(&bs->grown[nset % 3]);
      const u32 e = *(volatile u32*)&st->error, f = *(volatile u32*)&bs->fail[nset % 3];
      s.y[0] = nn;
      s.y[1] = gr;
      s.x[0] = e;
      s.x[1] = f;
      s.x[6] = lay.bins;
      s.x[7] = lay.stride;
    }
    __syncthreads();
    if (s.x[0]) return;
    if (s.x[1]) {  // the next buffer was too small: this window is run again after the host has grown it
      if (grp.bid == 0 && tid == 0) {
        bs->stopped = 1;
        bs->dense_start = 0;
        bs->op = w.op + first;
        bs->rows = N;
        bs->phase = ph;
        bs->bins = lay.bins;
        bs->stride = lay.stride;
        bs->cap = lay.cap;
        bs->rho = rho;
      }
      return;
    }
    const u64 nn = s.y[0];
    if (grp.bid == 0 && tid == 0) {
      if (w.noise) a.hist[w.op + G] = nn;
      u64 t;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
      a.stamps[w.op_end - 1] = t;
    }
    const float g = N ? (float)(N + s.y[1]) / (float)N : 1.0f;
    rho = fmaxf(g, 0.85f * rho);
    N = nn;
    lay = nlay;
    first = 0;
    ++ph;
    ++win;
    if (win >= a.n_windows) break;
  }
  if (grp.bid == 0 && tid == 0) {
    st->n[0] = N;
    st->end_op = a.windows[a.n_windows - 1].op_end;
  }
}
