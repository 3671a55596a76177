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
//     of the window's generators, of rank at most BIN_RANK (less on registers
//     whose key space can fill up): a group has at
//     most 2^rank keys, so one always fits in shared memory;
//   * disjoint windows: Pauli generators on pairwise disjoint qubits (they
//     commute; the rotations by pi among them may lie across any of them, and
//     change no key).  K is reduced only by the generators it anticommutes with --
//     the set no rotation of the window changes -- so their number is not
//     limited: a weight cut of at most BIN_RANK bounds that set's size, and
//     with it the group's, for every row.
//
// A bin that does not fit (its rows, or the rows it grows to) is run again in
// halves by further bits of the group hash, as often as it takes; nothing of
// a bin is written before all of it has fitted.  Two groups of one 32-bit hash
// cannot be told apart (a few pairs among 300,000 groups, or keys that differ
// by a kernel vector of the hash): if they do not fit together the run goes to
// the row sweep.  A window whose rows find their buffer too small stops; the
// host grows the buffer and the window is run again.
//
// Who takes a bin follows the rows per bin: while a bin of every warp of the
// grid holds the live set, each warp runs bins of its own, with no block
// barrier anywhere in a window (and hands a bin that outgrows it to its
// block); larger live sets go by blocks.  Small live sets run in one warp,
// then one block, with no grid barrier at all (solo_run).  Windows whose
// rotations all commute keep the set of rotations a term anticommutes with
// fixed, so a bin of a few rows runs only the rotations one of them
// anticommutes with.
//
// What bounds it: the dependent shared-memory round trips of a rotation's
// step (about 1 us on small bins; 2-3 us where a block's 1,500-3,000 rows
// branch often), no longer the grid barrier or DRAM.  Whole calls, row sweep
// -> binned sweep, on one box: 4-qubit circuit, 40 noisy rotations 0.68 ->
// 0.32 ms; 20-qubit TFIM (to 31k rows) 1.8 -> 0.80 ms; kicked Ising 10x10 x 20
// steps (4-word keys, to 476k rows) 23.6 -> 8.1 ms, 6x6 x 8 (2 words, to over
// 1M) 9.3 -> 2.7 ms, 12x15 x 8 (8 words) 32 -> 6.3 ms; Givens circuits of 24
// sites (15M rows) 44 -> 14 ms and 32 sites (99M rows) 428 -> 117 ms.
#pragma once

constexpr u32 TAB_EMPTY = 0xffffffffu;
constexpr u32 IDX_BITS = 13;  // row index bits of a shared-memory table slot, the rest is fingerprint
constexpr u32 IDX_MASK = (1u << IDX_BITS) - 1u;

// Rows of one unit -- a block (T = its threads) or a warp (T = 32).
template <int W, int T_, int R_, int SLOTS_>
struct BinSmem {
  static constexpr int T = T_, R = R_, SLOTS = SLOTS_;
  static_assert(R < (int)IDX_MASK && R <= 32 * T, "a table slot holds a row index, a thread 32 row bits");
  double coef[R];
  u64 key[W][R];  // by word: lanes of consecutive rows read consecutive addresses
  u32 h[R];
  __align__(16) u32 tab[SLOTS];
  __align__(16) GateDesc<W> gate[4];  // ring: the running rotation and the next two
  u32 born[WIN_MAX];             // this bin, per rotation: rows created
  unsigned short anti[WIN_MAX];  // ... rows anticommuting
  unsigned short list[R];        // the running rotation's anticommuting rows
  u32 n_list[2];                 // their number; the other one is zero for the next rotation
  u32 act[WIN_MAX / 32];         // rotations to run (commuting windows, few rows)
  __align__(8) WinDesc win[4];   // ring (solo): the running window and the next two
  u32 n, quit;
};

template <class S>
__device__ __forceinline__ void unit_sync() {
  if constexpr (S::T == 32) __syncwarp();
  else __syncthreads();
}
template <class S>
__device__ __forceinline__ int unit_tid() {
  if constexpr (S::T == 32) return threadIdx.x & 31;
  else return threadIdx.x;
}

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
  constexpr u32 PAIRS = S::SLOTS / 2;
  static_assert((PAIRS & (PAIRS - 1)) == 0, "table size");
  return (h * 0xC2B2AE35u) / (u32)(0x100000000ull / PAIRS);
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
// the caller sees n grow past R.  Run by the whole unit; the caller's barrier
// ends it.
//
// Every row in a run without a TermBudget floor is within the weight cut (the
// admission, each branch and each reclaim keep to it), so in a pair only the
// coefficient check can hold a branch back: S_DROP arises for a lone row's
// child alone.
template <int W, int ALG, class S>
__device__ __forceinline__ void rotate_rows(S& s, const GateDesc<W>& d, const BinRules& R, u32 n, u32 flip_flop,
                                            u32* born, unsigned short* anti) {
  using Ops = typename Alg<ALG>::T;
  constexpr int T = S::T, U = 4;
  const int tid = unit_tid<S>(), lane = tid & 31, warp = tid >> 5;
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
  unit_sync<S>();
  const u32 total = s.n_list[flip_flop];
  if (tid == 0) {
    s.n_list[flip_flop ^ 1] = 0;
    *anti = (unsigned short)total;
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

// Descriptors on their way into the ring (cp.async), by the unit's last warp,
// which has rows of its own only when the unit is nearly full: its waits
// overlap the other warps' work.
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

template <class S>
__device__ __forceinline__ void clear_table(S& s) {
  for (int i = unit_tid<S>(); i < S::SLOTS / 4; i += S::T)
    reinterpret_cast<uint4*>(s.tab)[i] = make_uint4(TAB_EMPTY, TAB_EMPTY, TAB_EMPTY, TAB_EMPTY);
}

// Which rotations [first, G) of a commuting window to run, for few rows: those
// some row anticommutes with (the rows they create anticommute with the same
// ones).  Between barriers of the caller.  A lane tests one rotation against
// every row.
constexpr u32 ACT_ROWS = 64;
template <int W, int ALG, class S>
__device__ __forceinline__ void find_active(S& s, const GateDesc<W>* gates, u32 first, u32 G, u32 n) {
  for (u32 g0 = first & ~31u; g0 < WIN_MAX; g0 += S::T) {
    const u32 g = g0 + unit_tid<S>();
    bool on = false;
    if (g >= first && g < G) {
      u64 am[W];
#pragma unroll
      for (int w = 0; w < W; ++w) am[w] = anti_word<W, ALG>(gates[g], w);
      for (u32 r = 0; r < n && !on; ++r) {
        u64 acc = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) acc ^= s.key[w][r] & am[w];
        on = popc(acc) & 1;
      }
    }
    const unsigned m = __ballot_sync(FULL, on);
    if ((threadIdx.x & 31) == 0 && g < WIN_MAX) s.act[g >> 5] = m;
  }
}
// The next rotation to run from g on (G: none).  `some`: by s.act, else all.
template <class S>
__device__ __forceinline__ u32 next_gate(const S& s, bool some, u32 g, u32 G) {
  if (!some || g >= G) return g < G ? g : G;
  u32 w = g >> 5, m = s.act[w] & (~0u << (g & 31u));
  while (!m) {
    if (++w * 32 >= G) return G;
    m = s.act[w];
  }
  g = 32 * w + __ffs(m) - 1;
  return g < G ? g : G;
}

// ------------------------------------------------------------ solo
// One unit runs windows from (win, first) on while the rows fit it (a rotation
// may double them), from and to the dense rows.  Returns with win / first at
// the rotation it stopped before (win == n_windows at the end) and n the live
// count.  Its rows must number at most R / 2 at entry.
template <int W, int ALG, class S>
__device__ __noinline__ void solo_run(const BinArgs& a, S& s, u32& win, u32& first, u32& n_io) {
  using Ops = typename Alg<ALG>::T;
  constexpr int T = S::T;
  constexpr u32 NONE = 0xffffffffu;
  const int tid = unit_tid<S>(), lane = tid & 31;
  const bool fetcher = tid >= T - 32;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  u32 n = n_io;
  auto fetch_window = [&](u32 x) {  // by the fetcher: window x into its place of the ring
    constexpr u32 WORDS = sizeof(WinDesc) / 8;
    if (x < a.n_windows && lane < (int)WORDS)
      cp_async8(reinterpret_cast<u64*>(&s.win[x & 3]) + lane, reinterpret_cast<const u64*>(a.windows + x) + lane);
  };
  clear_table(s);
  if (tid < 4) s.born[tid] = 0;
  if (tid < 2) s.n_list[tid] = 0;
  if (fetcher) {
    fetch_window(win);
    fetch_window(win + 1);
    cp_async_wait();
  }
  unit_sync<S>();
  for (u32 r = tid; r < n; r += T) {
    u64 k[W];
    load_key<W>(a.keys, r, k);
    const u32 h = lin_hash<W>(k, a.lin);
#pragma unroll
    for (int w = 0; w < W; ++w) s.key[w][r] = k[w];
    s.coef[r] = __ldcg(a.coeffs + r);
    s.h[r] = h;
    tab_insert(s, h, r, tab_start<S>(h));
  }
  BinRules R;
  R.n_units = a.n_units;
  R.minc = a.min_coeff;
  R.wcut = a.max_weight;
  R.ccut = a.has_min_coeff != 0;
  u32 step = 0;          // rotations run: counters born / anti [step & 3], descriptor gate[step & 3]
  u32 last = NONE;       // op whose counters are in [(step - 1) & 3], not yet taken
  u32 pa = NONE, pb = NONE;  // descriptors on their way for this step and the next
  // The live count after the last rotation; thread 0 records its counters.
  auto take = [&] {
    if (last == NONE) return;
    const u32 b = s.born[(step - 1) & 3];
    n += b;
    if (tid == 0) {
      a.born[last] = b;
      a.anti[last] = s.anti[(step - 1) & 3];
    }
    last = NONE;
  };
  bool stop = false;
  while (win < a.n_windows) {
    // Fetched while the window before the last began; every window waits for
    // all but its latest fetch and then meets a barrier, so it is here.
    bool met = false;
    const WinDesc& w = s.win[win & 3];
    if (fetcher) {
      fetch_window(win + 2);
      cp_async_commit();
    }
    const u32 G = w.n_gates;
    if (first < G) {
      bool some = false;
      if (w.commute && G - first > 4) {
        unit_sync<S>();
        take();
        some = n <= ACT_ROWS;
        if (some) {
          find_active<W, ALG>(s, gates + w.gate, first, G, n);
          unit_sync<S>();
        }
      }
      u32 g = next_gate(s, some, first, G);
      while (g < G) {
        const u32 g1 = next_gate(s, some, g + 1, G), g2 = next_gate(s, some, g1 + 1, G);
        const u32 id = w.gate + g, id1 = w.gate + (g1 < G ? g1 : G), id2 = g1 < G ? w.gate + (g2 < G ? g2 : G) : id1 + 1;
        if (pa != id) {  // not the one that was expected: now, with the next
          if (fetcher) {
            cp_async_wait();
            fetch_gate<W>(&s.gate[step & 3], gates + id);
            if (id1 < a.n_gdesc) fetch_gate<W>(&s.gate[(step + 1) & 3], gates + id1);
            cp_async_wait();
          }
          pb = id1;
        } else if (fetcher) {
          cp_async_wait_1();
        }
        unit_sync<S>();  // the step before is done; this rotation's descriptor is here
        met = true;
        take();
        if (2 * n > (u32)S::R) {
          stop = true;
          break;
        }
        if (fetcher) {
          if (id2 < a.n_gdesc) fetch_gate<W>(&s.gate[(step + 2) & 3], gates + id2);
          cp_async_commit();
        }
        pa = pb;
        pb = id2;
        if (tid == 0) s.born[(step + 2) & 3] = 0;
        rotate_rows<W, ALG>(s, s.gate[step & 3], R, n, step & 1, &s.born[step & 3], &s.anti[step & 3]);
        last = w.op + g;
        ++step;
        g = g1;
      }
      first = g;
      if (stop) break;
    }
    if (w.noise) {
      if (fetcher) cp_async_wait_1();
      unit_sync<S>();
      met = true;
      take();
      const double* factors = a.tables + (u64)w.table * a.table_len;
      const u32 lastw = a.table_len - 1;
      const bool reclaim = w.noise == 2;
      if (reclaim) {
        if (tid == 0) s.n = 0;
        clear_table(s);
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
          for (int x = 0; x < W; ++x) k[x] = s.key[x][r];
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
        unit_sync<S>();
        const unsigned m = __ballot_sync(FULL, kp);
        if (!m) continue;
        u32 at = 0;
        if (lane == 0) at = atomicAdd(&s.n, (u32)__popc(m));
        at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (!kp) continue;
#pragma unroll
        for (int x = 0; x < W; ++x) s.key[x][at] = k[x];
        s.coef[at] = c;
        s.h[at] = h;
        tab_insert(s, h, at, tab_start<S>(h));
      }
      if (reclaim) {
        unit_sync<S>();
        n = s.n;
      }
      if (tid == 0) a.hist[w.op + G] = n;
    }
    // (reading the clock takes about as long as a rotation)
    if (tid == T - 1 && (win & 7u) == 7u) stamp_op(a.stamps, w.op_end - 1);
    if (!met) {
      if (fetcher) cp_async_wait_1();
      unit_sync<S>();
    }
    ++win;
    first = 0;
  }
  unit_sync<S>();
  take();
  if (fetcher) cp_async_wait();
  for (u32 r = tid; r < n; r += T) {
    u64 k[W];
#pragma unroll
    for (int x = 0; x < W; ++x) k[x] = s.key[x][r];
    store_key<W>(a.keys, r, k);
    a.coeffs[r] = s.coef[r];
  }
  n_io = n;
}

// The window op `op` lies in (windows cover every op in order).
__device__ __forceinline__ u32 window_of(const BinArgs& a, u32 op) {
  u32 lo = 0, hi = a.n_windows;
  while (lo < hi) {
    const u32 mid = (lo + hi) / 2;
    if (a.windows[mid].op_end <= op) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// A block alone: its first warp while the rows fit it, then all of it; leaves
// the op it stopped before in st->end_op and the live count in st->n[0].
template <int W, int ALG, class SW, class SB>
__device__ __forceinline__ void solo_body(const BinArgs& a, SW& sw, SB& sb) {
  SweepState* st = a.st;
  if (threadIdx.x == 0) stamp_op(a.stamps, a.op_end);  // the start
  u32 win = window_of(a, a.op_begin), first = 0, n = 0;
  if (win < a.n_windows && a.op_begin > a.windows[win].op) first = a.op_begin - a.windows[win].op;
  const u64 n0 = a.n0;
  if (n0 > (u64)SB::R / 2 || win >= a.n_windows) {
    if (threadIdx.x == 0) {
      st->n[0] = n0;
      st->end_op = win < a.n_windows ? a.op_begin : a.op_end;
    }
    return;
  }
  n = (u32)n0;
  if (n <= (u32)SW::R / 2) {
    __shared__ u32 hand[3];
    if (threadIdx.x < 32) {
      solo_run<W, ALG>(a, sw, win, first, n);
      if (threadIdx.x == 0) {
        hand[0] = win;
        hand[1] = first;
        hand[2] = n;
      }
    }
    __syncthreads();
    win = hand[0];
    first = hand[1];
    n = hand[2];
  }
  if (win < a.n_windows) solo_run<W, ALG>(a, sb, win, first, n);
  if (threadIdx.x == 0) {
    const u32 end = win < a.n_windows ? a.windows[win].op + first : a.op_end;
    st->n[0] = n;
    st->end_op = end;
    if (end > a.op_begin) stamp_op(a.stamps, end - 1);
  }
}

// ------------------------------------------------------------ binned windows
// (the layout of the bins: pq_layout.cuh)
__device__ __forceinline__ u32 bin_of(u32 g, u32 bins) { return __umulhi(g * 0x9E3779B1u, bins); }
// The bits a bin is split by when it does not fit.
__device__ __forceinline__ u32 split_bits(u32 g) { return (g ^ (g >> 15)) * 0x85EBCA6Bu; }

// Group hash from the basis list itself (the slow way: splits only).
template <int W, int ALG>
__device__ __noinline__ u32 group_hash_list(const u64* k, u32 h, const BinArgs& a, const WinDesc& w) {
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

// Where finished rows go: into the bins of the next window (layout `l`,
// counters `cnt`), or dense.
struct Dest {
  u64* keys;
  double* coeffs;
  u32* h;
  u32* cnt;
  u32* spill_bin;
  u32* n_spill;    // spilled rows
  u64* n_dense;    // dense (no bins): rows written
  u32* fail;       // set when the buffer is full
  u32* ticket;     // bins handed out in the window that fills it
  u64 room;        // rows that may spill; dense: rows of the buffer
  Layout l;
  u32 dense;
};

// What every unit of a block shares in a window.
template <int W>
struct WinSmem {
  u64 pm[W];       // pivot bits of the next window's grouping
  u32 hv[64 * W];  // per pivot bit: hash of its basis vector
  unsigned char gate_of[64 * W];  // per pivot bit: the next window's rotation it belongs to (disjoint windows)
  u32 born_all[WIN_MAX], anti_all[WIN_MAX];  // this block's bins, per rotation
  WinDesc w, wn;
  Dest d;
  // the rows of this window's bins
  const u64* bk;
  const double* bc;
  const u32* bh;
  const u32* bsp;
  const u32* cnt;
  u64 y[2];       // words read after the grid barrier
  u32 x[2];
  Layout lay, prev;
  u32 spilled, first;
  float grow;     // expected growth of this window's bins, at least 1
  u32 kept, tick, n_defer;
  u32 defer[32];  // bins the block's warps could not hold
};

template <int W, int ALG>
__device__ __forceinline__ u32 group_hash(const WinSmem<W>& v, const u64* k, u32 h, const GateDesc<W>* gates) {
#pragma unroll
  for (int x = 0; x < W; ++x)
    for (u64 m = k[x] & v.pm[x]; m; m &= m - 1) {
      const int bit = 64 * x + __ffsll((long long)m) - 1;
      if (v.wn.disjoint) {
        const GateDesc<W>& d = gates[v.wn.gate + v.gate_of[bit]];
        u64 acc = 0;
#pragma unroll
        for (int y = 0; y < W; ++y) acc ^= k[y] & __ldg(&d.g.fold[y]);
        if (!(popc(acc) & 1)) continue;
      }
      h ^= v.hv[bit];
    }
  return h;
}

// Loads the grouping of window v.wn (after v.wn is visible to the block).
template <int W>
__device__ __forceinline__ void load_grouping(WinSmem<W>& v, const BinArgs& a) {
  if (threadIdx.x < W) v.pm[threadIdx.x] = 0;
  __syncthreads();
  for (u32 i = threadIdx.x; i < v.wn.n_basis; i += blockDim.x) {
    const BasisDesc b = a.basis[v.wn.basis + i];
    v.hv[b.bit] = b.hash;
    v.gate_of[b.bit] = (unsigned char)b.gate;
    atomicOr(&v.pm[b.bit >> 6], 1ull << (b.bit & 63));
  }
  __syncthreads();
}

// No further bin is handed out: the window starts again in a larger buffer.
// The dense rows at the end are all counted first, so they are grown once.
__device__ __noinline__ void too_small(const Dest& d) {
  if (!*(volatile u32*)d.fail && !atomicExch(d.fail, 1u) && !d.dense) atomicAdd(d.ticket, NO_MORE_BINS);
}

template <int W, int ALG>
__device__ __forceinline__ void put_row(const WinSmem<W>& v, const u64* k, double c, u32 h, bool act,
                                        const GateDesc<W>* gates) {
  const Dest& d = v.d;
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
      too_small(d);
      return;
    }
  } else {
    if (!act) return;
    const u32 bin = bin_of(group_hash<W, ALG>(v, k, h, gates), d.l.bins);
    const u32 pos = atomicAdd(d.cnt + (u64)bin * d.l.stride, 1u);
    if (pos < d.l.cap) {
      at = (u64)bin * d.l.cap + pos;
    } else {
      const u32 sp = atomicAdd(d.n_spill, 1u);
      if (sp >= d.room) {
        too_small(d);
        return;
      }
      at = (u64)d.l.bins * d.l.cap + sp;
      d.spill_bin[sp] = bin;
    }
    d.h[at] = h;
  }
  store_key<W>(d.keys, at, k);
  d.coeffs[at] = c;
}

// A finished row (1 if it is kept): the reclaim after the window, then its
// next bin.  Called by whole warps.
template <int W, int ALG>
__device__ __forceinline__ u32 finish_row_body(const WinSmem<W>& v, const BinArgs& a, const u64 (&k)[W], double c,
                                               u32 h, bool act) {
  using Ops = typename Alg<ALG>::T;
  if (act && v.w.noise) {
    const u32 lastw = a.table_len - 1;
    const u32 wt = Ops::template weight<W>(k, a.n_units);
    c = __dmul_rn(c, __ldg(a.tables + (u64)v.w.table * a.table_len + (wt < lastw ? wt : lastw)));
    if (v.w.noise == 2)
      act = (a.max_weight == NO_WEIGHT_CUT || wt <= a.max_weight) && (!a.has_min_coeff || fabs(c) >= a.min_coeff);
  }
  put_row<W, ALG>(v, k, c, h, act, reinterpret_cast<const GateDesc<W>*>(a.gates));
  return act ? 1u : 0u;
}
template <int W, int ALG>
__device__ __noinline__ u32 finish_row_call(const WinSmem<W>& v, const BinArgs& a, const u64 (&k)[W], double c, u32 h,
                                            bool act) {
  return finish_row_body<W, ALG>(v, a, k, c, h, act);
}
// Inlined at its four places it makes the 4- and 8-word kernels spill (kicked
// Ising 12x15 4.6 -> 5.6 ms); a call costs the narrow ones (6x6 2.14 -> 2.24).
template <int W, int ALG>
__device__ __forceinline__ u32 finish_row(const WinSmem<W>& v, const BinArgs& a, const u64 (&k)[W], double c, u32 h,
                                          bool act) {
  if constexpr (W <= 2) return finish_row_body<W, ALG>(v, a, k, c, h, act);
  else return finish_row_call<W, ALG>(v, a, k, c, h, act);
}

// One bin by one unit: its rows into shared memory, the window's rotations,
// and every row on to its next place.  A block splits what does not fit; a
// warp returns false instead, having written nothing.  depth0: how deep this
// block's bins of the window have been split so far by parts that held no more
// than their share of the bin.  (Two full groups that agree in many split bits
// go deep by themselves: counted too, one such pair had the block run all its
// later bins in 256 parts, 22 rotations that double one row to 2^22 in 4.1 ms
// instead of 0.9.)
template <int W, int ALG, class S>
__device__ __forceinline__ bool run_bin(const BinArgs& a, WinSmem<W>& v, S& s, u32 bin, u32& depth0, u32& kept) {
  constexpr int T = S::T;
  constexpr bool WARP = T == 32;
  constexpr u32 NONE = 0xffffffffu;
  const int tid = unit_tid<S>();
  const bool fetcher = tid >= T - 32;
  const u32 n_all = __ldcg(v.cnt + (u64)bin * v.lay.stride);
  if (!n_all) return true;
  const u32 n_bin = n_all < v.lay.cap ? n_all : v.lay.cap;
  const bool has_spill = n_all > v.lay.cap;
  const u64 row0 = (u64)bin * v.lay.cap, spill0 = (u64)v.lay.bins * v.lay.cap;
  const u32 G = v.w.n_gates, first = v.first, spilled = v.spilled;
  if (first >= G) {  // no rotation: straight through
    for (u32 r0 = 0; r0 < n_bin + (has_spill ? spilled : 0u); r0 += T) {
      const u32 r = r0 + tid;
      const bool in_bin = r < n_bin;
      const u64 src = in_bin ? row0 + r : spill0 + (r - n_bin);
      const bool act = in_bin || (has_spill && r < n_bin + spilled && __ldcg(v.bsp + (r - n_bin)) == bin);
      u64 k[W];
      double c = 0.0;
      u32 h = 0;
      if (act) {
        load_key<W>(v.bk, src, k);
        c = __ldcg(v.bc + src);
        h = __ldcg(v.bh + src);
      }
      kept += finish_row<W, ALG>(v, a, k, c, h, act);
    }
    return true;
  }
  // A warp runs its bin whole or not at all (a part that did not fit after
  // another was written would be run twice).
  if (WARP && (has_spill || n_all > (u32)S::R / 2)) return false;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates) + v.w.gate;
  BinRules R;
  R.n_units = a.n_units;
  R.minc = a.min_coeff;
  R.wcut = a.max_weight;
  R.ccut = a.has_min_coeff != 0;
  // Parts of the bin: `part` of 2^depth by split_bits, in order.
  u32 depth = WARP ? 0 : depth0, part = 0;
  // split at once what would outgrow the unit at the expected growth: failing
  // late in a window of 80 rotations takes as long as running it
  while (!WARP && depth < 24 && (float)(n_all >> depth) * v.grow > (float)S::R * 0.9f) ++depth;
  // Nothing more is run once the next buffer turned out too small: the window
  // starts again when the host has grown it.
  auto given_up = [&] {
    if (tid == 0) s.quit = !v.d.dense && *(volatile u32*)v.d.fail;
    unit_sync<S>();
    return s.quit != 0;
  };
  const u32 base = depth;
  u32 failed = 0;  // rows of the part that failed last: a half that holds them all fails too
  for (;;) {
    for (u32 i = tid; i < G; i += T) {
      s.born[i] = 0;
      s.anti[i] = 0;
    }
    clear_table(s);
    if (tid == 0) s.n = s.n_list[0] = s.n_list[1] = 0;
    unit_sync<S>();
    u32 n = n_all;
    if (depth == 0 && !has_spill) {
      for (u32 r = tid; r < n_bin; r += T) {
        u64 k[W];
        load_key<W>(v.bk, row0 + r, k);
        const double c = __ldcg(v.bc + row0 + r);
        const u32 h = __ldcg(v.bh + row0 + r);
#pragma unroll
        for (int x = 0; x < W; ++x) s.key[x][r] = k[x];
        s.coef[r] = c;
        s.h[r] = h;
        tab_insert(s, h, r, tab_start<S>(h));
      }
    } else {
      auto take = [&](u64 src) {
        u64 k[W];
        load_key<W>(v.bk, src, k);
        const u32 h = __ldcg(v.bh + src);
        if (depth && (split_bits(group_hash_list<W, ALG>(k, h, a, v.w)) >> (32 - depth)) != part) return;
        const u32 r = atomicAdd(&s.n, 1u);
        if (r >= (u32)S::R) return;
#pragma unroll
        for (int x = 0; x < W; ++x) s.key[x][r] = k[x];
        s.coef[r] = __ldcg(v.bc + src);
        s.h[r] = h;
        tab_insert(s, h, r, tab_start<S>(h));
      };
      for (u32 r = tid; r < n_bin; r += T) take(row0 + r);
      if (has_spill)
        for (u32 r = tid; r < spilled; r += T)
          if (__ldcg(v.bsp + r) == bin) take(spill0 + r);
      unit_sync<S>();
      n = s.n;
    }
    const u32 n_load = n;
    bool fits = n <= (u32)S::R && (!n || n != failed);
    if (fits && n) {
      const bool some = v.w.commute && n <= ACT_ROWS;
      if (some) {
        unit_sync<S>();
        find_active<W, ALG>(s, gates, first, G, n);
        unit_sync<S>();
      }
      u32 g = next_gate(s, some, first, G), before = NONE, step = 0;
      u32 g1 = next_gate(s, some, g + 1, G);
      if (fetcher && g < G) {
        fetch_gate<W>(&s.gate[0], gates + g);
        if (g1 < G) fetch_gate<W>(&s.gate[1], gates + g1);
        cp_async_wait();
      }
      for (; g < G; ++step) {
        if (fetcher) cp_async_wait_1();
        unit_sync<S>();
        if (before != NONE) {
          n += s.born[before];
          if (n > (u32)S::R) {
            fits = false;
            break;
          }
        }
        const u32 g2 = next_gate(s, some, g1 + 1, G);
        if (fetcher) {
          if (g2 < G) fetch_gate<W>(&s.gate[(step + 2) & 3], gates + g2);
          cp_async_commit();
        }
        rotate_rows<W, ALG>(s, s.gate[step & 3], R, n, step & 1, &s.born[g], &s.anti[g]);
        before = g;
        g = g1;
        g1 = g2;
      }
      if (fetcher) cp_async_wait();
      unit_sync<S>();
      if (fits && before != NONE) {
        n += s.born[before];
        fits = n <= (u32)S::R;
      }
    }
    if (!fits) {
      if (WARP) return false;
      failed = n_load;
      const bool fair = n_load <= (n_all >> depth) + (n_all >> (depth + 2));
      ++depth;  // run the part again in halves
      if (fair && depth0 < depth && depth <= 8) depth0 = depth;
      part <<= 1;
      if (depth > 24) {
        if (tid == 0) atomicOr(&a.st->error, ERR_CAPACITY);
        return true;
      }
      if (given_up()) return true;
      continue;
    }
    if (n) failed = 0;
    for (u32 i = tid; n && i < G; i += T) {
      if (s.born[i]) atomicAdd(&v.born_all[i], s.born[i]);
      if (s.anti[i]) atomicAdd(&v.anti_all[i], (u32)s.anti[i]);
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
      kept += finish_row<W, ALG>(v, a, k, c, h, r < n);
    }
    unit_sync<S>();
    while (depth && (part & 1u)) {
      part >>= 1;
      --depth;
    }
    if (!depth) return true;
    ++part;
    while (depth < base) {
      ++depth;
      part <<= 1;
    }
    if (given_up()) return true;
  }
}

// Bins of fill number `fill` (buffer fill & 1, counter set fill % 3) as a destination.
__device__ __forceinline__ Dest dest_bins(const BinArgs& a, u32 fill, const Layout& l) {
  BinState* bs = a.bs;
  Dest d;
  d.dense = 0;
  d.l = l;
  d.keys = a.bin_keys[fill & 1];
  d.coeffs = a.bin_coeffs[fill & 1];
  d.h = a.bin_hash[fill & 1];
  d.cnt = a.counts + (u64)(fill % 3) * a.count_words;
  d.spill_bin = a.spill_bin[fill & 1];
  d.room = spill_room(l, a.room[fill & 1]);
  if (a.spill_limit && d.room > spill_limit(a.room[fill & 1])) d.room = spill_limit(a.room[fill & 1]);
  d.n_spill = &bs->n_spill[fill % 3];
  d.n_dense = nullptr;
  d.fail = &bs->fail[fill % 3];
  d.ticket = &bs->ticket[(fill + 2) % 3];  // of the window before
  return d;
}

// A layout is made before the window that fills it has run.  A sweep whose
// rows came to more than this many times what their bins hold stops, and they
// are dealt again by their actual number (deal_body): one pass over the rows,
// where bins that are split into four parts and more are read as many times.
// (On 2^26 rows of 4-word keys and 2^25 of 1-word keys in the bins of a few
// thousand, the two rotations after a doubling window took 3,031 and 64 ms;
// the calls around them now take 22 and 8.)  A kernel of its own: a pass of
// this kind inside bins_body cost the 24-site Givens circuit 4% (10.95 ->
// 11.41 ms) in registers that every window's rotations need.
constexpr float REDEAL = 2.0f;

// The rows of the bins `from`, fill number `fill`, into the bins `to` of the
// next fill, grouped for window `win`.
template <int W, int ALG, int T>
__device__ __forceinline__ void deal_body(const BinArgs& a, WinSmem<W>& v, u32 win, u32 fill, const Layout& from,
                                          const Layout& to) {
  const int tid = threadIdx.x;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  if (tid == 0) {
    v.wn = a.windows[win];
    v.d = dest_bins(a, fill + 1, to);
  }
  __syncthreads();
  load_grouping<W>(v, a);
  auto put = [&](u64 src, bool act) {
    u64 k[W];
    double c = 0.0;
    u32 h = 0;
    if (act) {
      load_key<W>(a.bin_keys[fill & 1], src, k);
      c = __ldcg(a.bin_coeffs[fill & 1] + src);
      h = __ldcg(a.bin_hash[fill & 1] + src);
    }
    put_row<W, ALG>(v, k, c, h, act, gates);
  };
  const u32* cnt = a.counts + (u64)(fill % 3) * a.count_words;
  for (u32 b = blockIdx.x; b < from.bins; b += gridDim.x) {
    const u32 all = __ldcg(cnt + (u64)b * from.stride), n = all < from.cap ? all : from.cap;
    for (u32 r0 = 0; r0 < n; r0 += T) put((u64)b * from.cap + r0 + tid, r0 + tid < n);
  }
  const u32 spilled = a.bs->n_spill[fill % 3];
  for (u64 r0 = (u64)blockIdx.x * T; r0 < spilled; r0 += (u64)gridDim.x * T)
    put((u64)from.bins * from.cap + r0 + tid, r0 + tid < spilled);
}

// The windows from where the solo run (or a stopped sweep) left off, by the
// blocks of grp.  SB: a block's rows, SW: a warp's; both lie over one another
// in `rows`.
template <int W, int ALG, class SB, class SW>
__device__ __forceinline__ void bins_body(const BinArgs& a, const Grp grp, WinSmem<W>& v, SB& sb, SW* sw) {
  constexpr int T = SB::T, WARPS = T / 32;
  const int tid = threadIdx.x, lane = tid & 31;
  SweepState* st = a.st;
  BinState* bs = a.bs;
  const GateDesc<W>* gates = reinterpret_cast<const GateDesc<W>*>(a.gates);
  u32 gen = *(volatile u32*)&st->bar_gen;
  if (a.hold_us && grp.bid == a.hold_block && tid == 0) hold(a.hold_us);

  // Position: the window, the first rotation of it still to run, and the
  // number of buffer fills so far: fill ph lies in buffer ph & 1, its counters
  // in set ph % 3.
  const bool resumed = a.resume != 0;
  const u32 op_start = resumed ? bs->op : *(volatile u32*)&st->end_op;
  u64 N = resumed ? bs->rows : ld_volatile(&st->n[0]);
  u32 win = window_of(a, op_start);
  if (win >= a.n_windows) return;  // nothing left (the dense rows are the result)
  u32 first = op_start > a.windows[win].op ? op_start - a.windows[win].op : 0;
  u32 ph = resumed ? bs->phase : 0;
  Layout lay = resumed ? Layout{bs->bins, bs->stride, bs->cap} : Layout{0, 0, 0};

  // The layout for window x, entered by about n rows.  How they will grow: as
  // in an earlier window of the same rotations (host: WinDesc::like), if that
  // was entered by about as many rows, else as in the windows just before.
  // Bins 85% full where that is known and steady.  Less where the growth is
  // steep, for then it is uneven (kicked Ising 6x6, x18 in an RX layer: 381
  // -> 214 us at 45%), or not known, the more so the longer the window: a bin
  // that does not fit after all is run again in halves.
  float rho = resumed ? bs->rho : 1.5f;
  auto alike = [&](float n, u32 x) -> const float* {
    const u32 like = a.windows[x].like;
    if (like == 0xffffffffu) return nullptr;
    const float* h = a.growth + 3 * like;
    const float was = __ldcg(h + 2);
    return was > 0.0f && n < 8.0f * was && was < 8.0f * n ? h : nullptr;
  };
  float next_grow = resumed ? bs->grow : 1.0f;  // expected growth of the window dealt to last
  auto layout_for = [&](float n, u32 x, u64 room) {
    const float* h = alike(n, x);
    const float g = h ? fmaxf(__ldcg(h), 1.0f) : fminf(fmaxf(1.15f * rho, 1.5f), 3.0f);
    next_grow = 1.0f + 0.5f * (g - 1.0f);  // bins differ: followed half way
    const float fill = h ? (g < 3.0f ? 0.85f : 0.3f) : (a.windows[x].n_gates < 24 ? 1.0f : 0.7f);
    return choose_layout(n, g, fill, grp.nblk, WARPS, SB::R, room);
  };
  if (!resumed) {
    if (grp.bid == 0 && tid == 0) {  // where the grid began
      stamp_op(a.stamps, a.op_end + 1);
      a.stamps[a.op_end + 2] = op_start + 1;
    }
    // Deal the dense rows into the bins of the first window.
    lay = layout_for((float)N, win, a.room[0]);
    if (tid == 0) {
      v.wn = a.windows[win];
      v.d = dest_bins(a, 0, lay);
    }
    __syncthreads();
    load_grouping<W>(v, a);
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
      put_row<W, ALG>(v, k, c, h, r < N, gates);
    }
    grid_barrier(st, gen, grp);
    if (*(volatile u32*)&st->error) return;
    if (*(volatile u32*)&bs->fail[0]) {  // the first buffer is too small: the dense rows are untouched
      if (grp.bid == 0 && tid == 0) {
        bs->stopped = STOP_GROW;
        bs->dense_start = 1;
        bs->op = op_start;
        bs->rows = N;
      }
      return;
    }
  }

  Layout prev{0, 0, 0};  // of the counters to clear
  // Where a launch ends before the last window, for the host to go on from.
  auto stop = [&](u32 why, bool dense_end, float grow) {
    if (grp.bid != 0 || tid != 0) return;
    bs->stopped = why;
    bs->dense_start = 0;
    bs->dense_end = dense_end;
    bs->op = a.windows[win].op + first;
    bs->rows = N;
    bs->phase = ph;
    bs->bins = lay.bins;
    bs->stride = lay.stride;
    bs->cap = lay.cap;
    bs->rho = rho;
    bs->grow = grow;
  };
  for (;;) {
    const float grow = next_grow;
    const bool last = win + 1 >= a.n_windows;
    if ((float)N > REDEAL * (float)SB::R * (float)lay.bins && first < a.windows[win].n_gates &&
        a.windows[win].op + first != a.dealt_op) {
      stop(STOP_DEAL, false, grow);
      return;
    }
    if (2 * N > a.max_rows && first < a.windows[win].n_gates && a.windows[win].n_basis) {
      // the first rotation that branches could pass the row ceiling (every block sees the same)
      if (grp.bid == 0 && tid == 0) {
        bs->rows = N;
        atomicOr(&st->error, ERR_CEILING);
      }
      return;
    }
    const u32 set = ph % 3, nset = (ph + 1) % 3;
    // The rows that will leave this window: as many more or fewer as left the
    // earlier one like it; without one, a reclaim mostly undoes the growth.
    const float* h = alike((float)N, win);
    const float ratio = h ? __ldcg(h + 1) : (a.windows[win].noise == 2 ? 1.0f : 1.5f);
    const Layout nlay = last ? lay : layout_for((float)N * ratio, win + 1, a.room[(ph + 1) & 1]);
    if (tid == 0) {
      v.w = a.windows[win];
      v.wn = last ? WinDesc{} : a.windows[win + 1];
      if (last) {
        Dest d{};
        d.dense = 1;
        d.keys = a.keys;
        d.coeffs = a.coeffs;
        d.room = a.dense_room;
        d.n_dense = &bs->n_dense;
        d.fail = &bs->fail[nset];
        v.d = d;
      } else {
        v.d = dest_bins(a, ph + 1, nlay);
      }
      v.bk = a.bin_keys[ph & 1];
      v.bc = a.bin_coeffs[ph & 1];
      v.bh = a.bin_hash[ph & 1];
      v.bsp = a.spill_bin[ph & 1];
      v.cnt = a.counts + (u64)set * a.count_words;
      v.lay = lay;
      v.first = first;
      v.grow = grow;
      v.spilled = *(volatile u32*)&bs->n_spill[set];
      v.kept = v.n_defer = 0;
    }
    for (u32 i = tid; i < WIN_MAX; i += T) v.born_all[i] = v.anti_all[i] = 0;
    __syncthreads();
    load_grouping<W>(v, a);

    u32 kept = 0, depth0 = 0;
    if (lay.bins == grp.nblk * WARPS) {  // a bin a warp
      const u32 bin = grp.bid * WARPS + (tid >> 5);
      u32 unused = 0;
      if (!run_bin<W, ALG>(a, v, sw[tid >> 5], bin, unused, kept) && lane == 0) v.defer[atomicAdd(&v.n_defer, 1u)] = bin;
      __syncthreads();
      const u32 nd = v.n_defer;
      for (u32 i = 0; i < nd; ++i) {
        run_bin<W, ALG>(a, v, sb, v.defer[i], depth0, kept);
        __syncthreads();
      }
    } else {
      const bool dynamic = lay.bins > grp.nblk;
      u32 bin = grp.bid;
      for (;;) {
        if (dynamic) {
          if (tid == 0) v.tick = atomicAdd(&bs->ticket[set], 1u);
          __syncthreads();
          bin = v.tick;
          __syncthreads();
        }
        if (bin >= lay.bins) break;
        run_bin<W, ALG>(a, v, sb, bin, depth0, kept);
        __syncthreads();
        if (!dynamic) break;
      }
    }
    // Block totals: rows kept, rows created and rows branching per rotation.
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) kept += __shfl_xor_sync(FULL, kept, o);
    if (lane == 0 && kept) atomicAdd(&v.kept, kept);
    __syncthreads();
    if (tid == 0 && v.kept) atomicAdd(&bs->n[nset], (u64)v.kept);
    for (u32 i = tid; i < v.w.n_gates; i += T) {
      if (v.born_all[i]) {
        atomicAdd(a.born + v.w.op + i, v.born_all[i]);
        atomicAdd(&bs->grown[nset], (u64)v.born_all[i]);
      }
      if (v.anti_all[i]) atomicAdd(a.anti + v.w.op + i, (u64)v.anti_all[i]);
    }
    // The counter set after next: its last readers ran the window before this one.
    if (ph > a.phase0) {
      const u32 z = (ph + 2) % 3;
      u32* zc = a.counts + (u64)z * a.count_words;
      for (u32 b = grp.bid * T + tid; b < prev.bins; b += grp.nblk * T) zc[(u64)b * prev.stride] = 0;
      if (grp.bid == 0 && tid == 0) {
        bs->n[z] = bs->grown[z] = 0;
        bs->n_spill[z] = bs->ticket[z] = 0;
      }
    }
    __syncthreads();
    if (tid == 0) {
      if (barrier_arrive(st, grp)) barrier_release(st, gen);
      else barrier_wait(st, gen);
      ++gen;
      const u64 nn = ld_volatile(&bs->n[nset]), gr = ld_volatile(&bs->grown[nset]);
      const u32 e = *(volatile u32*)&st->error, f = *(volatile u32*)&bs->fail[nset];
      v.y[0] = nn;
      v.y[1] = gr;
      v.x[0] = e;
      v.x[1] = f;
    }
    __syncthreads();
    if (v.x[0]) return;
    if (v.x[1]) {  // the next buffer was too small: this window is run again after the host has grown it
      stop(STOP_GROW, last, grow);
      return;
    }
    const u64 nn = v.y[0];
    if (grp.bid == 0 && tid == 0) {
      if (v.w.noise) a.hist[v.w.op + v.w.n_gates] = nn;
      stamp_op(a.stamps, v.w.op_end - 1);
      if (N && !first) {  // read by windows at least 3 further on
        a.growth[3 * win] = (float)(N + v.y[1]) / (float)N;
        a.growth[3 * win + 1] = (float)nn / (float)N;
        a.growth[3 * win + 2] = (float)N;
      }
    }
    rho = fmaxf(N ? (float)(N + v.y[1]) / (float)N : 1.0f, 0.85f * rho);
    N = nn;
    prev = lay;
    lay = nlay;
    first = 0;
    ++ph;
    ++win;
    if (win >= a.n_windows) break;
    __syncthreads();  // v is rewritten
  }
  if (grp.bid == 0 && tid == 0) {
    st->n[0] = N;
    st->end_op = a.op_end;
  }
}
