// move_core.cuh -- device code of the move phase shared by its kernels: the
// arguments, gains, reductions, and the evaluation of vertices by lane groups
// (degree <= 32), warps and CTAs with shared-memory tables.
#ifndef NIDO_MOVE_CORE_CUH_
#define NIDO_MOVE_CORE_CUH_
#include "common.cuh"
#include "engine.cuh"

namespace nido {

constexpr unsigned long long kNoKey = ~0ull;
constexpr unsigned kNoId = 0xFFFFFFFFu;

struct MoveArgs {
  const int64_t* __restrict__ off;
  const int32_t* __restrict__ adj;
  const double* __restrict__ w;
  const double* __restrict__ k;
  // not __restrict__: the persistent phase loop writes them between sweeps
  const int32_t* comm;
  const double* a;
  int32_t* newc;
  double m;
  unsigned long long* err;  // probe-limit failures (never expected)
  // many-graph mode: graph of every vertex and mass of every graph (null for
  // one graph, whose mass is m)
  const int32_t* __restrict__ gid;
  const double* __restrict__ mg;
  // integer phases: reciprocals of the mass (one graph) or of every graph's
  // mass, RN(1/m) and its error term; {0, 0} where quotients by m need the divide
  double zh, zl;
  const double2* __restrict__ zg;
  // every weight integral and every vertex's sum of |w| below 2^31: the
  // shared-memory tables then add int32 (a native shared-memory atomic; the
  // FP64 one is several times slower) and every partial sum is exact, so
  // the e_vc read back are the FP64 sums bit for bit
  int ints;
  int64_t nv;  // vertices of the current graph (all graphs in many-graph mode)
};

MoveArgs move_args(nido_graph_s* g);  // of the current phase (move.cu)

// The mass a vertex's gains are divided by, with its reciprocal zh = RN(1/m)
// and zl = (1 - m zh) zh (zh = 0: use the divide).
struct Mass {
  double m, zh, zl;
};

// The mass of v's graph (kernels are instantiated per mode, so the
// one-graph kernels carry no graph-id lookup).
template <bool kMulti>
__device__ __forceinline__ Mass vertex_mass(const MoveArgs& p, int v) {
  if constexpr (kMulti) {
    const int g = p.gid[v];
    const double2 z = p.zg ? p.zg[g] : make_double2(0., 0.);
    return Mass{p.mg[g], z.x, z.y};
  } else {
    return Mass{p.m, p.zh, p.zl};
  }
}

// RN(a / m) from the reciprocal: q0 = RN(a zh + RN(a zl)) is within one ulp
// of the quotient, its remainder a - m q0 is exact in one fused
// multiply-add, and RN(q0 + remainder * zh) is the correctly rounded quotient
// (P. W. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990, theorem 8.5).  Four multiply-adds instead of
// a divide; every entry of every vertex needs two.  Only in integer phases:
// their operands are 0 or between 2^-120 and 2^100, so nothing under- or
// overflows; in FP64 phases the range checks cost what the divides do (sweeps
// of a 250,007-vertex lognormal SBM: 1.634 ms with divides, 1.655 ms).
__device__ __forceinline__ double div_mass(double a, const Mass& M) {
  const double q0 = __fma_rn(a, M.zh, __dmul_rn(a, M.zl));
  return __fma_rn(__fma_rn(-M.m, q0, a), M.zh, q0);
}

// (e - ki*ac/(2m)) / m in the reference's operation order; RN(y/(2m)) is
// RN(y/m)/2 (a power of two).
__device__ __forceinline__ double gain_of(double e, double ki, double ac, const Mass& M) {
  const double y = __dmul_rn(ki, ac);
  if (M.zh != 0.) return div_mass(__dsub_rn(e, __dmul_rn(0.5, div_mass(y, M))), M);
  const double t = __ddiv_rn(y, __dmul_rn(2.0, M.m));
  return __ddiv_rn(__dsub_rn(e, t), M.m);
}

__device__ __forceinline__ double self_of(double eown, double ki, double aown, const Mass& M) {
  return gain_of(eown, ki, __dsub_rn(aown, ki), M);
}

__device__ __forceinline__ unsigned long long nido_key(unsigned rank) {
  return ((unsigned long long)bitrev3(rank & 7u) << 32) | rank;
}

// Sum of `wt` over the lanes in `peers`, for every lane that is ok.  Every lane of
// the warp must call it; the order is fixed by the peers alone.  Groups of more
// than four lanes are summed one after the other by a butterfly of the whole
// warp (about twenty instructions a group), the rest by a loop over their
// lanes in ascending order (eleven an iteration): once communities have formed, most
// of a chunk's edges end in one, and the loop alone ran once for each of them
// (planted 65,536 vertices 1.83 -> 1.68 ms a run, SBM 2^21 -b 32 96.0 -> 91.9 ms).
constexpr int kFoldLoop = 4;
__device__ __forceinline__ double fold_peers(unsigned peers, bool ok, double wt) {
  const int lane = threadIdx.x & 31;
  const int cnt = ok ? __popc(peers) : 0;
  double e = 0.;
  for (unsigned big = __ballot_sync(NIDO_FULL_MASK, cnt > kFoldLoop); big != 0u;) {
    const unsigned mask = __shfl_sync(NIDO_FULL_MASK, peers, __ffs(big) - 1);
    const bool in = mask >> lane & 1u;
    double x = in ? wt : 0.;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(NIDO_FULL_MASK, x, o);
    if (in) e = x;
    big &= ~mask;
  }
  unsigned rem = cnt <= kFoldLoop && ok ? peers : 0u;
  const int maxcnt = __reduce_max_sync(NIDO_FULL_MASK, (unsigned)__popc(rem));
  for (int i = 0; i < maxcnt; ++i) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    const double x = __shfl_sync(NIDO_FULL_MASK, wt, src);
    if (rem) {
      e += x;
      rem &= rem - 1;
    }
  }
  return e;
}

// Butterfly argmax over groups of G lanes (every lane ends with the result).
template <int G>
__device__ __forceinline__ void group_best(double& g, unsigned long long& tk, int& cand) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const double g2 = __shfl_xor_sync(NIDO_FULL_MASK, g, o, G);
    const unsigned long long t2 = __shfl_xor_sync(NIDO_FULL_MASK, tk, o, G);
    const int c2 = __shfl_xor_sync(NIDO_FULL_MASK, cand, o, G);
    if (better(g2, t2, g, tk)) { g = g2; tk = t2; cand = c2; }
  }
}

// The same under the smallest-id rule: larger gain, then smaller id.
template <int G>
__device__ __forceinline__ void group_best_id(double& g, unsigned& id) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const double g2 = __shfl_xor_sync(NIDO_FULL_MASK, g, o, G);
    const unsigned i2 = __shfl_xor_sync(NIDO_FULL_MASK, id, o, G);
    if (g2 > g || (g2 == g && i2 < id)) { g = g2; id = i2; }
  }
}

template <int G>
__device__ __forceinline__ double group_max(double g) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) g = fmax(g, __shfl_xor_sync(NIDO_FULL_MASK, g, o, G));
  return g;
}

template <int G>
__device__ __forceinline__ double group_sum(double x) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) x += __shfl_xor_sync(NIDO_FULL_MASK, x, o, G);
  return x;
}

// Warp argmax of (gain, smallest id) under the smallest-id rule (id kNoId
// without a candidate) with three 32-bit warp reductions instead of a shuffle
// tree: the gain as an order-preserving 64-bit key (+0 for -0, which compares
// equal to it), then the smallest id among the lanes holding the largest gain.
// Every lane of the warp must call it; all end with the result.
__device__ __forceinline__ void warp_best_id(double& g, unsigned& id) {
  const long long b = __double_as_longlong(g + 0.0);
  const unsigned long long key = b < 0 ? ~(unsigned long long)b : ((unsigned long long)b | 0x8000000000000000ull);
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(NIDO_FULL_MASK, hi);
  const unsigned ml = __reduce_max_sync(NIDO_FULL_MASK, hi == mh ? lo : 0u);
  id = __reduce_min_sync(NIDO_FULL_MASK, hi == mh && lo == ml ? id : kNoId);
  const unsigned long long top = ((unsigned long long)mh << 32) | ml;
  g = __longlong_as_double((long long)(top >> 63 ? top & 0x7fffffffffffffffull : ~top));
}

__device__ __forceinline__ void decide(const MoveArgs& p, const Mass& m, int v, int own, double ki, double aown,
                                       double eown, double g, unsigned id) {
  const double self = self_of(eown, ki, aown, m);
  const double tot = __dsub_rn(g, self);
  p.newc[v] = (id != kNoId && tot > 0.) ? (int)id : own;
}

// ---- degree <= 32: registers ---------------------------------------------------
// The vertices of list[0, n) by lane groups of G: this warp takes the sets
// of 32/G vertices warp, warp + nw, ...; fold: 32 ints of shared memory per warp
// (integer phases: per-lane group sums).
template <int G, bool kMulti, bool kTie>
__device__ __forceinline__ void group_list(const int32_t* __restrict__ list, int64_t n, int64_t warp, int64_t nw,
                                           const MoveArgs& p, int* fold) {
  constexpr int VPW = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gid = lane / G;
  for (int64_t b = warp * VPW; b < n; b += nw * VPW) {
    const int64_t idx = b + gid;
    const bool vok = idx < n;
    int v = 0, own = -1;
    int64_t s = 0, d = 0;
    double ki = 0., aown = 0.;
    Mass m{p.m, p.zh, p.zl};
    if (vok) {
      v = list[idx];
      s = p.off[v];
      d = p.off[v + 1] - s;
      own = p.comm[v];
      ki = p.k[v];
      aown = p.a[own];
      m = vertex_mass<kMulti>(p, v);
    }
    const bool ok = gl < d;
    int c = -1;
    double wt = 0.;
    if (ok) {
      const int u = p.adj[s + gl];
      c = p.comm[u];
      wt = (u == v) ? 0. : p.w[s + gl];
    }
    // lanes of one vertex with equal communities: a 32-bit match where the
    // group index fits above the ids (invalid lanes, c = -1, may match across
    // groups; they add nothing), else a 64-bit one
    unsigned peers;
    if constexpr (G == 32) {
      peers = __match_any_sync(NIDO_FULL_MASK, (unsigned)c);
    } else if (p.nv <= (int64_t)1 << 29) {
      peers = __match_any_sync(NIDO_FULL_MASK, (unsigned)c | ((unsigned)gid << 29));
    } else {
      peers = __match_any_sync(NIDO_FULL_MASK, ((unsigned long long)(unsigned)gid << 32) | (unsigned)c);
    }
    const int leader = __ffs(peers) - 1;
    const bool lead = ok && lane == leader;
    double e;
    if (p.ints) {
      // integer weights: every lane adds its weight into its group leader's
      // shared-memory slot (int32 adds, exact in any order; equal addresses
      // are serialised by the atomic unit, not by instructions)
      fold[lane] = 0;
      __syncwarp();
      if (ok) atomicAdd(&fold[leader], __double2int_rn(wt));
      __syncwarp();
      e = (double)fold[lane];
    } else {
      e = fold_peers(peers, ok, wt);
    }
    double g = -NIDO_MAX_FLOAT, eown = 0.;
    unsigned id = kNoId;
    if (lead) {
      if (c == own) {
        eown = e;
      } else {
        g = gain_of(e, ki, p.a[c], m);
        id = (unsigned)c;
      }
    }
    eown = group_sum<G>(eown);
    if constexpr (kTie) {
      const double gm = group_max<G>(g);
      unsigned rank = 0;
      const int gbase = gid * G;
      for (int j = 0; j < G; ++j) {
        const int cj = __shfl_sync(NIDO_FULL_MASK, c, gbase + j);
        const int lj = __shfl_sync(NIDO_FULL_MASK, (int)lead, gbase + j);
        rank += (lj && cj < c) ? 1u : 0u;
      }
      unsigned long long tk = (id != kNoId && g == gm) ? nido_key(rank) : kNoKey;
      int cand = (int)id;
      if (tk == kNoKey) { g = -NIDO_MAX_FLOAT; cand = -1; }
      group_best<G>(g, tk, cand);
      id = (unsigned)cand;
    } else if constexpr (G == 32) {
      warp_best_id(g, id);
    } else {
      group_best_id<G>(g, id);
    }
    if (gl == 0 && vok) decide(p, m, v, own, ki, aown, eown, g, id);
  }
}

// ---- shared-memory tables -------------------------------------------------------
// Open addressing over a power-of-two slot array.  Integer phases: one 64-bit
// word a slot, the community id in the high half (-1: empty) and the int32 sum
// in the low half; FP64 phases: ids and FP64 sums in two arrays.  The lane that
// inserts a community owns its slot: it evaluates it, clears it, and keeps the
// slot's number in a register, so there is no list of occupied slots.  A table has
// at least 4/3 as many slots as the vertex has edges, so a free slot always
// exists; probing is still bounded by the table size, and a full table is
// reported through *err.
constexpr unsigned long long kEmptySlot = 0xFFFFFFFF00000000ull;
__device__ __forceinline__ int slot_key(unsigned long long x) { return (int)(x >> 32); }
__device__ __forceinline__ int slot_sum(unsigned long long x) { return (int)(unsigned)x; }

template <bool kInts>
struct SharedTable;

template <>
struct SharedTable<true> {
  unsigned long long* slots;
  __device__ __forceinline__ void place(void* mem, int) { slots = static_cast<unsigned long long*>(mem); }
  __device__ __forceinline__ void clear(int h) const { slots[h] = kEmptySlot; }
  __device__ __forceinline__ int* sum(int h) const { return reinterpret_cast<int*>(slots + h); }
  __device__ __forceinline__ int* key(int h) const { return reinterpret_cast<int*>(slots + h) + 1; }
  __device__ __forceinline__ void get(int h, int& key, double& val) const {
    const unsigned long long x = slots[h];
    key = slot_key(x);
    val = (double)slot_sum(x);
  }
};

template <>
struct SharedTable<false> {
  double* vals;
  int* keys;
  __device__ __forceinline__ void place(void* mem, int cap) {
    vals = static_cast<double*>(mem);
    keys = reinterpret_cast<int*>(vals + cap);
  }
  __device__ __forceinline__ void clear(int h) const { keys[h] = -1; vals[h] = 0.; }
  __device__ __forceinline__ int* key(int h) const { return keys + h; }
  __device__ __forceinline__ void get(int h, int& k, double& val) const {
    k = keys[h];
    val = vals[h];
  }
};

// Slots of up to kChunks communities, two 16-bit numbers a register
// (kNoSlot: none): the largest table has 16,384 slots.
constexpr unsigned kNoSlot = 0xFFFFu;
template <int kChunks>
struct OwnSlots {
  static_assert(kChunks % 2 == 0, "whole registers");
  unsigned r[kChunks / 2];
  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int i = 0; i < kChunks / 2; ++i) r[i] = 0xFFFFFFFFu;
  }
  // constant k: a byte permute
  __device__ __forceinline__ void set(int k, int s) {
    r[k / 2] = k & 1 ? __byte_perm(r[k / 2], (unsigned)s, 0x5410) : __byte_perm(r[k / 2], (unsigned)s, 0x3254);
  }
  __device__ __forceinline__ unsigned get(int k) const { return k & 1 ? r[k / 2] >> 16 : r[k / 2] & 0xFFFFu; }
};

constexpr size_t table_bytes(int slots, bool ints) { return (size_t)slots * (ints ? 8 : 12); }

// Slot of community c, inserted when absent (*isnew: by this lane); -1 when
// the table is full.
template <bool kInts>
__device__ __forceinline__ int table_slot(const SharedTable<kInts>& t, unsigned mask, int c, bool* isnew,
                                          unsigned long long* err) {
  unsigned h = hash_slot(c, mask);
  *isnew = false;
  for (unsigned probe = 0; probe <= mask; ++probe) {
    int k = *static_cast<volatile int*>(t.key((int)h));
    if (k == -1) {
      k = atomicCAS(t.key((int)h), -1, c);
      if (k == -1) {
        *isnew = true;
        return (int)h;
      }
    }
    if (k == c) return (int)h;
    h = (h + probe + 1) & mask;  // triangular steps: every slot once
  }
  atomicAdd(err, 1ull);
  return -1;
}

// Edge ids and weights are read once per sweep: loaded without allocating in
// L1, which keeps L1 for the comm[u] and a[c] gathers (-2% on the move phase).
__device__ __forceinline__ int ld_stream(const int* q) {
  int v;
  asm("ld.global.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(q));
  return v;
}
__device__ __forceinline__ double ld_stream(const double* q) {
  double v;
  asm("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(q));
  return v;
}

// smallest power of two >= max(64, 2d) (shared-memory tiers: d <= 2^30)
__device__ __forceinline__ unsigned next_pow2_cap(int d) {
  const unsigned x = (unsigned)max(64, 2 * min(d, 1 << 30));
  return 1u << (32 - __clz(x - 1));
}

// Adds the d edges of vertex v (ids at ap, weights at wp) to the table with a
// team of kTeam threads (a warp or a CTA): thread t takes the edges t, t +
// kTeam, ...  On return h holds the slots of the communities this thread
// inserted.  The loads of up to four edges a thread are in flight before the
// first is added.
// Integer phases: every lane adds its own edge (int32 atomics, exact in any
// order).  FP64 phases: equal communities of a 32-edge chunk are folded onto the
// first lane, which adds them (a warp adds its chunks in
// order; the warps of a CTA add atomically).
template <int kTeam, int kChunks, bool kInts, bool kStaged>
__device__ __forceinline__ void team_accumulate(const MoveArgs& p, int v, const int32_t* ap, const double* wp, int d,
                                                const SharedTable<kInts>& t, unsigned mask, OwnSlots<kChunks>& h) {
  constexpr int kU = kChunks % 4 == 0 ? 4 : 3;
  static_assert(kChunks % kU == 0, "whole groups of chunks");
  const int lane = threadIdx.x & 31;
  const int tid = kTeam == 32 ? lane : (int)threadIdx.x;
  h.reset();
#pragma unroll
  for (int b = 0; b < kChunks; b += kU) {
    if (b * kTeam + (tid - lane) >= d) break;  // warp-uniform
    int c[kU];
    double wt[kU];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      const int j = (b + k) * kTeam + tid;
      c[k] = -1;
      wt[k] = 0.;
      if (j < d) {
        c[k] = kStaged ? ap[j] : ld_stream(ap + j);
        wt[k] = kStaged ? wp[j] : ld_stream(wp + j);
        if (c[k] == v) wt[k] = 0.;
      }
    }
#pragma unroll
    for (int k = 0; k < kU; ++k)
      if (c[k] >= 0) c[k] = p.comm[c[k]];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      if ((b + k) * kTeam + (tid - lane) >= d) break;  // warp-uniform
      bool isnew = false;
      if constexpr (kInts) {
        if (c[k] >= 0) {
          const int s = table_slot(t, mask, c[k], &isnew, p.err);
          if (s >= 0) atomicAdd(t.sum(s), __double2int_rn(wt[k]));
          if (isnew) h.set(b + k, s);
        }
      } else {
        const bool ok = c[k] >= 0;
        const unsigned peers = __match_any_sync(NIDO_FULL_MASK, c[k]);
        const bool lead = ok && lane == __ffs(peers) - 1;
        const double e = fold_peers(peers, ok, wt[k]);
        if (lead) {
          const int s = table_slot(t, mask, c[k], &isnew, p.err);
          if (s >= 0) {
            if constexpr (kTeam == 32) t.vals[s] += e;
            else atomicAdd(&t.vals[s], e);
          }
          if (isnew) h.set(b + k, s);
        }
        __syncwarp();
      }
    }
  }
}

// Best community of this thread's own slots (larger gain, then smaller id) and
// the weight to the vertex's own community where this thread owns that slot
// (has_own).  kClear: the slots are emptied on the way.  The a_c gathers of up
// to four slots are in flight together.
template <int kChunks, bool kInts, bool kClear>
__device__ __forceinline__ void team_scan(const MoveArgs& p, const Mass& m, const SharedTable<kInts>& t, int own,
                                          double ki, const OwnSlots<kChunks>& h, double& g, unsigned& id,
                                          double& eown, bool& has_own) {
  constexpr int kU = kChunks % 4 == 0 ? 4 : 2;
#pragma unroll
  for (int b = 0; b < kChunks; b += kU) {
    unsigned all = 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < kU / 2; ++k) all &= h.r[b / 2 + k];
    if (!__any_sync(NIDO_FULL_MASK, all != 0xFFFFFFFFu)) continue;
    int c[kU];
    double val[kU], ac[kU];
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      c[k] = -1;
      val[k] = 0.;
      ac[k] = 0.;
      const unsigned s = h.get(b + k);
      if (s != kNoSlot) {
        t.get((int)s, c[k], val[k]);
        if (c[k] != own) ac[k] = p.a[c[k]];
        if constexpr (kClear) t.clear((int)s);
      }
    }
#pragma unroll
    for (int k = 0; k < kU; ++k) {
      if (c[k] < 0) continue;
      if (c[k] == own) {
        eown = val[k];
        has_own = true;
      } else {
        const double gg = gain_of(val[k], ki, ac[k], m);
        const unsigned cc = (unsigned)c[k];
        if (gg > g || (gg == g && cc < id)) { g = gg; id = cc; }
      }
    }
  }
}

// The reference's tie rule over a team's slots, once the largest gain gm is
// known: among the communities whose gain equals gm, the smallest (bitrev3(rank
// mod 8), rank), where rank counts the neighbour communities with a smaller id.
// The tied ids are taken in ascending order, each ranked by one team-wide
// count of the smaller ids, until a rank divisible by 8 appears (no later one
// can win) or none is left.  tmin / tsum: team-wide reductions of an unsigned.
// (Ranking every tied id by a walk over the whole list made a sweep quadratic
// in the ties: R-MAT scale 18, unit weights, run 171 -> 141 ms.)
template <int kChunks, bool kInts, typename Min, typename Sum>
__device__ __forceinline__ unsigned team_nido_tie(const MoveArgs& p, const Mass& m, const SharedTable<kInts>& t,
                                                  int own, double ki, double gm, const OwnSlots<kChunks>& h, Min tmin,
                                                  Sum tsum) {
  unsigned tied = 0u;
  int c[kChunks];
#pragma unroll
  for (int k = 0; k < kChunks; ++k) {
    c[k] = -1;
    const unsigned s = h.get(k);
    if (s != kNoSlot) {
      double val;
      t.get((int)s, c[k], val);
      if (c[k] != own && gain_of(val, ki, p.a[c[k]], m) == gm) tied |= 1u << k;
    }
  }
  unsigned left = tsum((unsigned)__popc(tied));
  unsigned best_id = kNoId;
  unsigned long long best = kNoKey;
  const bool one = left == 1u;
  while (left > 0u) {
    unsigned x = kNoId;
#pragma unroll
    for (int k = 0; k < kChunks; ++k)
      if (tied >> k & 1u) x = min(x, (unsigned)c[k]);
    x = tmin(x);
    if (one) return x;
    unsigned below = 0u;
#pragma unroll
    for (int k = 0; k < kChunks; ++k) {
      below += (c[k] >= 0 && (unsigned)c[k] < x) ? 1u : 0u;
      if ((tied >> k & 1u) && (unsigned)c[k] == x) tied &= ~(1u << k);
    }
    const unsigned rank = tsum(below);
    const unsigned long long key = nido_key(rank);
    if (key < best) { best = key; best_id = x; }
    if ((rank & 7u) == 0u) break;
    --left;
  }
  return best_id;
}

// ---- 32 < degree <= 192: one warp per vertex -------------------------------------
// The vertices warp, warp + nw, ... of list[0, n) on this warp; t: an empty
// table of kCap slots, left empty.
template <int kCap, int kChunks, bool kMulti, bool kInts, bool kTie>
__device__ __forceinline__ void warp_list(const int32_t* __restrict__ list, int64_t n, int64_t warp, int64_t nw,
                                          const MoveArgs& p, const SharedTable<kInts>& t) {
  const int lane = threadIdx.x & 31;
  for (int64_t task = warp; task < n; task += nw) {
    const int v = list[task];
    const int64_t s = p.off[v];
    const int d = (int)(p.off[v + 1] - s);
    const unsigned mask = min((unsigned)kCap, next_pow2_cap(d)) - 1;
    const int own = p.comm[v];
    const double ki = p.k[v], aown = p.a[own];
    OwnSlots<kChunks> h;
    team_accumulate<32, kChunks, kInts, false>(p, v, p.adj + s, p.w + s, d, t, mask, h);
    __syncwarp();
    const Mass m = vertex_mass<kMulti>(p, v);
    double g = -NIDO_MAX_FLOAT, eown = 0.;
    unsigned id = kNoId;
    bool has_own = false;
    team_scan<kChunks, kInts, !kTie>(p, m, t, own, ki, h, g, id, eown, has_own);
    // at most one lane owns the slot of the vertex's own community
    const unsigned ob = __ballot_sync(NIDO_FULL_MASK, has_own);
    if (ob) eown = __shfl_sync(NIDO_FULL_MASK, eown, __ffs(ob) - 1);
    warp_best_id(g, id);
    if constexpr (kTie) {
      if (id != kNoId)
        id = team_nido_tie<kChunks, kInts>(
            p, m, t, own, ki, g, h, [](unsigned x) { return __reduce_min_sync(NIDO_FULL_MASK, x); },
            [](unsigned x) { return __reduce_add_sync(NIDO_FULL_MASK, x); });
      __syncwarp();
#pragma unroll
      for (int k = 0; k < kChunks; ++k)
        if (h.get(k) != kNoSlot) t.clear((int)h.get(k));
    }
    if (lane == 0) decide(p, m, v, own, ki, aown, eown, g, id);
    __syncwarp();
  }
}

// ---- larger degrees: one CTA per vertex ------------------------------------------
// shared memory of the block-wide reductions
struct CtaShared {
  double g[32];
  double eown;
  unsigned id[32];
  unsigned red[32];
};

// Block-wide minimum / sum of an unsigned (every thread gets the result).
template <int kThreads>
__device__ __forceinline__ unsigned cta_min(unsigned x, unsigned* red) {
  x = __reduce_min_sync(NIDO_FULL_MASK, x);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) x = min(x, red[i]);
  __syncthreads();
  return x;
}
template <int kThreads>
__device__ __forceinline__ unsigned cta_sum(unsigned x, unsigned* red) {
  x = __reduce_add_sync(NIDO_FULL_MASK, x);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
  __syncthreads();
  unsigned s = 0u;
#pragma unroll
  for (int i = 0; i < kThreads / 32; ++i) s += red[i];
  __syncthreads();
  return s;
}

// One vertex whose d edges are at ap / wp, on the whole CTA: two block
// barriers, one after the inserts and one before warp 0 combines the warps'
// bests and decides; the other warps go on to the next vertex meanwhile (they
// write the warps' results again only after its first barrier).  between() runs
// after the first barrier (every thread has read its edges).  sh.eown is 0 and
// t is empty on entry and on return.
template <int kThreads, int kCap, int kChunks, bool kInts, bool kTie, bool kStaged, typename Between>
__device__ __forceinline__ void cta_vertex(const MoveArgs& p, const Mass& m, int v, const int32_t* ap,
                                           const double* wp, int d, int own, double ki, double aown,
                                           const SharedTable<kInts>& t, CtaShared& sh, Between between) {
  constexpr int kWarps = kThreads / 32;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const unsigned mask = min((unsigned)kCap, next_pow2_cap(d)) - 1;
  OwnSlots<kChunks> h;
  team_accumulate<kThreads, kChunks, kInts, kStaged>(p, v, ap, wp, d, t, mask, h);
  __syncthreads();
  between();
  double g = -NIDO_MAX_FLOAT, eown = 0.;
  unsigned id = kNoId;
  bool has_own = false;
  team_scan<kChunks, kInts, !kTie>(p, m, t, own, ki, h, g, id, eown, has_own);
  if (has_own) sh.eown = eown;  // at most one thread
  warp_best_id(g, id);
  if (lane == 0) { sh.g[wid] = g; sh.id[wid] = id; }
  __syncthreads();
  if constexpr (kTie) {
    // every thread learns the largest gain, then the tied ids are ranked
    g = lane < kWarps ? sh.g[lane] : -NIDO_MAX_FLOAT;
    id = lane < kWarps ? sh.id[lane] : kNoId;
    warp_best_id(g, id);
    unsigned* red = sh.red;
    if (id != kNoId)
      id = team_nido_tie<kChunks, kInts>(
          p, m, t, own, ki, g, h, [red](unsigned x) { return cta_min<kThreads>(x, red); },
          [red](unsigned x) { return cta_sum<kThreads>(x, red); });
    __syncthreads();  // every thread has read its slots and the warps' results
#pragma unroll
    for (int k = 0; k < kChunks; ++k)
      if (h.get(k) != kNoSlot) t.clear((int)h.get(k));
    if (threadIdx.x == 0) {
      decide(p, m, v, own, ki, aown, sh.eown, g, id);
      sh.eown = 0.;
    }
    __syncthreads();  // the slots are clear
  } else if (wid == 0) {
    g = lane < kWarps ? sh.g[lane] : -NIDO_MAX_FLOAT;
    id = lane < kWarps ? sh.id[lane] : kNoId;
    warp_best_id(g, id);
    if (lane == 0) {
      decide(p, m, v, own, ki, aown, sh.eown, g, id);
      sh.eown = 0.;
    }
  }
}

}  // namespace nido
#endif
