// hub_core.cuh -- device code of the hub vertices: their tables live in global
// memory (L2), many CTAs merge the edges, and table slices are evaluated in
// parallel.
#ifndef NIDO_HUB_CORE_CUH_
#define NIDO_HUB_CORE_CUH_
#include "move_core.cuh"

namespace nido {

constexpr int kHubThreads = 256;
constexpr int kHubSlice = 4096;

// A hub's table: FP64 sums in two arrays, or packed 64-bit slots (id, int32
// sum) in integer phases.  Read and written past L1 (other CTAs' atomics).
template <bool kInts>
struct HubTable;
template <>
struct HubTable<false> {
  int* keys;
  double* vals;
  __device__ __forceinline__ HubTable at(int64_t o) const { return {keys + o, vals + o}; }
  __device__ __forceinline__ int key(int i) const { return __ldcg(keys + i); }
  __device__ __forceinline__ void get(int i, int& k, double& v) const { k = __ldcg(keys + i); v = __ldcg(vals + i); }
  __device__ __forceinline__ void clear(int i) const { keys[i] = -1; vals[i] = 0.; }
};
template <>
struct HubTable<true> {
  unsigned long long* slots;
  __device__ __forceinline__ HubTable at(int64_t o) const { return {slots + o}; }
  __device__ __forceinline__ int key(int i) const { return slot_key(__ldcg(slots + i)); }
  __device__ __forceinline__ void get(int i, int& k, double& v) const {
    const unsigned long long x = __ldcg(slots + i);
    k = slot_key(x);
    v = (double)slot_sum(x);
  }
  __device__ __forceinline__ void clear(int i) const { slots[i] = kEmptySlot; }
};

// Hub segments: the edges [first, eend) of vertex v in 32-edge chunks into a
// global table; every lane keeps the compare-and-swaps of its kUnroll chunks in
// flight together instead of finishing one chunk's probe before the next.
// Equal communities within a chunk are still folded onto one lane first.
template <int kUnroll>
__device__ __forceinline__ void merge_edges_global(const MoveArgs& p, int v, int64_t first, int64_t eend,
                                                   int64_t stride, int* keys, double* vals, unsigned mask) {
  const int lane = threadIdx.x & 31;
  for (int64_t base = first; base < eend; base += kUnroll * stride) {
    int u[kUnroll], c[kUnroll];
    double wt[kUnroll];
    unsigned h[kUnroll];
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      const int64_t j = base + k * stride + lane;
      u[k] = -1;
      wt[k] = 0.;
      if (j < eend) {
        u[k] = p.adj[j];
        wt[k] = p.w[j];
      }
    }
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      c[k] = u[k] >= 0 ? p.comm[u[k]] : -1;
      if (u[k] == v) wt[k] = 0.;
    }
    unsigned pending = 0u;
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      const bool ok = u[k] >= 0;
      const unsigned peers = __match_any_sync(NIDO_FULL_MASK, c[k]);
      wt[k] = fold_peers(peers, ok, wt[k]);
      if (ok && lane == __ffs(peers) - 1) pending |= 1u << k;
      h[k] = ok ? hash_slot(c[k], mask) : 0u;
    }
    for (unsigned probe = 0; pending != 0u && probe <= mask; ++probe) {
      int old[kUnroll];
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) old[k] = (pending >> k & 1u) ? atomicCAS(&keys[h[k]], -1, c[k]) : 0;
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        if (!(pending >> k & 1u)) continue;
        if (old[k] == -1 || old[k] == c[k]) {
          atomicAdd(&vals[h[k]], wt[k]);
          pending &= ~(1u << k);
        } else {
          h[k] = (h[k] + 1) & mask;
        }
      }
    }
    if (pending != 0u) atomicAdd(p.err, 1ull);
  }
}

// merge_edges_global for packed integer tables (integer-weight phases): one
// 64-bit slot per community (id, int32 sum), so a new community is one
// compare-and-swap that also carries its first sum, an existing one one
// 32-bit add.  Equal communities within a chunk are still folded onto one
// lane first (fewer L2 atomics).
template <int kUnroll>
__device__ __forceinline__ void merge_edges_packed(const MoveArgs& p, int v, int64_t first, int64_t eend,
                                                   int64_t stride, unsigned long long* slots, unsigned mask) {
  const int lane = threadIdx.x & 31;
  for (int64_t base = first; base < eend; base += kUnroll * stride) {
    int u[kUnroll], c[kUnroll], x[kUnroll];
    double wt[kUnroll];
    unsigned h[kUnroll];
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      const int64_t j = base + k * stride + lane;
      u[k] = -1;
      wt[k] = 0.;
      if (j < eend) {
        u[k] = p.adj[j];
        wt[k] = p.w[j];
      }
    }
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      c[k] = u[k] >= 0 ? p.comm[u[k]] : -1;
      if (u[k] == v) wt[k] = 0.;
    }
    unsigned pending = 0u;
#pragma unroll
    for (int k = 0; k < kUnroll; ++k) {
      const bool ok = u[k] >= 0;
      const unsigned peers = __match_any_sync(NIDO_FULL_MASK, c[k]);
      x[k] = __double2int_rn(fold_peers(peers, ok, wt[k]));
      if (ok && lane == __ffs(peers) - 1) pending |= 1u << k;
      h[k] = ok ? hash_slot(c[k], mask) : 0u;
    }
    for (unsigned probe = 0; pending != 0u && probe <= mask; ++probe) {
      unsigned long long old[kUnroll];
#pragma unroll
      for (int k = 0; k < kUnroll; ++k)
        old[k] = (pending >> k & 1u)
                     ? atomicCAS(&slots[h[k]], kEmptySlot, ((unsigned long long)(unsigned)c[k] << 32) | (unsigned)x[k])
                     : 0ull;
#pragma unroll
      for (int k = 0; k < kUnroll; ++k) {
        if (!(pending >> k & 1u)) continue;
        if (old[k] == kEmptySlot) {
          pending &= ~(1u << k);
        } else if (slot_key(old[k]) == c[k]) {
          atomicAdd(reinterpret_cast<int*>(&slots[h[k]]), x[k]);
          pending &= ~(1u << k);
        } else {
          h[k] = (h[k] + 1) & mask;
        }
      }
    }
    if (pending != 0u) atomicAdd(p.err, 1ull);
  }
}

template <int kUnroll>
__device__ __forceinline__ void merge_edges(const MoveArgs& p, int v, int64_t first, int64_t eend, int64_t stride,
                                            const HubTable<false>& t, unsigned mask) {
  merge_edges_global<kUnroll>(p, v, first, eend, stride, t.keys, t.vals, mask);
}
template <int kUnroll>
__device__ __forceinline__ void merge_edges(const MoveArgs& p, int v, int64_t first, int64_t eend, int64_t stride,
                                            const HubTable<true>& t, unsigned mask) {
  merge_edges_packed<kUnroll>(p, v, first, eend, stride, t.slots, mask);
}

// Segment `seg` of hub v's edges into its table, by a CTA of kHubThreads.
template <bool kInts>
__device__ __forceinline__ void hub_segment(const MoveArgs& p, int v, int seg, const HubTable<kInts>& t, int cap) {
  const int64_t s0 = p.off[v] + (int64_t)seg * kHubSeg;
  merge_edges<4>(p, v, s0 + (threadIdx.x & ~31), min(p.off[v + 1], s0 + kHubSeg), kHubThreads, t, (unsigned)cap - 1);
}

// shared memory of the hubs' block-wide reductions
struct HubShared {
  double g[32];
  double e[32];
  unsigned id[32];
};

// Block-wide best (larger gain, then smaller id) and sum of e_own (nonzero in
// one thread at most, so exact in any order): the result in warp 0's lanes.
__device__ __forceinline__ void hub_reduce(double& g, unsigned& id, double& eown, HubShared& sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  eown = group_sum<32>(eown);
  warp_best_id(g, id);
  if (lane == 0) { sh.g[wid] = g; sh.id[wid] = id; sh.e[wid] = eown; }
  __syncthreads();
  if (wid == 0) {
    const bool in = lane < kHubThreads / 32;
    g = in ? sh.g[lane] : -NIDO_MAX_FLOAT;
    id = in ? sh.id[lane] : kNoId;
    eown = in ? sh.e[lane] : 0.;
    eown = group_sum<32>(eown);
    warp_best_id(g, id);
  }
  __syncthreads();
}

// Slots [0, len) of t on the whole CTA: this thread's best community and the
// weight to v's own.  Four slots at a time, so that their a_c gathers are in
// flight together.  kClear: empties the slots on the way.
template <bool kInts, bool kClear>
__device__ __forceinline__ void hub_scan(const MoveArgs& p, const Mass& m, const HubTable<kInts>& t, int len, int own,
                                         double ki, double& g, unsigned& id, double& eown) {
  constexpr int U = 4;
  for (int i0 = threadIdx.x; i0 < len; i0 += U * kHubThreads) {
    int cc[U];
    double val[U], ac[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int i = i0 + k * kHubThreads;
      cc[k] = -1;
      val[k] = 0.;
      if (i < len) t.get(i, cc[k], val[k]);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) ac[k] = (cc[k] >= 0 && cc[k] != own) ? p.a[cc[k]] : 0.;
#pragma unroll
    for (int k = 0; k < U; ++k) {
      if (cc[k] < 0) continue;
      if constexpr (kClear) t.clear(i0 + k * kHubThreads);
      if (cc[k] == own) {
        eown = val[k];
      } else {
        const double gg = gain_of(val[k], ki, ac[k], m);
        if (gg > g || (gg == g && (unsigned)cc[k] < id)) { g = gg; id = (unsigned)cc[k]; }
      }
    }
  }
}

struct SliceResult {
  double g;
  double eown;
  unsigned id;
  int pad;
};

// Slots of one slice of hub v's table, read and cleared in order: the slice's
// result in thread 0.  (A per-hub list of occupied slots, appended during the
// merge, measured twice as slow on R-MAT scale 22: the hub tables are mostly
// full and the list's counter is one contended address per hub.)
template <bool kMulti, bool kInts>
__device__ __forceinline__ SliceResult hub_slice(const MoveArgs& p, int v, const HubTable<kInts>& t, int len,
                                                 HubShared& sh) {
  SliceResult r{-NIDO_MAX_FLOAT, 0., kNoId, 0};
  hub_scan<kInts, true>(p, vertex_mass<kMulti>(p, v), t, len, p.comm[v], p.k[v], r.g, r.id, r.eown);
  hub_reduce(r.g, r.id, r.eown, sh);
  return r;
}

// One warp combines the slices of hub v and decides.
template <bool kMulti>
__device__ __forceinline__ void hub_combine(const MoveArgs& p, int v, const SliceResult* res, int64_t n) {
  const int lane = threadIdx.x & 31;
  double g = -NIDO_MAX_FLOAT, eown = 0.;
  unsigned id = kNoId;
  for (int64_t r = lane; r < n; r += 32) {
    const double xg = __ldcg(&res[r].g);
    const unsigned xi = __ldcg(&res[r].id);
    eown += __ldcg(&res[r].eown);
    if (xg > g || (xg == g && xi < id)) { g = xg; id = xi; }
  }
  eown = group_sum<32>(eown);
  warp_best_id(g, id);
  if (lane == 0) {
    const int own = p.comm[v];
    decide(p, vertex_mass<kMulti>(p, v), v, own, p.k[v], p.a[own], eown, g, id);
  }
}

// ---- the reference's tie rule on a hub ----------------------------------------------
constexpr int kTieList = 1024;  // tied ids held at once
constexpr int kTieCand = 64;    // ids ranked by one walk over the table

struct TieShared {
  int list[kTieList];
  int sorted[kTieList];
  unsigned hist[kTieCand + 1];
  int n;
  unsigned best;
};

// The whole CTA evaluates hub v's filled table of cap slots under the
// reference's tie rule, writes newc[v] and empties the table.  Of the
// communities with the largest gain the smallest (bitrev3(rank mod 8), rank)
// wins, where rank counts the neighbour communities with a smaller id.  The
// tied ids are taken in ascending order (a range of ids at a time when there
// are more than kTieList), kTieCand of them ranked by one walk that
// histograms every id among them, until a rank divisible by 8 appears: no
// later id can beat it, and one of eight ids has such a rank.  (Ranking every
// tied id by its own walk over the table: 110 of 122 ms of an R-MAT scale 18
// run with unit weights, where most neighbours of a hub tie at first.)
template <bool kMulti, bool kInts>
__device__ __forceinline__ void hub_tie(const MoveArgs& p, int v, const HubTable<kInts>& t, int cap, HubShared& sh,
                                        TieShared& ts) {
  const int own = p.comm[v];
  const double ki = p.k[v];
  const Mass m = vertex_mass<kMulti>(p, v);
  double g = -NIDO_MAX_FLOAT, eown = 0.;
  unsigned id = kNoId;
  hub_scan<kInts, false>(p, m, t, cap, own, ki, g, id, eown);
  hub_reduce(g, id, eown, sh);
  if (threadIdx.x == 0) { sh.g[0] = g; sh.id[0] = id; sh.e[0] = eown; }
  __syncthreads();
  const double gm = sh.g[0];
  unsigned win = sh.id[0];
  const double e = sh.e[0];
  __syncthreads();
  if (win != kNoId) {
    unsigned long long best = kNoKey;
    const long long kEnd = 1ll << 31;
    long long lo = win;  // the smallest tied id
    long long hi = kEnd;
    bool done = false;
    while (!done && lo < kEnd) {
      // the tied ids in [lo, hi)
      if (threadIdx.x == 0) ts.n = 0;
      __syncthreads();
      for (int i0 = threadIdx.x; i0 < cap; i0 += 4 * kHubThreads) {
        int cc[4];
        double val[4], ac[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int i = i0 + k * kHubThreads;
          cc[k] = -1;
          val[k] = 0.;
          if (i < cap) t.get(i, cc[k], val[k]);
          if (cc[k] == own || cc[k] < lo || cc[k] >= hi) cc[k] = -1;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) ac[k] = cc[k] >= 0 ? p.a[cc[k]] : 0.;
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (cc[k] >= 0 && gain_of(val[k], ki, ac[k], m) == gm) {
            const int at = atomicAdd(&ts.n, 1);
            if (at < kTieList) ts.list[at] = cc[k];
          }
      }
      __syncthreads();
      const int n = ts.n;
      __syncthreads();
      if (n > kTieList) {  // too many for the list: half the range
        hi = lo + (hi - lo) / 2;
        continue;
      }
      if (n == 1 && hi == kEnd && best == kNoKey) break;  // the only tied id: win
      for (int i = threadIdx.x; i < n; i += kHubThreads) {
        const int x = ts.list[i];
        int r = 0;
        for (int q = 0; q < n; ++q) r += ts.list[q] < x ? 1 : 0;
        ts.sorted[r] = x;
      }
      __syncthreads();
      for (int b = 0; b < n && !done; b += kTieCand) {
        const int nc = min(kTieCand, n - b);
        const int* cand = ts.sorted + b;
        for (int i = threadIdx.x; i <= kTieCand; i += kHubThreads) ts.hist[i] = 0u;
        __syncthreads();
        for (int i0 = threadIdx.x; i0 < cap; i0 += 4 * kHubThreads) {
          int x[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) x[k] = i0 + k * kHubThreads < cap ? t.key(i0 + k * kHubThreads) : -1;
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (x[k] < 0 || x[k] >= cand[nc - 1]) continue;
            int l = 0, u = nc - 1;  // first candidate above x
            while (l < u) {
              const int mid = (l + u) >> 1;
              if (cand[mid] > x[k]) u = mid; else l = mid + 1;
            }
            atomicAdd(&ts.hist[l], 1u);
          }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
          unsigned rank = 0u;
          unsigned long long bk = best;
          unsigned bw = win;
          for (int i = 0; i < nc; ++i) {
            rank += ts.hist[i];
            const unsigned long long key = nido_key(rank);
            if (key < bk) { bk = key; bw = (unsigned)cand[i]; }
            if ((rank & 7u) == 0u) break;
          }
          sh.g[0] = __longlong_as_double((long long)bk);
          ts.best = bw;
        }
        __syncthreads();
        best = (unsigned long long)__double_as_longlong(sh.g[0]);
        win = ts.best;
        done = (best >> 32) == 0ull;
        __syncthreads();
      }
      lo = hi;
      hi = kEnd;
    }
  }
  for (int i = threadIdx.x; i < cap; i += kHubThreads) t.clear(i);
  if (threadIdx.x == 0) decide(p, m, v, own, ki, p.a[own], e, gm, win);
  __syncthreads();
}

}  // namespace nido
#endif
