// phase_step.cu -- the coarsening of a small phase and the set-up of the next
// one as a single persistent kernel.
//
// For a small graph the aggregation (graph_gpu.cpp:1382-1545) and the next
// phase's k, m, cuts and tier lists are some forty launches and four readbacks,
// 390 us a phase whatever its size.  Here they are stages of one cooperative
// kernel with grid barriers (phase_loop.cuh) and one readback.
//
// The coarse edges come from one hash table keyed by (coarse vertex, coarse
// neighbour) over all edges at once.  Each entry sums its weights and keeps the
// first list position it occurs at, where the lists are the members' edges in
// ascending member order, one coarse vertex after the other; a bitmap of the
// first positions then ranks every entry by a popcount prefix, which is its
// place in the coarse CSR in the reference's first-occurrence order.  Equal
// neighbours of a 32-edge chunk are folded before they are added; across
// chunks the adds are atomic (exact for integer weights, as in
// the CTA tiers of coarsen.cu).  In FP64 phases the weights of coarse vertices
// of at most 1024 member edges are added in list order instead: every edge notes
// its entry and weight at its list position, and a warp walks the list.  Up to
// 256 each weight is added to its entry, as in the warp tier of coarsen.cu, above
// each 32-edge chunk's sum, as in its CTA tiers (in some order there).
#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

#include "cuts.cuh"
#include "phase_loop.cuh"

namespace nido {
namespace {

constexpr int kStepThreads = 256;
constexpr int kStepKeys = 2048;              // (tier, batch) lists at most
constexpr int64_t kStepMaxEdges = (int64_t)1 << 21;
// members of a coarse vertex above which a block finds their positions in one
// ordered walk over the vertices; below, each member adds up the degrees of the
// smaller members itself
constexpr int kStepBigList = 2048;
constexpr unsigned long long kNoEntry = ~0ull;

struct StepOut {  // read back by the host; cuts and list offsets follow
  long long nvp, nep, done;
  double m;
  unsigned long long maxdeg, flags[2];
};

struct StepArgs {
  const int64_t* __restrict__ off;
  const int32_t* __restrict__ adj;
  const double* __restrict__ w;
  int64_t nv, nv0;
  const int32_t* comm;
  double* k;
  int32_t* clus;
  int32_t* perm;
  const int64_t* tier_off;  // of the finished phase, kNumTiers * nb + 1
  int nb;                   // its batches
  int nbn;                  // batches of the next phase; 0: no cuts and lists (colour classes)
  const int2* items;        // its hub segments
  int64_t nitems;
  const int32_t* hub_v;
  // scratch, one entry a vertex (and one more where scanned)
  int32_t *used, *newid, *cnt, *cursor, *mo, *deg, *p0, *member, *pos;
  int32_t* bsum;            // 2 per block
  double* part;             // 4096 mass partials
  // coarse graph
  int64_t* coff;
  int32_t* cadj;
  double* cw;
  // table, bitmap of first positions and its prefix counts
  unsigned long long* keys;
  double* vals;
  unsigned* first;
  unsigned mask;
  uint32_t* bm;
  int32_t* wpre;
  int64_t nwords;
  // next phase
  int64_t* cuts;            // nb + 1, then parts of nb + 2
  int64_t* parts;
  int32_t* counts;          // kNumTiers * nb + 1 counts, then cursors
  int32_t* ccur;
  int32_t* vkey;
  int64_t* toff;            // list offsets of the next phase
  StepOut* out;
  PhaseCtl* ctl;
  unsigned long long* err;
  // many graphs: each one's first vertex, and its first coarse vertex (written).
  // Vertices with a negative community are dropped; every vertex's edges are
  // walked, as the lists hold only the graphs that still iterate.
  const int64_t* gbase;
  int64_t* gbase2;
  int ng;
  bool coarsen;             // false: only the set-up of the current graph
  bool setup;               // false: only the coarsening
  bool ordered;             // FP64 phase: short lists are summed in list order
  int warp, ctas, ctam, ctal;
};

__device__ __forceinline__ int warp_incl(int x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(NIDO_FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Exclusive block scan of x; *tot: the block's sum.
__device__ __forceinline__ int block_excl(int x, int* tot, int* ws) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int inc = warp_incl(x);
  if (lane == 31) ws[wid] = inc;
  __syncthreads();
  int pre = 0, all = 0;
#pragma unroll
  for (int i = 0; i < kStepThreads / 32; ++i) {
    const int y = ws[i];
    if (i < wid) pre += y;
    all += y;
  }
  __syncthreads();
  *tot = all;
  return pre + inc - x;
}

__device__ __forceinline__ int block_total(int x, int* ws) {
  int tot;
  block_excl(x, &tot, ws);
  return tot;
}

// The elements [lo, hi) this block scans of n.
__device__ __forceinline__ void scan_share(int64_t n, int64_t* lo, int64_t* hi) {
  const int64_t per = ((n + gridDim.x - 1) / gridDim.x + kStepThreads - 1) / kStepThreads * kStepThreads;
  *lo = min(n, per * (int64_t)blockIdx.x);
  *hi = min(n, *lo + per);
}

// First half of a grid-wide exclusive scan: this block's sum of get(i) into
// bsum[blockIdx.x].
template <typename Get>
__device__ __forceinline__ void scan_sums(int64_t n, Get get, int32_t* bsum, int* ws) {
  int64_t lo, hi;
  scan_share(n, &lo, &hi);
  int s = 0;
  for (int64_t i = lo + threadIdx.x; i < hi; i += kStepThreads) s += get(i);
  s = block_total(s, ws);
  if (threadIdx.x == 0) bsum[blockIdx.x] = s;
}

// Second half, after a grid barrier: put(i, prefix) for every element, and
// put(n, total).
template <typename Get, typename Put>
__device__ __forceinline__ void scan_apply(int64_t n, Get get, const int32_t* bsum, Put put, int* ws) {
  int64_t lo, hi;
  scan_share(n, &lo, &hi);
  int b = 0, all = 0;
  for (int i = threadIdx.x; i < (int)gridDim.x; i += kStepThreads) {
    const int y = __ldcg(bsum + i);
    if (i < (int)blockIdx.x) b += y;
    all += y;
  }
  int run = block_total(b, ws);
  all = block_total(all, ws);
  for (int64_t t = lo; t < hi; t += kStepThreads) {
    const int64_t i = t + threadIdx.x;
    const int x = i < hi ? get(i) : 0;
    int tot;
    const int pre = block_excl(x, &tot, ws);
    if (i < hi) put(i, run + pre);
    run += tot;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) put(n, all);
}

// member edges of a list summed in order: a chunk takes a warp about two
// microseconds (planted, 7,900 edges a list: 2.7 ms a run in order, 2.1 without)
constexpr int kStepOrdered = 1024;
constexpr int kStepOneByOne = 256;   // and of one whose weights are added one by one

// Entry of (cu, cv) with `at` among its positions; adds x unless the list is
// summed in order.
__device__ __forceinline__ int table_put(const StepArgs& A, int cu, int cv, bool add, double x, unsigned at) {
  const unsigned long long key = (unsigned long long)(unsigned)cu << 32 | (unsigned)cv;
  unsigned h = (unsigned)((key * 0x9E3779B97F4A7C15ull) >> 32) & A.mask;
  for (unsigned probe = 0; probe <= A.mask; ++probe) {
    unsigned long long o = __ldcg(A.keys + h);
    if (o == kNoEntry) o = atomicCAS(A.keys + h, kNoEntry, key);
    if (o == kNoEntry || o == key) {
      if (add) atomicAdd(A.vals + h, x);
      if (__ldcg(A.first + h) > at) atomicMin(A.first + h, at);
      return (int)h;
    }
    h = (h + probe + 1) & A.mask;
  }
  atomicAdd(A.err, 1ull);
  return 0;
}

// One edge a lane (ok): list position `at`, from coarse vertex cu to cv with
// weight x; peers: the lanes with the same entry.
__device__ __forceinline__ void put_chunk(const StepArgs& A, unsigned peers, bool ok, int cu, int cv, double x,
                                          unsigned at) {
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  const bool in_order = A.ordered && ok && A.deg[cu] <= kStepOrdered;
  const double s = fold_peers(peers, ok, x);
  int h = 0;
  if (ok && lane == leader) h = table_put(A, cu, cv, !in_order, s, at);
  if (A.ordered) {
    h = __shfl_sync(NIDO_FULL_MASK, h, leader);
    if (in_order) {  // the coarse graph's arrays are free until the entries are written
      A.cadj[at] = h;
      A.cw[at] = x;
    }
  }
}

// Edges [j0, j1) of vertex v, 32 at a time every `stride`, by a warp.
__device__ __forceinline__ void put_edges(const StepArgs& A, int v, int64_t e0, int64_t j0, int64_t j1, int64_t stride) {
  const int lane = threadIdx.x & 31;
  const int cu = A.newid[v], at = A.pos[v];
  for (int64_t b = j0; b < j1; b += stride) {
    const int64_t j = b + lane;
    const bool ok = j < j1;
    int cv = -1;
    double x = 0.;
    if (ok) {
      cv = A.newid[A.adj[e0 + j]];
      x = A.w[e0 + j];
    }
    put_chunk(A, __match_any_sync(NIDO_FULL_MASK, cv), ok, cu, cv, x, (unsigned)at + (unsigned)j);
  }
}

// Vertices of list[0, n) with at most G edges, 32/G at a time by a warp.
template <int G>
__device__ __forceinline__ void put_groups(const StepArgs& A, const int32_t* list, int64_t n, int64_t gw, int64_t nw) {
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gid = lane / G;
  for (int64_t b = gw * (32 / G); b < n; b += nw * (32 / G)) {
    const int64_t i = b + gid;
    int cu = 0, cv = -1;
    unsigned at = 0;
    double x = 0.;
    bool ok = false;
    if (i < n) {
      const int v = list[i];
      const int64_t e0 = A.off[v];
      ok = gl < A.off[v + 1] - e0;
      cu = A.newid[v];
      at = (unsigned)A.pos[v] + (unsigned)gl;
      if (ok) {
        cv = A.newid[A.adj[e0 + gl]];
        x = A.w[e0 + gl];
      }
    }
    put_chunk(A, __match_any_sync(NIDO_FULL_MASK, ((unsigned long long)(unsigned)gid << 32) | (unsigned)cv), ok, cu, cv,
              x, at);
  }
}

// The lists summed in order, a warp per coarse vertex: the lanes' weights are
// folded in lane (= list) order.
__device__ __forceinline__ void sum_in_order(const StepArgs& A, int64_t nvp, int64_t gw, int64_t nw) {
  const int lane = threadIdx.x & 31;
  for (int64_t c = gw; c < nvp; c += nw) {
    const int D = A.deg[c], p = A.p0[c];
    if (D > kStepOrdered) continue;
    // the next chunk's entries and weights are loaded ahead
    int hn = lane < D ? A.cadj[p + lane] : -1;
    double xn = lane < D ? A.cw[p + lane] : 0.;
    for (int b = 0; b < D; b += 32) {
      const bool ok = b + lane < D;
      const int h = hn;
      const double x = xn;
      hn = -1;
      if (b + 32 + lane < D) {
        hn = A.cadj[p + b + 32 + lane];
        xn = A.cw[p + b + 32 + lane];
      }
      const unsigned peers = __match_any_sync(NIDO_FULL_MASK, h);
      const bool leads = ok && lane == __ffs(peers) - 1;
      const double old = leads ? A.vals[h] : 0.;
      double acc = D <= kStepOneByOne ? old : 0.;
      unsigned rem = ok ? peers : 0u;
      const int maxcnt = __reduce_max_sync(NIDO_FULL_MASK, (unsigned)__popc(rem));
      for (int i = 0; i < maxcnt; ++i) {
        const int src = rem ? __ffs(rem) - 1 : lane;
        const double y = __shfl_sync(NIDO_FULL_MASK, x, src);
        if (rem) { acc += y; rem &= rem - 1; }
      }
      if (leads) A.vals[h] = D <= kStepOneByOne ? acc : old + acc;
      __syncwarp();
    }
  }
}

__device__ __forceinline__ int step_tier(const StepArgs& A, int64_t d) {
  if (d <= 4) return kTierG4;
  if (d <= 8) return kTierG8;
  if (d <= 16) return kTierG16;
  if (d <= 32) return kTierG32;
  if (d <= A.warp) return kTierWarp;
  if (d <= A.ctas) return kTierCtaS;
  if (d <= A.ctam) return kTierCtaM;
  if (d <= A.ctal) return kTierCtaL;
  return kTierHub;
}

__global__ void __launch_bounds__(kStepThreads, 4) k_phase_step(const __grid_constant__ StepArgs A) {
  __shared__ int ws[32];
  __shared__ double wd[32];
  __shared__ int ok;
  __shared__ int soff[kStepKeys + 1];
  PhaseCtl* const ctl = A.ctl;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t gt = (int64_t)blockIdx.x * kStepThreads + threadIdx.x, nt = (int64_t)gridDim.x * kStepThreads;
  const int64_t gw = gt >> 5, nw = nt >> 5;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  const int64_t nv = A.nv;
  unsigned target = 0;
#define STEP_BARRIER()                                  \
  if (!loop_barrier(ctl, target, &ok)) {                \
    if (lead) atomicAdd(A.err, 1ull);                   \
    return;                                             \
  }
  int64_t nvn = nv;             // vertices of the next phase
  const int64_t* noff = A.off;  // and its offsets and weights
  const double* nwt = A.w;
  if (A.coarsen) {
    // ---- renumber: communities in use get their rank (ascending old id)
    for (int64_t i = gt; i < nv; i += nt) {
      A.used[i] = 0;
      A.cnt[i] = 0;
      A.deg[i] = 0;
      A.cursor[i] = 0;
    }
    for (int64_t i = gt; i <= (int64_t)A.mask; i += nt) {
      A.keys[i] = kNoEntry;
      A.vals[i] = 0.;
      A.first[i] = 0xFFFFFFFFu;
    }
    for (int64_t i = gt; i < A.nwords; i += nt) A.bm[i] = 0u;
    STEP_BARRIER();
    for (int64_t v = gt; v < nv; v += nt) {
      const int c = A.comm[v];
      if (c >= 0) A.used[c] = 1;
    }
    STEP_BARRIER();
    auto used = [&](int64_t i) { return A.used[i]; };
    scan_sums(nv, used, A.bsum, ws);
    STEP_BARRIER();
    // the prefix replaces the flag of ids in use
    scan_apply(nv, used, A.bsum, [&](int64_t i, int x) {
      A.mo[i] = x;
      if (i == nv) A.out->nvp = x;
    }, ws);
    STEP_BARRIER();
    const int64_t nvp = (int64_t)__ldcg(&A.out->nvp);
    // ---- new ids, members and member edges of every coarse vertex; the
    // clustering of the original vertices is composed with the renumber
    for (int64_t v = gt; v < nv; v += nt) {
      const int oc = A.comm[v], c = oc >= 0 ? A.mo[oc] : -1;
      A.newid[v] = c;
      if (c < 0) continue;
      atomicAdd(A.cnt + c, 1);
      atomicAdd(A.deg + c, (int)(A.off[v + 1] - A.off[v]));
    }
    for (int64_t i = gt; i < A.nv0; i += nt) {
      const int v = A.clus[i];
      if (v < 0) continue;
      const int oc = A.comm[v];
      A.clus[i] = oc >= 0 ? A.mo[oc] : -1;
    }
    if (A.gbase)  // communities never span graphs, so neither does the renumber
      for (int64_t i = gt; i <= A.ng; i += nt) A.gbase2[i] = A.mo[A.gbase[i]];
    if (nvp == nv || nvp == 1) {  // graph_gpu.cpp:1391-1392
      if (lead) A.out->done = 1;
      return;
    }
    STEP_BARRIER();
    auto cnt = [&](int64_t i) { return A.cnt[i]; };
    auto deg = [&](int64_t i) { return A.deg[i]; };
    scan_sums(nvp, cnt, A.bsum, ws);
    scan_sums(nvp, deg, A.bsum + gridDim.x, ws);
    STEP_BARRIER();
    scan_apply(nvp, cnt, A.bsum, [&](int64_t i, int x) { A.mo[i] = x; }, ws);
    scan_apply(nvp, deg, A.bsum + gridDim.x, [&](int64_t i, int x) { A.p0[i] = x; }, ws);
    STEP_BARRIER();
    for (int64_t v = gt; v < nv; v += nt) {
      const int c = A.newid[v];
      if (c < 0) continue;
      A.member[A.mo[c] + atomicAdd(A.cursor + c, 1)] = (int)v;
    }
    STEP_BARRIER();
    // ---- list position of every member's first edge
    for (int64_t v = gt; v < nv; v += nt) {
      const int c = A.newid[v];
      if (c < 0) continue;
      const int m0 = A.mo[c], m1 = A.mo[c + 1];
      if (m1 - m0 > kStepBigList) continue;
      int x = A.p0[c];
      for (int i = m0; i < m1; ++i) {
        const int u = A.member[i];
        if (u < v) x += (int)(A.off[u + 1] - A.off[u]);
      }
      A.pos[v] = x;
    }
    for (int64_t c = blockIdx.x; c < nvp; c += gridDim.x) {
      if (A.mo[c + 1] - A.mo[c] <= kStepBigList) continue;  // block-uniform
      int run = A.p0[c];
      for (int64_t b = 0; b < nv; b += 4 * kStepThreads) {
        const int64_t v0 = b + 4 * (int64_t)threadIdx.x;
        int d[4], s = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          d[q] = -1;
          if (v0 + q < nv && A.newid[v0 + q] == c) {
            d[q] = (int)(A.off[v0 + q + 1] - A.off[v0 + q]);
            s += d[q];
          }
        }
        int tot;
        int x = run + block_excl(s, &tot, ws);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (d[q] >= 0) {
            A.pos[v0 + q] = x;
            x += d[q];
          }
        run += tot;
      }
    }
    STEP_BARRIER();
    // ---- edges into the table, by the finished phase's tier lists
    if (A.gbase) {
      for (int64_t v = gw; v < nv; v += nw)
        if (A.newid[v] >= 0) put_edges(A, (int)v, A.off[v], 0, A.off[v + 1] - A.off[v], 32);
    } else {
      const int64_t* to = A.tier_off;
      const int nb = A.nb;
      for (int64_t i = blockIdx.x; i < A.nitems; i += gridDim.x) {
        const int2 it = A.items[i];
        const int v = A.hub_v[it.x];
        const int64_t e0 = A.off[v], s0 = (int64_t)it.y * kHubSeg;
        put_edges(A, v, e0, s0 + 32 * wid, min(A.off[v + 1] - e0, s0 + kHubSeg), kStepThreads);
      }
      const int64_t c0 = to[(int64_t)kTierCtaS * nb], c1 = to[(int64_t)kTierHub * nb];
      for (int64_t i = c0 + blockIdx.x; i < c1; i += gridDim.x) {
        const int v = A.perm[i];
        put_edges(A, v, A.off[v], 32 * wid, A.off[v + 1] - A.off[v], kStepThreads);
      }
      const int64_t w0 = to[(int64_t)kTierWarp * nb];
      for (int64_t i = w0 + gw; i < c0; i += nw) {
        const int v = A.perm[i];
        put_edges(A, v, A.off[v], 0, A.off[v + 1] - A.off[v], 32);
      }
      const int64_t g8 = to[(int64_t)kTierG8 * nb], g16 = to[(int64_t)kTierG16 * nb], g32 = to[(int64_t)kTierG32 * nb];
      put_groups<32>(A, A.perm + g32, w0 - g32, gw, nw);
      put_groups<16>(A, A.perm + g16, g32 - g16, gw, nw);
      put_groups<8>(A, A.perm + g8, g16 - g8, gw, nw);
      put_groups<4>(A, A.perm + to[0], g8 - to[0], gw, nw);
    }
    STEP_BARRIER();
    // ---- rank the entries by their first positions
    for (int64_t i = gt; i <= (int64_t)A.mask; i += nt) {
      if (__ldcg(A.keys + i) == kNoEntry) continue;
      const unsigned f = __ldcg(A.first + i);
      atomicOr(A.bm + (f >> 5), 1u << (f & 31));
    }
    if (A.ordered) sum_in_order(A, nvp, gw, nw);
    STEP_BARRIER();
    auto bits = [&](int64_t i) { return __popc(__ldcg(A.bm + i)); };
    scan_sums(A.nwords, bits, A.bsum, ws);
    STEP_BARRIER();
    scan_apply(A.nwords, bits, A.bsum, [&](int64_t i, int x) {
      if (i < A.nwords) A.wpre[i] = x;
      else A.out->nep = x;
    }, ws);
    STEP_BARRIER();
    const int nep = (int)__ldcg(&A.out->nep);
    auto rank = [&](unsigned f) { return A.wpre[f >> 5] + __popc(__ldcg(A.bm + (f >> 5)) & ((1u << (f & 31)) - 1u)); };
    for (int64_t i = gt; i <= (int64_t)A.mask; i += nt) {
      const unsigned long long key = __ldcg(A.keys + i);
      if (key == kNoEntry) continue;
      const int x = rank(__ldcg(A.first + i));
      A.cadj[x] = (int32_t)(unsigned)key;
      A.cw[x] = __ldcg(A.vals + i);
    }
    for (int64_t c = gt; c <= nvp; c += nt) {
      const unsigned p = (unsigned)A.p0[c];
      A.coff[c] = (int64_t)(p >> 5) < A.nwords ? rank(p) : nep;
    }
    STEP_BARRIER();
    nvn = nvp;
    noff = A.coff;
    nwt = A.cw;
    if (!A.setup) return;
  }
  // ---- set-up of the next phase: k (lane l sums edges l, l+32, ... then a
  // shuffle-down tree, graph_cuda.cu:302-346), weight flags, cuts
  const int nb = A.nbn;
  const int nkeys = kNumTiers * nb;
  {
    unsigned long long bad = 0;
    double amax = 0.;
    for (int64_t v = gw; v < nvn; v += nw) {
      const int64_t s = noff[v], e = noff[v + 1];
      double x = 0., ax = 0.;
      for (int64_t j = s + lane; j < e; j += 32) {
        const double y = nwt[j];
        x += y;
        ax += fabs(y);
        if (!(fabs(y) < 9.0e15) || y != trunc(y)) ++bad;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        x += __shfl_down_sync(NIDO_FULL_MASK, x, o);
        ax += __shfl_down_sync(NIDO_FULL_MASK, ax, o);
      }
      if (lane == 0) {
        A.k[v] = x;
        amax = fmax(amax, ax);
      }
    }
    const bool anybad = __any_sync(NIDO_FULL_MASK, bad != 0);
    if (lane == 0) {
      if (anybad) atomicOr(&A.out->flags[0], 1ull);
      const unsigned long long ab = (unsigned long long)__double_as_longlong(amax);
      if (amax > 0. && __ldcg(&A.out->flags[1]) < ab) atomicMax(&A.out->flags[1], ab);
    }
    for (int64_t i = gt; i < 2 * (nkeys + 1); i += nt) A.counts[i] = 0;  // and the cursors behind them
    if (nb > 0 && blockIdx.x == gridDim.x - 1 && threadIdx.x == kStepThreads - 1) batch_cuts(noff, nvn, nb, A.cuts, A.parts);
  }
  STEP_BARRIER();
  // ---- mass partials (graph_cuda.cu:1786-1804), tier and batch of every vertex
  for (int64_t b = gw; b < 4096; b += nw) {
    double x = 0.;
    for (int64_t i = lane + 32 * b; i < nvn; i += 32 * 4096) x += A.k[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(NIDO_FULL_MASK, x, o);
    if (lane == 0) A.part[b] = x;
  }
  if (nb > 0) {
    unsigned md = 0;
    for (int64_t base = gt - lane; base < nvn; base += nt) {
      const int64_t v = base + lane;
      int key = -1;
      if (v < nvn) {
        const int64_t d = noff[v + 1] - noff[v];
        md = max(md, (unsigned)d);
        if (d > 0) {  // vertices without edges never move: no list
          int lo = 0, hi = nb;
          while (hi - lo > 1) {
            const int mid = (lo + hi) / 2;
            if (A.cuts[mid] <= v) lo = mid; else hi = mid;
          }
          key = step_tier(A, d) * nb + lo;
        }
        A.vkey[v] = key;
      }
      const unsigned peers = __match_any_sync(NIDO_FULL_MASK, key);
      if (key >= 0 && lane == __ffs(peers) - 1) atomicAdd(A.counts + key, __popc(peers));
    }
    md = __reduce_max_sync(NIDO_FULL_MASK, md);
    if (lane == 0 && md) atomicMax(&A.out->maxdeg, (unsigned long long)md);
  }
  STEP_BARRIER();
  // ---- list offsets (every block for itself), the lists, and m
  if (nb > 0) {
    int run = 0;
    for (int t = 0; t <= nkeys; t += kStepThreads) {
      const int i = t + (int)threadIdx.x;
      int tot;
      const int pre = block_excl(i < nkeys ? __ldcg(A.counts + i) : 0, &tot, ws);
      if (i <= nkeys) soff[i] = run + pre;
      run += tot;
    }
    __syncthreads();
    if (blockIdx.x == 0)
      for (int i = threadIdx.x; i <= nkeys; i += kStepThreads) A.toff[i] = soff[i];
    for (int64_t base = gt - lane; base < nvn; base += nt) {
      const int64_t v = base + lane;
      const int key = v < nvn ? A.vkey[v] : -1;
      const unsigned peers = __match_any_sync(NIDO_FULL_MASK, key);
      const int leader = __ffs(peers) - 1;
      int at = 0;
      if (key >= 0 && lane == leader) at = atomicAdd(A.ccur + key, __popc(peers));
      at = __shfl_sync(NIDO_FULL_MASK, at, leader);
      if (key >= 0) A.perm[soff[key] + at + __popc(peers & lanemask_lt())] = (int32_t)v;
    }
  }
  if (blockIdx.x == gridDim.x - 1) {
    const double s = loop_reduce_1024(A.part, 4096, wd);
    if (threadIdx.x == 0) A.out->m = 0.5 * s;
  }
#undef STEP_BARRIER
}

int64_t g_step_resident = kSMs;

int step(nido_graph_s* g, bool coarsen, int* done, bool* unsupported) {
  cudaStream_t s = g->ctx->stream;
  const bool colored = g->color_mode && !g->gid;  // the coarse graph is coloured first: no lists here
  const bool many = g->gid != nullptr;            // only the coarsening
  const int nb = colored || many ? 0 : g->nb_user;
  const int nkeys = kNumTiers * nb;
  const int64_t nold = (int64_t)kNumTiers * g->nbatches;
  *unsupported = true;
  const int64_t nv = g->nv, ne = g->ne;
  if (nv < 1 || nv > kStepMaxEdges || ne > kStepMaxEdges || nkeys > kStepKeys || g->host_edges)
    return NIDO_OK;
  if (many ? !coarsen
           : !loop_plan_fits(g, std::max(nb, 1)) || (coarsen && (!g->loop_plan || !g->bins_valid)))
    return NIDO_OK;
  StepArgs A;
  memset(&A, 0, sizeof(A));
  A.off = g->off;
  A.adj = g->adj;
  A.w = g->w;
  A.nv = nv;
  A.nv0 = g->nv0;
  A.comm = g->comm;
  A.k = g->k;
  A.clus = g->clus;
  A.perm = g->perm;
  A.nb = g->nbatches;
  A.nbn = nb;
  A.nitems = g->nhubs > 0 ? g->hub_nitems : 0;
  A.items = g->hub_items;
  A.hub_v = g->hub_v;
  const int64_t blocks = std::max<int64_t>(1, std::min(g_step_resident, std::max(ne / 256, nv / 128)));
  Arena ar(g->scratch, g->scratch_bytes);
  // results and control first: one memset, one readback
  const int64_t nres = (int64_t)sizeof(StepOut) / 8 + (nb + 1) + (nkeys + 1);
  int64_t* res = ar.take<int64_t>(nres);
  A.ctl = ar.take<PhaseCtl>(1);
  int64_t* tier = ar.take<int64_t>(nold + 1);
  A.parts = ar.take<int64_t>(nb + 2);
  A.counts = ar.take<int32_t>(2 * (nkeys + 1));
  A.bsum = ar.take<int32_t>(2 * blocks);
  A.part = ar.take<double>(4096);
  A.used = ar.take<int32_t>(nv);
  A.newid = ar.take<int32_t>(nv);
  A.cnt = ar.take<int32_t>(nv);
  A.cursor = ar.take<int32_t>(nv);
  A.mo = ar.take<int32_t>(nv + 1);
  A.deg = ar.take<int32_t>(nv);
  A.p0 = ar.take<int32_t>(nv + 1);
  A.member = ar.take<int32_t>(nv);
  A.pos = ar.take<int32_t>(nv);
  A.vkey = ar.take<int32_t>(nv);
  if (!A.vkey) return NIDO_OK;
  A.ccur = A.counts + nkeys + 1;
  A.out = reinterpret_cast<StepOut*>(res);
  A.cuts = res + sizeof(StepOut) / 8;
  A.toff = A.cuts + nb + 1;
  A.tier_off = tier;
  A.coarsen = coarsen;
  A.setup = !many;
  if (many) {
    A.gbase = g->gbase;
    A.gbase2 = g->gbase2;
    A.ng = g->ngraphs;
  }
  A.ordered = !g->int_weights;
  if (coarsen) {
    int64_t slots = 64;
    while (slots < 2 * ne) slots <<= 1;
    A.mask = (unsigned)(slots - 1);
    A.nwords = (ne + 31) / 32;
    const size_t bytes = (size_t)slots * 20 + 8 * (size_t)(A.nwords + 1) + 8 * 256;
    if (bytes > g->agg_buf_bytes) {
      NIDO_CUDA_TRY(cudaStreamSynchronize(s));
      raw_free(g->ctx, g->agg_buf);
      g->agg_buf = nullptr;
      g->agg_buf_bytes = 0;
      NIDO_CUDA_TRY(raw_alloc(g->ctx, (void**)&g->agg_buf, bytes));
      g->agg_buf_bytes = bytes;
    }
    Arena pa(g->agg_buf, g->agg_buf_bytes);
    A.keys = pa.take<unsigned long long>(slots);
    A.vals = pa.take<double>(slots);
    A.first = pa.take<unsigned>(slots);
    A.bm = pa.take<uint32_t>(A.nwords + 1);
    A.wpre = pa.take<int32_t>(A.nwords + 1);
    if (!A.wpre) return NIDO_OK;
    A.coff = g->off2;
    A.cadj = g->adj2;
    A.cw = g->w2;
    if (!many)
      NIDO_CUDA_TRY(cudaMemcpyAsync(tier, g->tier_off.data(), sizeof(int64_t) * (nold + 1), cudaMemcpyHostToDevice, s));
  }
  A.err = reinterpret_cast<unsigned long long*>(g->dcount + 1);
  A.warp = g->cfg.warp_max;
  A.ctas = g->cfg.ctas_max;
  A.ctam = g->cfg.ctam_max;
  A.ctal = kCtaLMaxDeg;
  NIDO_CUDA_TRY(cudaMemsetAsync(res, 0, sizeof(StepOut), s));
  NIDO_CUDA_TRY(cudaMemsetAsync(A.ctl, 0, sizeof(PhaseCtl), s));
  void* ptr[] = {&A};
  NIDO_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_phase_step, dim3((unsigned)blocks), dim3(kStepThreads), ptr, 0, s));
  nido_count_launch();
  std::vector<int64_t> h((size_t)nres);
  PhaseCtl hc;
  int64_t nerr = 0;
  NIDO_CUDA_TRY(cudaMemcpyAsync(h.data(), res, sizeof(int64_t) * nres, cudaMemcpyDeviceToHost, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(&hc, A.ctl, sizeof(hc), cudaMemcpyDeviceToHost, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(&nerr, g->dcount + 1, sizeof(nerr), cudaMemcpyDeviceToHost, s));
  NIDO_CUDA_TRY(cudaStreamSynchronize(s));
  *unsupported = false;
  if (hc.fail) return nido_set_error(NIDO_E_TIMEOUT, "the phase step's grid barrier gave up");
  if (nerr) return nido_set_error(NIDO_E_CUDA, "hash table overflow in %lld probes", (long long)nerr);
  StepOut o;
  memcpy(&o, h.data(), sizeof(o));
  *done = (int)o.done;
  if (o.done) return NIDO_OK;
  if (coarsen) {
    std::swap(g->offA, g->off2);
    std::swap(g->adjA, g->adj2);
    std::swap(g->wA, g->w2);
    g->off = g->offA;
    g->adj = g->adjA;
    g->w = g->wA;
    g->coarsened = true;
    g->nv = o.nvp;
    g->ne = o.nep;
  }
  if (many) {
    g->bins_valid = false;
    return NIDO_OK;
  }
  g->m = o.m;
  // where the separate stages look for them
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->dm, &A.out->m, sizeof(double), cudaMemcpyDeviceToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->dcount + 2, A.out->flags, sizeof(A.out->flags), cudaMemcpyDeviceToDevice, s));
  double amax = 0.;
  memcpy(&amax, &o.flags[1], sizeof(amax));
  g->int_weights = o.flags[0] == 0 && amax < 2147483648.0;
  if (colored) {
    g->bins_valid = false;
    return build_batches(g);
  }
  g->nbatches = nb;
  const int64_t* cuts = h.data() + sizeof(StepOut) / 8;
  g->cuts.assign(cuts, cuts + nb + 1);
  g->tier_off.assign(cuts + nb + 1, cuts + nb + 1 + nkeys + 1);
  g->max_degree = (int64_t)o.maxdeg;
  g->loop_plan = true;
  g->bins_valid = true;
  ++g->plan_epoch;
  return plan_hubs(g);
}

}  // namespace

int phase_step_init() {
  int dev = 0, sms = kSMs, per_sm = 0;
  NIDO_CUDA_TRY(cudaGetDevice(&dev));
  NIDO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  NIDO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_phase_step, kStepThreads, 0));
  static std::mutex mu;  // contexts may be created from several threads
  std::lock_guard<std::mutex> lk(mu);
  g_step_resident = (int64_t)std::max(per_sm, 1) * sms;
  return NIDO_OK;
}

int phase_step(nido_graph_s* g, int* done, bool* unsupported) { return step(g, true, done, unsupported); }

int phase_setup(nido_graph_s* g, bool* unsupported) {
  int done = 0;
  return step(g, false, &done, unsupported);
}

}  // namespace nido
