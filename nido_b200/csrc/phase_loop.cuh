// phase_loop.cuh -- the iteration loop of a Louvain phase as one persistent
// kernel.
//
// Driven from the host, a sweep of a small phase is a chain of some thirty
// launches on three streams and a readback of Q, 200-250 us for work that takes
// the GPU 20 (R-MAT of 20,011 vertices: 62 sweeps, 15 ms).  Here a cooperative
// grid keeps the phase: the move of every tier, the commit and the modularity
// are stages of one kernel with a grid barrier between them, the reference's
// loop control (louvain_gpu.cpp:53-90) runs in the block that finishes Q, and
// the host launches once and reads back once a phase.  The stages are the
// device code of the per-stage kernels (move_core.cuh, hub_core.cuh,
// phase_core.cuh), so results are theirs.
//
// All blocks are resident (cooperative launch).  The barrier's wait is bounded
// by about four seconds; a wait that gives up is counted in p.err, every block
// leaves, and the run returns an error.
#ifndef NIDO_PHASE_LOOP_CUH_
#define NIDO_PHASE_LOOP_CUH_
#include "hub_core.cuh"
#include "move_core.cuh"
#include "phase_core.cuh"

namespace nido {

constexpr int kLoopThreads = 256;
constexpr int kLoopCtaCap = 4096;      // slots of a CTA's table: degrees up to 3072
constexpr int kLoopCtaChunks = kCtaLMaxDeg / kLoopThreads;
constexpr int kLoopWarpCap = 256;      // slots of a warp's table: degrees up to 192
constexpr int kLoopWarpChunks = kWarpMaxDeg / 32;
constexpr unsigned long long kLoopBarrierNs = 4000000000ull;

// state of the loop in device memory, read back by the host
struct PhaseCtl {
  double q, q_old, q_tmp, dq;
  long long loops;
  int go, restore;
  unsigned bar, ticket;       // barrier arrivals and the ticket of the blocks that finished their part of Q
  int fail, pad;
  unsigned long long move_ns, q_ns;
  unsigned long long counters[4];  // many graphs: [0] iterating [1] restoring [2] vertices of iterating graphs
};

template <bool kInts>
struct LoopArgs {
  MoveArgs p;
  int32_t* comm;
  int32_t* newc;
  double* a;
  const int32_t* perm;
  const int64_t* tier_off;    // kNumTiers * nb + 1 list offsets
  const int64_t* cuts;        // nb + 1, or null: a batch is its tier lists (colour classes, many graphs)
  const int64_t* hub_rng;     // per batch: items [0, 1), slices [2, 3)
  int nb;
  int64_t nv, S, ngroups;
  double* selfv;
  double* modv;
  PhaseCtl* ctl;
  double* log;                // Qtmp, dQ of the first log_cap iterations
  int64_t log_cap;
  double tau;
  int64_t max_iter;
  // hubs (null without)
  int64_t nhubs, nitems;
  const int2* items;
  const int2* slices;
  const int64_t* slice_first;
  const int64_t* item_first;
  const int32_t* hub_v;
  const int64_t* hub_toff;
  const int32_t* hub_cap;
  int32_t* hub_done;
  SliceResult* res;
  double* part;
  HubTable<kInts> tab;
  // many graphs: the listed graphs with their modularity groups (qoff), the
  // first nbig reduced by a block each, and the per-graph loop state
  const int32_t* gl;
  const int64_t* qoff;
  int nl, nbig;
  const int64_t* gbase;
  double* gq;
  double* gq_old;
  int32_t* loops_phase;
  int64_t* loops_total;
  int32_t* giter;
  int32_t* grest;
  int64_t relist_below;       // leave the loop when the iterating graphs hold fewer vertices
};

template <bool kTie>
struct LoopTieShared {};
template <>
struct LoopTieShared<true> {
  TieShared ts;
};

__device__ __forceinline__ unsigned long long loop_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Grid barrier: arrivals are counted up from 0 for the whole kernel, so
// nothing is reset.  False when the wait gave up (here or in another block).
__device__ __forceinline__ bool loop_barrier(PhaseCtl* c, unsigned& target, int* ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    unsigned seen = 0;
    // release / acquire: with the block barriers around them, the block's
    // writes before are visible to every block after
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->bar) : "memory");
    const unsigned long long t0 = loop_ns();
    int good = 1;
    for (int i = 0;; ++i) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&c->bar) : "memory");
      if ((int)(seen - target) >= 0) break;
      if ((i & 255) == 255 && (*(volatile int*)&c->fail || loop_ns() - t0 > kLoopBarrierNs)) {
        *(volatile int*)&c->fail = 1;
        good = 0;
        break;
      }
    }
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

// The reference's 1024-thread reduction (reduce_vector_kernel<32><<<1,1024>>>,
// graph_cuda.cu:1806-1835) of x[0, n) by a block of 256: every thread is four
// of its threads.  The sum in thread 0; ws: 32 doubles.
__device__ __forceinline__ double loop_reduce_1024(const double* x, int64_t n, double* ws) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double s[4] = {0., 0., 0., 0.};
  for (int64_t b = 0; b < n; b += 1024) {
    double y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = b + 256 * j + threadIdx.x;
      y[j] = i < n ? __ldcg(x + i) : 0.;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (b + 256 * j + threadIdx.x < n) s[j] += y[j];
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[j] += __shfl_down_sync(NIDO_FULL_MASK, s[j], o);
    if (lane == 0) ws[8 * j + wid] = s[j];
  }
  __syncthreads();
  double t = 0.;
  if (wid == 0) {
    t = ws[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(NIDO_FULL_MASK, t, o);
  }
  __syncthreads();
  return t;
}

// largest i in [0, n) with offs[i] <= x
__device__ __forceinline__ int loop_find(const int64_t* __restrict__ offs, int n, int64_t x) {
  int lo = 0, hi = n;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (offs[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

// Four blocks of 256 threads an SM (64 registers): the tables take 32 KB
// (integer phases) or 48 KB of shared memory a block.
template <bool kMulti, bool kInts, bool kTie>
__global__ void __launch_bounds__(kLoopThreads, 4) k_phase_loop(const __grid_constant__ LoopArgs<kInts> A) {
  extern __shared__ __align__(128) double smem[];
  __shared__ CtaShared sh;
  __shared__ HubShared hs;
  __shared__ LoopTieShared<kTie> tie;
  __shared__ int fold[kLoopThreads];
  __shared__ double ws[32];
  __shared__ int flag, ok;
  const MoveArgs& p = A.p;
  PhaseCtl* const ctl = A.ctl;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t gw = (int64_t)blockIdx.x * (kLoopThreads / 32) + wid;
  const int64_t nw = (int64_t)gridDim.x * (kLoopThreads / 32);
  const int64_t gt = (int64_t)blockIdx.x * kLoopThreads + threadIdx.x;
  const int64_t nt = (int64_t)gridDim.x * kLoopThreads;
  // the CTA's table; the warps' tables are parts of it
  SharedTable<kInts> t, tw;
  t.place(smem, kLoopCtaCap);
  tw = t;
  if constexpr (kInts) {
    tw.slots += wid * kLoopWarpCap;
  } else {
    tw.vals += wid * kLoopWarpCap;
    tw.keys += wid * kLoopWarpCap;
  }
  for (int i = threadIdx.x; i < kLoopCtaCap; i += kLoopThreads) t.clear(i);
  if (threadIdx.x == 0) sh.eown = 0.;
  __syncthreads();
  unsigned target = 0;
  unsigned long long move_ns = 0, q_ns = 0, t0 = 0;
  const bool clock = blockIdx.x == 0 && threadIdx.x == 0;
  const int nb = A.nb;
  long long loops = 0;
  for (bool first = !kMulti || A.gq_old != nullptr;;) {
    if (!first) {
      for (int b = 0; b < nb; ++b) {
        if (clock) t0 = loop_ns();
        const int64_t* to = A.tier_off + b;
        // ---- move: hub segments, CTA tiers, warp tier, lane groups.  Each
        // tier starts at the block (warp) after the last one's end.
        int64_t rot = 0;
        if (A.nhubs > 0) {
          const int64_t i0 = A.hub_rng[4 * b], n = A.hub_rng[4 * b + 1] - i0;
          for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
            const int2 it = A.items[i0 + i];
            hub_segment<kInts>(p, A.hub_v[it.x], it.y, A.tab.at(A.hub_toff[it.x]), A.hub_cap[it.x]);
          }
          rot = n % gridDim.x;
        }
        // A vertex of 100 to 190 edges takes a warp eight to ten microseconds,
        // chunk after chunk, and a CTA three: while the batch has at most two of
        // them a block, CTAs take the warp tier as well.  Integer phases only: a
        // CTA's FP64 sums are atomic, a warp's are in a fixed order.
        const int64_t nwarp = to[(int64_t)kTierWarp * nb + 1] - to[(int64_t)kTierWarp * nb];
        const int lowest = kInts && nwarp <= 2 * (int64_t)gridDim.x ? kTierWarp : kTierCtaS;
        for (int tier = kTierCtaL; tier >= lowest; --tier) {
          const int64_t l0 = to[(int64_t)tier * nb], n = to[(int64_t)tier * nb + 1] - l0;
          int64_t i = (int64_t)blockIdx.x - rot;
          if (i < 0) i += gridDim.x;
          for (; i < n; i += gridDim.x) {
            const int v = A.perm[l0 + i];
            const int64_t s = p.off[v];
            const int d = (int)(p.off[v + 1] - s);
            const int own = p.comm[v];
            cta_vertex<kLoopThreads, kLoopCtaCap, kLoopCtaChunks, kInts, kTie, false>(
                p, vertex_mass<kMulti>(p, v), v, p.adj + s, p.w + s, d, own, p.k[v], p.a[own], t, sh, []() {});
          }
          rot = (rot + n) % gridDim.x;
        }
        int64_t wr = gw - rot * (kLoopThreads / 32);
        if (wr < 0) wr += nw;
        const int32_t* list = A.perm + to[(int64_t)kTierWarp * nb];
        int64_t n = lowest == kTierWarp ? 0 : nwarp;
        warp_list<kLoopWarpCap, kLoopWarpChunks, kMulti, kInts, kTie>(list, n, wr, nw, p, tw);
        auto rotate = [&](int64_t used) {
          wr -= used % nw;
          if (wr < 0) wr += nw;
        };
        rotate(n);
        list = A.perm + to[(int64_t)kTierG32 * nb];
        n = to[(int64_t)kTierG32 * nb + 1] - to[(int64_t)kTierG32 * nb];
        group_list<32, kMulti, kTie>(list, n, wr, nw, p, fold + 32 * wid);
        rotate(n);
        list = A.perm + to[(int64_t)kTierG16 * nb];
        n = to[(int64_t)kTierG16 * nb + 1] - to[(int64_t)kTierG16 * nb];
        group_list<16, kMulti, kTie>(list, n, wr, nw, p, fold + 32 * wid);
        rotate((n + 1) / 2);
        list = A.perm + to[(int64_t)kTierG8 * nb];
        n = to[(int64_t)kTierG8 * nb + 1] - to[(int64_t)kTierG8 * nb];
        group_list<8, kMulti, kTie>(list, n, wr, nw, p, fold + 32 * wid);
        rotate((n + 3) / 4);
        list = A.perm + to[(int64_t)kTierG4 * nb];
        n = to[(int64_t)kTierG4 * nb + 1] - to[(int64_t)kTierG4 * nb];
        group_list<4, kMulti, kTie>(list, n, wr, nw, p, fold + 32 * wid);
        if (!loop_barrier(ctl, target, &ok)) goto failed;
        if (A.nhubs > 0) {
          // ---- the filled hub tables of this batch
          const int64_t s0 = A.hub_rng[4 * b + 2], ns = A.hub_rng[4 * b + 3] - s0;
          if (ns > 0) {
            if constexpr (kTie) {
              // one block per hub: its first slice stands for it
              for (int64_t i = blockIdx.x; i < ns; i += gridDim.x) {
                const int2 sl = A.slices[s0 + i];
                if (sl.y == 0)
                  hub_tie<kMulti, kInts>(p, A.hub_v[sl.x], A.tab.at(A.hub_toff[sl.x]), A.hub_cap[sl.x], hs, tie.ts);
              }
            } else {
              for (int64_t i = blockIdx.x; i < ns; i += gridDim.x) {
                const int2 sl = A.slices[s0 + i];
                const int len = min(kHubSlice, A.hub_cap[sl.x] - sl.y * kHubSlice);
                const SliceResult r = hub_slice<kMulti, kInts>(
                    p, A.hub_v[sl.x], A.tab.at(A.hub_toff[sl.x] + (int64_t)sl.y * kHubSlice), len, hs);
                const int64_t r0 = A.slice_first[sl.x], nr = A.slice_first[sl.x + 1] - r0;
                if (threadIdx.x == 0) {
                  A.res[s0 + i] = r;
                  __threadfence();
                  flag = atomicAdd(&A.hub_done[sl.x], 1) == (int)nr - 1;  // nobody waits
                }
                __syncthreads();
                if (flag) {
                  __threadfence();
                  if (wid == 0) hub_combine<kMulti>(p, A.hub_v[sl.x], A.res + r0, nr);
                  if (threadIdx.x == 0) A.hub_done[sl.x] = 0;
                }
                __syncthreads();
              }
            }
            if (!loop_barrier(ctl, target, &ok)) goto failed;
          }
        }
        if (clock) move_ns += loop_ns() - t0;
        // ---- commit
        if (A.cuts) {
          const int64_t v1 = A.cuts[b + 1];
          for (int64_t base = A.cuts[b] + gt - lane; base < v1; base += nt) {
            const int64_t v = base + lane;
            commit_vertex(v, v < v1, p.k, A.comm, A.newc, A.a);
          }
        } else {
          for (int tier = 0; tier < kNumTiers; ++tier) {
            const int64_t l0 = to[(int64_t)tier * nb], m = to[(int64_t)tier * nb + 1] - l0;
            for (int64_t base = gt - lane; base < m; base += nt) {
              const int64_t x = base + lane;
              int v = 0;
              bool in = x < m;
              if (in) {
                v = A.perm[l0 + x];
                if (kMulti && !__ldcg(&A.giter[p.gid[v]])) in = false;
              }
              commit_vertex(v, in, p.k, A.comm, A.newc, A.a);
            }
          }
        }
        if (!loop_barrier(ctl, target, &ok)) goto failed;
      }
    }
    if (clock) t0 = loop_ns();
    // ---- modularity: in-community weight of every listed vertex
    if (kMulti && clock)
      for (int i = 0; i < 4; ++i) ctl->counters[i] = 0ull;
    {
      int64_t rot = 0;
      if (A.nhubs > 0) {
        for (int64_t i = blockIdx.x; i < A.nitems; i += gridDim.x) {
          const int2 it = A.items[i];
          const int v = A.hub_v[it.x];
          const int64_t e0 = p.off[v], e1 = p.off[v + 1];
          if (e1 - e0 <= kCtaXMaxDeg) {  // the first segment's block takes the vertex
            if (it.y == 0) {
              const double s = q_self_block<kLoopThreads>(p.adj, p.w, p.comm, p.comm[v], e0, e1, ws);
              if (threadIdx.x == 0) A.selfv[v] = s;
            }
            continue;
          }
          const int64_t s0 = e0 + (int64_t)it.y * kHubSeg;
          const double s = q_self_block<kLoopThreads>(p.adj, p.w, p.comm, p.comm[v], s0, min(e1, s0 + kHubSeg), ws);
          const int64_t f0 = A.item_first[it.x], nf = A.item_first[it.x + 1] - f0;
          if (threadIdx.x == 0) {
            A.part[i] = s;
            __threadfence();
            flag = atomicAdd(&A.hub_done[it.x], 1) == (int)nf - 1;
          }
          __syncthreads();
          if (flag) {
            __threadfence();
            if (wid == 0) {  // the segments' sums, as k_q_hub_sum adds them
              double x = 0.;
              for (int64_t j = lane; j < nf; j += 32) x += __ldcg(A.part + f0 + j);
#pragma unroll
              for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(NIDO_FULL_MASK, x, o);
              if (lane == 0) A.selfv[v] = x;
            }
            if (threadIdx.x == 0) A.hub_done[it.x] = 0;
          }
          __syncthreads();
        }
        rot = A.nitems % gridDim.x;
      }
      const int64_t* to = A.tier_off;
      {
        const int64_t l0 = to[(int64_t)kTierCtaL * nb], n = to[(int64_t)(kTierCtaL + 1) * nb] - l0;
        int64_t i = (int64_t)blockIdx.x - rot;
        if (i < 0) i += gridDim.x;
        for (; i < n; i += gridDim.x) {
          const int v = A.perm[l0 + i];
          const double s = q_self_block<kLoopThreads>(p.adj, p.w, p.comm, p.comm[v], p.off[v], p.off[v + 1], ws);
          if (threadIdx.x == 0) A.selfv[v] = s;
        }
        rot = (rot + n) % gridDim.x;
      }
      int64_t wr = gw - rot * (kLoopThreads / 32);
      if (wr < 0) wr += nw;
      // CTA-M, CTA-S, warp and 32-lane tiers, largest degrees first
      for (int tier = kTierCtaM; tier >= kTierG32; --tier) {
        const int64_t l0 = to[(int64_t)tier * nb], n = to[(int64_t)(tier + 1) * nb] - l0;
        q_self_list<32>(A.perm + l0, n, wr, nw, p.off, p.adj, p.w, p.comm, A.selfv);
        wr -= n % nw;
        if (wr < 0) wr += nw;
      }
      const int64_t o16 = to[(int64_t)kTierG16 * nb], o8 = to[(int64_t)kTierG8 * nb], o4 = to[(int64_t)kTierG4 * nb];
      const int64_t e16 = to[(int64_t)kTierG32 * nb];
      q_self_list<16>(A.perm + o16, e16 - o16, wr, nw, p.off, p.adj, p.w, p.comm, A.selfv);
      q_self_list<8>(A.perm + o8, o16 - o8, wr, nw, p.off, p.adj, p.w, p.comm, A.selfv);
      q_self_list<4>(A.perm + o4, o8 - o4, wr, nw, p.off, p.adj, p.w, p.comm, A.selfv);
    }
    if (!loop_barrier(ctl, target, &ok)) goto failed;
    if constexpr (!kMulti) {
      // the reference's thread slots and 16-lane groups
      // (compute_modularity_reduce_kernel<128,16>, graph_cuda.cu:2096-2134)
      for (int64_t base = gt - threadIdx.x; base < A.ngroups * 16; base += nt) {
        const int64_t x = base + threadIdx.x;
        double s = 0., ac = 0.;
        if (x < A.ngroups * 16) {
          for (int64_t v = x; v < A.nv; v += A.S) {
            s += A.selfv[v];
            ac = fma(A.a[v], A.a[v], ac);
          }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          s += __shfl_down_sync(NIDO_FULL_MASK, s, o, 16);
          ac += __shfl_down_sync(NIDO_FULL_MASK, ac, o, 16);
        }
        if ((x & 15) == 0 && x < A.ngroups * 16) A.modv[x >> 4] = q_part(s, ac, p.m);
      }
      // the block that finishes last reduces the groups and decides
      // (louvain_gpu.cpp:76-90); the others go on to the barrier
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0) flag = atomicAdd(&ctl->ticket, 1u) == gridDim.x - 1;
      __syncthreads();
      if (flag) {
        __threadfence();
        const double qt = loop_reduce_1024(A.modv, A.ngroups, ws);
        if (threadIdx.x == 0) {
          ctl->ticket = 0u;
          if (first) {
            ctl->q = ctl->q_old = qt;
            ctl->restore = 0;
            ctl->go = A.max_iter > 0;
          } else {
            const double dq = __dsub_rn(qt, ctl->q);
            ctl->dq = dq;
            ctl->restore = dq < 0;
            if (!(dq < 0)) ctl->q = qt;
            if (loops < A.log_cap) {
              A.log[2 * loops] = qt;
              A.log[2 * loops + 1] = dq;
            }
            ctl->loops = loops + 1;
            ctl->go = A.tau < dq && loops + 1 < A.max_iter;
          }
        }
      }
    } else {
      // the same per graph, each with the shapes of a run of that graph alone
      const int64_t total = A.qoff[A.nl] * 16;
      for (int64_t base = gt - threadIdx.x; base < total; base += nt) {
        const int64_t x = base + threadIdx.x;
        double s = 0., ac = 0., m = 0.;
        if (x < total) {
          const int i = loop_find(A.qoff, A.nl, x >> 4);
          const int g = A.gl[i];
          const int64_t gb = A.gbase[g], nvg = A.gbase[g + 1] - gb;
          int64_t grid = (nvg + 7) / 8;
          if (grid > 65535) grid = 65535;
          const int64_t S = 128 * grid;
          for (int64_t v = ((x >> 4) - A.qoff[i]) * 16 + (x & 15); v < nvg; v += S) {
            s += A.selfv[gb + v];
            ac = fma(A.a[gb + v], A.a[gb + v], ac);
          }
          m = p.mg[g];
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
          s += __shfl_down_sync(NIDO_FULL_MASK, s, o, 16);
          ac += __shfl_down_sync(NIDO_FULL_MASK, ac, o, 16);
        }
        if ((x & 15) == 0 && x < total) A.modv[x >> 4] = q_part(s, ac, m);
      }
      if (!loop_barrier(ctl, target, &ok)) goto failed;
      // per graph: Q, then its loop control
      auto control = [&](int i, double qt) {
        const int g = A.gl[i];
        if (first) {
          A.gq[g] = qt;
          A.gq_old[g] = qt;
          A.grest[g] = 0;
          if (A.giter[g]) atomicAdd(&ctl->counters[0], 1ull);
          return;
        }
        A.grest[g] = 0;
        if (!A.giter[g]) return;
        const double dq = qt - A.gq[g];
        const int lp = ++A.loops_phase[g];
        A.loops_total[g] += 1;
        if (dq < 0) {
          A.grest[g] = 1;
          atomicAdd(&ctl->counters[1], 1ull);
        } else {
          A.gq[g] = qt;
        }
        const bool go = A.tau < dq && lp < A.max_iter;
        A.giter[g] = go ? 1 : 0;
        if (go) {
          atomicAdd(&ctl->counters[0], 1ull);
          atomicAdd(&ctl->counters[2], (unsigned long long)(A.gbase[g + 1] - A.gbase[g]));
        }
      };
      for (int i = blockIdx.x; i < A.nbig; i += gridDim.x) {
        const double qt = loop_reduce_1024(A.modv + A.qoff[i], A.qoff[i + 1] - A.qoff[i], ws);
        if (threadIdx.x == 0) control(i, qt);
      }
      // at most 1024 values: one warp replays the 32 virtual warps' trees
      for (int64_t i = A.nbig + gw; i < A.nl; i += nw) {
        const double* x = A.modv + A.qoff[i];
        const int64_t cnt = A.qoff[i + 1] - A.qoff[i];
        double mine = 0.;
        for (int w = 0; 32 * w < cnt; ++w) {
          double s = 0.;
          const int64_t j = 32 * w + lane;
          if (j < cnt) s += __ldcg(x + j);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(NIDO_FULL_MASK, s, o);
          const double r = __shfl_sync(NIDO_FULL_MASK, s, 0);
          if (lane == w) mine = r;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_down_sync(NIDO_FULL_MASK, mine, o);
        if (lane == 0) control((int)i, mine);
      }
    }
    if (!loop_barrier(ctl, target, &ok)) goto failed;
    if (clock) q_ns += loop_ns() - t0;
    bool go, restore;
    if constexpr (!kMulti) {
      go = __ldcg(&ctl->go) != 0;
      restore = __ldcg(&ctl->restore) != 0;
    } else {
      const unsigned long long it = __ldcg(&ctl->counters[0]);
      restore = __ldcg(&ctl->counters[1]) != 0ull;
      go = it > 0ull && (first || (int64_t)__ldcg(&ctl->counters[2]) >= A.relist_below);
    }
    if (!first) ++loops;
    first = false;
    if (restore) {  // undo the sweep that lowered Q
      if constexpr (!kMulti) {
        for (int64_t base = gt - lane; base < A.nv; base += nt)
          commit_vertex(base + lane, base + lane < A.nv, p.k, A.comm, A.newc, A.a);
      } else {
        const int64_t m = A.tier_off[(int64_t)kNumTiers * nb];
        for (int64_t base = gt - lane; base < m; base += nt) {
          const int64_t x = base + lane;
          int v = 0;
          bool in = x < m;
          if (in) {
            v = A.perm[x];
            in = __ldcg(&A.grest[p.gid[v]]) != 0;
          }
          commit_vertex(v, in, p.k, A.comm, A.newc, A.a);
        }
      }
    }
    if (!go) break;
    if (kMulti || restore) {  // many graphs: the counters are read before they are reset
      if (!loop_barrier(ctl, target, &ok)) goto failed;
    }
  }
  if (clock) {
    ctl->move_ns = move_ns;
    ctl->q_ns = q_ns;
    ctl->loops = loops;
  }
  return;
failed:
  if (clock) atomicAdd(p.err, 1ull);
}

template <bool kMulti, bool kInts>
struct PhaseLoopKernel {
  // shared-memory attribute and resident blocks per SM, [tie rule]
  static int init(int sms, int64_t resident[2]);
  static int launch(const LoopArgs<kInts>& A, bool tie, int64_t blocks, cudaStream_t s);
};

constexpr size_t loop_smem(bool ints) { return table_bytes(kLoopCtaCap, ints); }

#ifdef NIDO_LOOP_KERNELS
template <bool kMulti, bool kInts>
int PhaseLoopKernel<kMulti, kInts>::init(int sms, int64_t resident[2]) {
  auto one = [sms](auto kernel, int64_t* out) -> int {
    NIDO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)loop_smem(kInts)));
    int per_sm = 0;
    NIDO_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kLoopThreads, loop_smem(kInts)));
    *out = (int64_t)per_sm * sms;
    return NIDO_OK;
  };
  NIDO_TRY(one(k_phase_loop<kMulti, kInts, false>, &resident[0]));
  return one(k_phase_loop<kMulti, kInts, true>, &resident[1]);
}

template <bool kMulti, bool kInts>
int PhaseLoopKernel<kMulti, kInts>::launch(const LoopArgs<kInts>& A, bool tie, int64_t blocks, cudaStream_t s) {
  LoopArgs<kInts> args = A;
  void* ptr[] = {&args};
  const void* k = tie ? (const void*)k_phase_loop<kMulti, kInts, true> : (const void*)k_phase_loop<kMulti, kInts, false>;
  NIDO_CUDA_TRY(cudaLaunchCooperativeKernel(k, dim3((unsigned)blocks), dim3(kLoopThreads), ptr, loop_smem(kInts), s));
  nido_count_launch();
  return NIDO_OK;
}
#endif

}  // namespace nido
#endif
