// move.cu -- the Louvain move phase for one -b batch.
//
// Replaces the reference's sort-based move (graph_gpu.cpp:457-517 +
// louvain_update_kernel, graph_cuda.cu:1450-1540): instead of building
// (vertex, community) keys for every edge and sorting them, each vertex's
// neighbour-community weights e_vc are accumulated on chip:
//   degree <= 32       a group of 4/8/16/32 lanes holds one edge per lane;
//                      equal communities are found with __match_any_sync and
//                      their weights folded (registers only)
//   degree <= 192      one warp, open-addressing table in shared memory
//   degree <= 12288    one CTA of 128 to 1024 threads, table in shared memory
//   larger             many CTAs, tables in L2-resident global memory
// The device code is in move_core.cuh and hub_core.cuh, the kernels of the
// tiers below the hubs in move_tiers.cuh.
// Gains and the final decision use the reference's operation order
// (graph_cuda.cu:1505-1506, 1530-1533):
//   gain_c = (e_vc - ki*a_c/(2m)) / m,  self = (e_own - ki*(a_own-ki)/(2m)) / m,
//   move to the best c when gain_best - self > 0.
// Self-loops contribute weight 0 but their community still counts as a
// neighbour community (copy_weights_exclude_self_loops_kernel,
// graph_cuda.cu:2306-2316).  Equal gains go to the smallest community id, or,
// with NIDO_TIE_NIDO, to the entry the reference's 8-lane strided scan and
// shuffle tree picks: among tied entries of rank r in the id-sorted list of
// the vertex's neighbour communities, the smallest (bitrev3(r mod 8), r).
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "engine.cuh"
#include "hub_core.cuh"
#include "move_core.cuh"
#include "move_tiers.cuh"

namespace nido {
namespace {

namespace cg = cooperative_groups;

// Self-check of the bounded waits: one thread waits on an mbarrier that
// expects an arrival nobody makes.  The wait must give up and the kernel
// report it (out[0] = 1, out[1] = milliseconds waited), leaving the context
// usable.
__global__ void k_check_bounded_wait(int32_t* out) {
  __shared__ unsigned long long bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  const unsigned long long t0 = gtimer_ns();
  const bool done = mbar_wait(&bar, 0);
  out[0] = done ? 0 : 1;
  out[1] = (int32_t)min((gtimer_ns() - t0) / 1000000ull, 1ull << 30);
}

// ---- hubs: segments of kHubSeg edges, tables in global memory ----------------------
// The reference's tie rule: each CTA takes one (hub, segment) item and merges
// its edges into the hub's table; the CTA that finishes a hub's last segment (an
// atomic ticket; nobody waits) evaluates and clears the table.
template <bool kMulti, bool kInts>
__global__ void __launch_bounds__(kHubThreads) k_move_hub(const int2* __restrict__ items, int64_t n,
                                                          const int32_t* __restrict__ hub_v,
                                                          const int64_t* __restrict__ hub_toff,
                                                          const int32_t* __restrict__ hub_cap,
                                                          const int32_t* __restrict__ hub_nseg,
                                                          int32_t* __restrict__ hub_done, HubTable<kInts> tab,
                                                          MoveArgs p) {
  __shared__ HubShared sh;
  __shared__ TieShared ts;
  __shared__ int last_s;
  for (int64_t it = blockIdx.x; it < n; it += gridDim.x) {
    const int2 item = items[it];
    const int h = item.x;
    const int v = hub_v[h];
    const HubTable<kInts> t = tab.at(hub_toff[h]);
    hub_segment<kInts>(p, v, item.y, t, hub_cap[h]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_s = atomicAdd(&hub_done[h], 1) == hub_nseg[h] - 1;
    __syncthreads();
    if (last_s) {
      __threadfence();
      hub_tie<kMulti, kInts>(p, v, t, hub_cap[h], sh, ts);
      if (threadIdx.x == 0) hub_done[h] = 0;
    }
    __syncthreads();
  }
}

// The smallest-id rule: segments only merge (k_hub_insert), then every
// kHubSlice-slot slice of a table is scanned and cleared by its own CTA
// (k_hub_slices), and one warp per hub combines the slice results
// (k_hub_combine).  The table slots of one wave of hubs come from the graph's
// tier configuration (default 4M slots: 48 MB of keys and values, which leaves
// room in the 126 MB L2 for the streamed adjacency and the gathers).
template <bool kInts>
__global__ void __launch_bounds__(kHubThreads) k_hub_insert(const int2* __restrict__ items, int64_t n,
                                                            const int32_t* __restrict__ hub_v,
                                                            const int64_t* __restrict__ hub_toff,
                                                            const int32_t* __restrict__ hub_cap, HubTable<kInts> tab,
                                                            MoveArgs p) {
  for (int64_t it = blockIdx.x; it < n; it += gridDim.x) {
    const int2 item = items[it];
    const int h = item.x;
    hub_segment<kInts>(p, hub_v[h], item.y, tab.at(hub_toff[h]), hub_cap[h]);
  }
}

template <bool kMulti, bool kInts>
__global__ void __launch_bounds__(kHubThreads) k_hub_slices(const int2* __restrict__ slices, int64_t n,
                                                            const int32_t* __restrict__ hub_v,
                                                            const int64_t* __restrict__ hub_toff,
                                                            const int32_t* __restrict__ hub_cap, HubTable<kInts> tab,
                                                            MoveArgs p, SliceResult* __restrict__ res) {
  __shared__ HubShared sh;
  for (int64_t it = blockIdx.x; it < n; it += gridDim.x) {
    const int2 sl = slices[it];
    const int len = min(kHubSlice, hub_cap[sl.x] - sl.y * kHubSlice);
    const SliceResult r =
        hub_slice<kMulti, kInts>(p, hub_v[sl.x], tab.at(hub_toff[sl.x] + (int64_t)sl.y * kHubSlice), len, sh);
    if (threadIdx.x == 0) res[it] = r;
  }
}

__global__ void k_fill_u64(unsigned long long* __restrict__ x, int64_t n, unsigned long long val) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    x[i] = val;
}

template <bool kMulti>
__global__ void k_hub_combine(int64_t nh, const int32_t* __restrict__ hub_v, const int64_t* __restrict__ slice_first,
                              const SliceResult* __restrict__ res, MoveArgs p) {
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t h = warp; h < nh; h += nw) {
    const int64_t r0 = slice_first[h], r1 = slice_first[h + 1];
    if (r1 > r0) hub_combine<kMulti>(p, hub_v[h], res + r0, r1 - r0);  // else a hub of another batch
  }
}

// ---- hubs in thread-block clusters (integer-weight phases) ---------------------
// One cluster of kCtas CTAs per hub: the hub's table spans the clusters'
// shared memory, kClSlots slots in each CTA, so every insert is a
// distributed-shared-memory access instead of an L2 round trip.  The edges
// are spread over all warps of the cluster; after a cluster barrier each CTA
// evaluates (and clears) its own slots, the per-CTA bests meet in rank 0's
// shared memory, and after a second barrier rank 0 decides.  Sums are int32
// (integer weights, every vertex's sum of |w| below 2^31), so the shared
// atomics are native 32-bit ones and exact; the smallest-id tie rule picks
// the same entry in any order of evaluation.
constexpr int kClThreads = 1024;
constexpr int kClSlots = 16384;   // 192 KB of keys and values per CTA
constexpr int kClusterBins = 4;   // clusters of 2, 4, 8 and 16 CTAs

constexpr int64_t cluster_max_degree(int bin) { return (int64_t)(2 << bin) * kClSlots * 3 / 4; }

// cluster size bin of a hub of degree d (-1: more than a 16-CTA table holds)
inline int cluster_bin(int64_t d) {
  for (int b = 0; b < kClusterBins; ++b)
    if (d <= cluster_max_degree(b)) return b;
  return -1;
}

// whether clusters of each size can be resident on this GPU (set once per
// process by move_init_attributes; unlaunchable bins keep hubs on the
// global-memory path)
bool g_cluster_ok[kClusterBins] = {false, false, false, false};
inline bool cluster_launchable(int bin) { return bin >= 0 && g_cluster_ok[bin]; }

__device__ __forceinline__ void cluster_add(cg::cluster_group& cl, int* keys, double* vals, unsigned mask, int c,
                                            int x, unsigned long long* err) {
  unsigned h = hash_slot(c, mask);
  for (unsigned probe = 0; probe <= mask; ++probe) {
    const unsigned owner = h / kClSlots, loc = h % kClSlots;
    int* kp = cl.map_shared_rank(keys, owner) + loc;
    const int kk = *reinterpret_cast<volatile int*>(kp);
    bool hit = kk == c;
    if (!hit && kk == -1) {
      const int old = atomicCAS(kp, -1, c);
      hit = old == -1 || old == c;
    }
    if (hit) {
      atomicAdd(reinterpret_cast<int*>(cl.map_shared_rank(vals, owner) + loc), x);
      return;
    }
    h = (h + 1) & mask;
  }
  atomicAdd(err, 1ull);
}

template <int kCtas, bool kMulti>
__global__ void __launch_bounds__(kClThreads, 1) k_move_cluster(const int32_t* __restrict__ list, int64_t n,
                                                                MoveArgs p) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ double smem[];
  double* vals = smem;                                    // int32 sums in the low words
  int* keys = reinterpret_cast<int*>(smem + kClSlots);
  __shared__ double sg[32], se[32];
  __shared__ unsigned long long stk[32];
  __shared__ int sc[32];
  __shared__ double rg[kCtas], re[kCtas];                 // the ranks' bests, in rank 0
  __shared__ unsigned long long rtk[kCtas];
  __shared__ int rc[kCtas];
  constexpr unsigned kMask = (unsigned)kCtas * kClSlots - 1;
  constexpr int kWarps = kCtas * (kClThreads / 32);
  const unsigned rank = cluster.block_rank();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int gw = (int)rank * (kClThreads / 32) + wid;
  for (int i = threadIdx.x; i < kClSlots; i += kClThreads) { keys[i] = -1; vals[i] = 0.; }
  cluster.sync();
  const int64_t ncl = gridDim.x / kCtas;
  for (int64_t task = blockIdx.x / kCtas; task < n; task += ncl) {
    const int v = list[task];
    const int64_t s = p.off[v], e = p.off[v + 1];
    for (int64_t base = s + (int64_t)gw * 32; base < e; base += (int64_t)4 * kWarps * 32) {
      int u[4], c[4];
      double wt[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int64_t j = base + (int64_t)k * kWarps * 32 + lane;
        u[k] = -1;
        wt[k] = 0.;
        if (j < e) {
          u[k] = p.adj[j];
          wt[k] = p.w[j];
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        c[k] = u[k] >= 0 ? p.comm[u[k]] : -1;
        if (u[k] == v) wt[k] = 0.;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const bool ok = u[k] >= 0;
        if (!__any_sync(NIDO_FULL_MASK, ok)) break;
        const unsigned peers = __match_any_sync(NIDO_FULL_MASK, c[k]);
        const double x = fold_peers(peers, ok, wt[k]);
        if (ok && lane == __ffs(peers) - 1) cluster_add(cluster, keys, vals, kMask, c[k], __double2int_rn(x), p.err);
      }
    }
    cluster.sync();  // every insert of this hub is in place
    const int own = p.comm[v];
    const double ki = p.k[v], aown = p.a[own];
    const Mass m = vertex_mass<kMulti>(p, v);
    double g = -NIDO_MAX_FLOAT, eown = 0.;
    unsigned long long tk = kNoKey;
    int cand = -1;
    for (int i0 = threadIdx.x; i0 < kClSlots; i0 += 4 * kClThreads) {
      int cc[4];
      double val[4], ac[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int i = i0 + k * kClThreads;
        cc[k] = keys[i];
        val[k] = (double)*reinterpret_cast<const int*>(vals + i);
        if (cc[k] >= 0) {  // this thread is the slot's only reader
          keys[i] = -1;
          vals[i] = 0.;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) ac[k] = (cc[k] >= 0 && cc[k] != own) ? p.a[cc[k]] : 0.;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (cc[k] < 0) continue;
        if (cc[k] == own) {
          eown = val[k];
        } else {
          const double gg = gain_of(val[k], ki, ac[k], m);
          if (better(gg, (unsigned)cc[k], g, tk)) { g = gg; tk = (unsigned)cc[k]; cand = cc[k]; }
        }
      }
    }
    eown = group_sum<32>(eown);  // nonzero in one lane of the cluster at most: exact
    group_best<32>(g, tk, cand);
    if (lane == 0) { sg[wid] = g; stk[wid] = tk; sc[wid] = cand; se[wid] = eown; }
    __syncthreads();
    if (wid == 0) {
      g = sg[lane];
      tk = stk[lane];
      cand = sc[lane];
      double e2 = se[lane];
      group_best<32>(g, tk, cand);
      e2 = group_sum<32>(e2);
      if (lane == 0) {
        *cluster.map_shared_rank(&rg[rank], 0) = g;
        *cluster.map_shared_rank(&rtk[rank], 0) = tk;
        *cluster.map_shared_rank(&rc[rank], 0) = cand;
        *cluster.map_shared_rank(&re[rank], 0) = e2;
      }
    }
    cluster.sync();  // the ranks' bests are in rank 0; every slot is clear again
    if (rank == 0 && threadIdx.x == 0) {
      double bg = -NIDO_MAX_FLOAT, be = 0.;
      unsigned long long bt = kNoKey;
      int bc = -1;
      for (int r = 0; r < kCtas; ++r) {
        be += re[r];
        if (better(rg[r], rtk[r], bg, bt)) { bg = rg[r]; bt = rtk[r]; bc = rc[r]; }
      }
      decide(p, m, v, own, ki, aown, be, bg, (unsigned)bc);
    }
  }
}

__global__ void k_hub_degrees(const int32_t* __restrict__ list, int64_t n, const int64_t* __restrict__ off,
                              int64_t* __restrict__ out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int v = list[i];
    out[2 * i] = v;
    out[2 * i + 1] = off[v + 1] - off[v];
  }
}

inline unsigned grid_cap(int64_t blocks, int64_t cap) {
  if (blocks < 1) blocks = 1;
  return (unsigned)std::min<int64_t>(blocks, cap);
}

template <typename T>
int ensure(nido_graph_s* g, T** p, int64_t* cap, int64_t n) {
  if (n <= *cap) return NIDO_OK;
  raw_free(g->ctx, *p);
  *p = nullptr;
  *cap = 0;
  const int64_t m = std::max<int64_t>(n, 1024);
  NIDO_CUDA_TRY(raw_alloc(g->ctx, (void**)p, sizeof(T) * (size_t)m));
  *cap = m;
  return NIDO_OK;
}

}  // namespace

// Per-phase plan of the hub tier: table offsets, segment items per batch.
int plan_hubs(nido_graph_s* g) {
  const int nb = g->nbatches;
  const int64_t h0 = g->tier_off[(size_t)kTierHub * nb], h1 = g->tier_off[(size_t)(kTierHub + 1) * nb];
  const int64_t nh = h1 - h0;
  g->hub_waves.clear();
  g->hub_wave_off.assign(nb + 1, 0);
  g->nhubs = nh;
  g->hub_nitems = 0;
  g->hub_cl_ok = false;
  g->hub_cl_off.assign((size_t)nb * kClusterBins + 1, 0);
  if (nh == 0) return NIDO_OK;
  cudaStream_t s = g->ctx->stream;
  Arena ar(g->scratch, g->scratch_bytes);
  int64_t* vd = ar.take<int64_t>(2 * nh);
  if (!vd) return nido_set_error(NIDO_E_NOMEM, "scratch arena too small (hubs)");
  k_hub_degrees<<<grid_cap((nh + 255) / 256, kSMs * 4), 256, 0, s>>>(g->perm + h0, nh, g->off, vd);
  NIDO_LAUNCH_CHECK();
  std::vector<int64_t> h(2 * nh);
  NIDO_CUDA_TRY(cudaMemcpyAsync(h.data(), vd, sizeof(int64_t) * 2 * nh, cudaMemcpyDeviceToHost, s));
  NIDO_CUDA_TRY(cudaStreamSynchronize(s));
  std::vector<int32_t> hv(nh), hcap(nh), hseg(nh);
  std::vector<int64_t> htoff(nh);
  std::vector<int2> items;
  for (int64_t i = 0; i < nh; ++i) {
    const int64_t d = h[2 * i + 1];
    const int64_t u = std::min<int64_t>(d, g->nv);
    int64_t cap = 64;
    while (cap < 2 * u) cap <<= 1;
    hv[i] = (int32_t)h[2 * i];
    hcap[i] = (int32_t)cap;
    hseg[i] = (int32_t)((d + kHubSeg - 1) / kHubSeg);
  }
  // Hubs are listed by batch within the tier.  Each batch's hubs are cut into
  // waves whose tables together hold at most cfg.hub_wave_slots slots (so they stay
  // in L2); table offsets are relative to the wave, and every wave reuses the
  // same region because its slice scan clears the tables.  Items and table
  // slices of a hub follow one another.
  std::vector<int2> slices;
  std::vector<int64_t> sfirst(nh + 1, 0);
  std::vector<int64_t> ifirst(nh + 1, 0);
  g->hub_waves.clear();
  g->hub_wave_off.assign(nb + 1, 0);
  int64_t maxslots = 0;
  for (int b = 0; b < nb; ++b) {
    const int64_t a0 = g->tier_off[(size_t)kTierHub * nb + b] - h0;
    const int64_t a1 = g->tier_off[(size_t)kTierHub * nb + b + 1] - h0;
    int64_t wslots = 0;
    for (int64_t i = a0; i < a1; ++i) {
      if (i == a0 || wslots + hcap[i] > g->cfg.hub_wave_slots) {
        g->hub_waves.push_back({(int64_t)items.size(), 0, (int64_t)slices.size(), 0, i, 0});
        wslots = 0;
      }
      htoff[i] = wslots;
      wslots += hcap[i];
      maxslots = std::max(maxslots, wslots);
      ifirst[i] = (int64_t)items.size();
      for (int sgi = 0; sgi < hseg[i]; ++sgi) items.push_back(make_int2((int)i, sgi));
      sfirst[i] = (int64_t)slices.size();
      for (int sl = 0; sl * kHubSlice < hcap[i]; ++sl) slices.push_back(make_int2((int)i, sl));
      sfirst[i + 1] = (int64_t)slices.size();
      nido_graph_s::HubWave& w = g->hub_waves.back();
      w.i1 = (int64_t)items.size();
      w.s1 = (int64_t)slices.size();
      w.h1 = i + 1;
    }
    g->hub_wave_off[b + 1] = (int64_t)g->hub_waves.size();
  }
  ifirst[nh] = (int64_t)items.size();
  g->hub_nitems = (int64_t)items.size();
  const int64_t toff = maxslots;
  g->gslab_need = toff;
  NIDO_TRY(ensure(g, &g->hub_v, &g->hub_cap_hubs_v, nh));
  NIDO_TRY(ensure(g, &g->hub_capv, &g->hub_cap_hubs_c, nh));
  NIDO_TRY(ensure(g, &g->hub_nseg, &g->hub_cap_hubs_s, nh));
  NIDO_TRY(ensure(g, &g->hub_toff, &g->hub_cap_hubs_t, nh));
  NIDO_TRY(ensure(g, &g->hub_done, &g->hub_cap_hubs_d, nh));
  NIDO_TRY(ensure(g, &g->hub_items, &g->hub_cap_items, (int64_t)items.size()));
  NIDO_TRY(ensure(g, &g->hub_slices, &g->hub_cap_slices, (int64_t)slices.size()));
  NIDO_TRY(ensure(g, &g->hub_slice_first, &g->hub_cap_first, nh + 1));
  NIDO_TRY(ensure(g, &g->hub_res, &g->hub_cap_res, (int64_t)(slices.size() * sizeof(SliceResult))));
  NIDO_TRY(ensure(g, &g->hub_item_first, &g->hub_cap_ifirst, nh + 1));
  NIDO_TRY(ensure(g, &g->hub_part, &g->hub_cap_part, (int64_t)items.size()));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_item_first, ifirst.data(), sizeof(int64_t) * (nh + 1), cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_slices, slices.data(), sizeof(int2) * slices.size(), cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_slice_first, sfirst.data(), sizeof(int64_t) * (nh + 1), cudaMemcpyHostToDevice, s));
  // FP64 tables, or packed ones in integer-weight phases; both are kept empty
  // between waves by the kernels that evaluate them
  if (!g->int_weights && toff > g->gslab) {
    raw_free(g->ctx, g->gkeys);
    raw_free(g->ctx, g->gvals);
    g->gkeys = nullptr;
    g->gvals = nullptr;
    g->gslab = 0;
    NIDO_CUDA_TRY(raw_alloc(g->ctx, (void**)&g->gkeys, sizeof(int32_t) * (size_t)toff));
    NIDO_CUDA_TRY(raw_alloc(g->ctx, (void**)&g->gvals, sizeof(double) * (size_t)toff));
    NIDO_CUDA_TRY(cudaMemsetAsync(g->gkeys, 0xff, sizeof(int32_t) * (size_t)toff, s));
    NIDO_CUDA_TRY(cudaMemsetAsync(g->gvals, 0, sizeof(double) * (size_t)toff, s));
    g->gslab = toff;
  }
  if (g->int_weights && toff > g->gslab_packed) {
    raw_free(g->ctx, g->gpacked);
    g->gpacked = nullptr;
    g->gslab_packed = 0;
    NIDO_CUDA_TRY(raw_alloc(g->ctx, (void**)&g->gpacked, sizeof(unsigned long long) * (size_t)toff));
    k_fill_u64<<<grid_cap((toff + 255) / 256, kSMs * 8), 256, 0, s>>>(g->gpacked, toff, kEmptySlot);
    NIDO_LAUNCH_CHECK();
    g->gslab_packed = toff;
  }
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_v, hv.data(), sizeof(int32_t) * nh, cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_capv, hcap.data(), sizeof(int32_t) * nh, cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_nseg, hseg.data(), sizeof(int32_t) * nh, cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_toff, htoff.data(), sizeof(int64_t) * nh, cudaMemcpyHostToDevice, s));
  NIDO_CUDA_TRY(cudaMemsetAsync(g->hub_done, 0, sizeof(int32_t) * nh, s));
  NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_items, items.data(), sizeof(int2) * items.size(), cudaMemcpyHostToDevice, s));
  // cluster bins of every batch's hubs (the tier is used when all fit)
  std::vector<int32_t> clv;
  clv.reserve((size_t)nh);
  bool cl_ok = g->cfg.hub_clusters;
  for (int b = 0; b < nb && cl_ok; ++b) {
    const int64_t a0 = g->tier_off[(size_t)kTierHub * nb + b] - h0;
    const int64_t a1 = g->tier_off[(size_t)kTierHub * nb + b + 1] - h0;
    for (int bin = 0; bin < kClusterBins; ++bin) {
      g->hub_cl_off[(size_t)b * kClusterBins + bin] = (int64_t)clv.size();
      for (int64_t i = a0; i < a1; ++i)
        if (cluster_bin(h[2 * i + 1]) == bin) clv.push_back(hv[i]);
    }
    for (int64_t i = a0; i < a1; ++i)
      if (cluster_bin(h[2 * i + 1]) < 0 || !cluster_launchable(cluster_bin(h[2 * i + 1]))) cl_ok = false;
  }
  g->hub_cl_off[(size_t)nb * kClusterBins] = (int64_t)clv.size();
  if (cl_ok && !clv.empty()) {
    NIDO_TRY(ensure(g, &g->hub_cl_v, &g->hub_cap_cl, (int64_t)clv.size()));
    NIDO_CUDA_TRY(cudaMemcpyAsync(g->hub_cl_v, clv.data(), sizeof(int32_t) * clv.size(), cudaMemcpyHostToDevice, s));
    g->hub_cl_ok = true;
  }
  NIDO_CUDA_TRY(cudaStreamSynchronize(s));  // the host vectors go out of scope
  return NIDO_OK;
}


namespace {
// CTAs of the hub kernels resident on the GPU at once, and of every tier
// kernel (filled by TierKernels::init)
struct HubResident {
  int64_t mv = kSMs, ins = kSMs, sl = kSMs;
};
HubResident g_hub_resident[2][2];   // [many graphs][integer tables]
TierResident g_resident[2][2][2];   // [many graphs][integer tables][reference tie rule]

template <bool kMulti, bool kInts>
int init_mode() {
  int dev = 0, sms = kSMs;
  NIDO_CUDA_TRY(cudaGetDevice(&dev));
  NIDO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  static std::mutex mu;  // contexts may be created from several threads
  std::lock_guard<std::mutex> lk(mu);
  TierResident(&R)[2] = g_resident[kMulti ? 1 : 0][kInts ? 1 : 0];
  NIDO_TRY((TierKernels<kMulti, kInts, false>::init(sms, &R[0])));
  NIDO_TRY((TierKernels<kMulti, kInts, true>::init(sms, &R[1])));
  HubResident& H = g_hub_resident[kMulti ? 1 : 0][kInts ? 1 : 0];
  H.mv = resident_ctas(k_move_hub<kMulti, kInts>, kHubThreads, 0, sms);
  H.ins = resident_ctas(k_hub_insert<kInts>, kHubThreads, 0, sms);
  H.sl = resident_ctas(k_hub_slices<kMulti, kInts>, kHubThreads, 0, sms);
  return NIDO_OK;
}

int64_t g_cluster_max[kClusterBins] = {0, 0, 0, 0};  // clusters resident on the GPU at once

template <int kCtas>
cudaLaunchConfig_t cluster_config(int64_t clusters, cudaStream_t s, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(clusters * kCtas), 1, 1);
  cfg.blockDim = dim3(kClThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)kClSlots * 12;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// shared memory and cluster-size attributes of one cluster kernel, and how
// many of its clusters fit on the GPU (0: none, the bin stays off)
template <int kCtas, bool kMulti>
int64_t cluster_setup() {
  auto k = k_move_cluster<kCtas, kMulti>;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSlots * 12) != cudaSuccess ||
      (kCtas > 8 && cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = cluster_config<kCtas>(1, nullptr, attr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int cluster_init() {
  const int64_t m[kClusterBins] = {std::min(cluster_setup<2, false>(), cluster_setup<2, true>()),
                                   std::min(cluster_setup<4, false>(), cluster_setup<4, true>()),
                                   std::min(cluster_setup<8, false>(), cluster_setup<8, true>()),
                                   std::min(cluster_setup<16, false>(), cluster_setup<16, true>())};
  for (int b = 0; b < kClusterBins; ++b) {
    g_cluster_max[b] = m[b];
    g_cluster_ok[b] = m[b] > 0;
  }
  return NIDO_OK;
}

template <int kCtas, bool kMulti>
int launch_cluster_bin(int bin, const int32_t* list, int64_t n, const MoveArgs& p, cudaStream_t s) {
  cudaLaunchAttribute attr[1];
  cudaLaunchConfig_t cfg = cluster_config<kCtas>(std::min<int64_t>(n, g_cluster_max[bin]), s, attr);
  NIDO_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_move_cluster<kCtas, kMulti>, list, n, p));
  return NIDO_OK;
}

// the hubs of one batch on clusters of 2, 4, 8 and 16 CTAs by degree
template <bool kMulti>
int launch_clusters(nido_graph_s* g, int batch, const MoveArgs& p, cudaStream_t s) {
  for (int bin = 0; bin < kClusterBins; ++bin) {
    const int64_t c0 = g->hub_cl_off[(size_t)batch * kClusterBins + bin];
    const int64_t c1 = g->hub_cl_off[(size_t)batch * kClusterBins + bin + 1];
    if (c1 <= c0) continue;
    const int32_t* list = g->hub_cl_v + c0;
    switch (bin) {
      case 0: NIDO_TRY((launch_cluster_bin<2, kMulti>(bin, list, c1 - c0, p, s))); break;
      case 1: NIDO_TRY((launch_cluster_bin<4, kMulti>(bin, list, c1 - c0, p, s))); break;
      case 2: NIDO_TRY((launch_cluster_bin<8, kMulti>(bin, list, c1 - c0, p, s))); break;
      default: NIDO_TRY((launch_cluster_bin<16, kMulti>(bin, list, c1 - c0, p, s))); break;
    }
  }
  return NIDO_OK;
}

// the tier kernels of one batch; kMulti: many graphs (per-vertex mass).  The
// tiers cover disjoint vertices and only read comm and a, so they run on
// three streams: the hub chain and the CTA tiers on the context's side
// streams, the rest on its stream, joined before the function returns.
template <bool kMulti, bool kInts>
int launch_tiers(nido_graph_s* g, int batch, int tie, const MoveArgs& p) {
  nido_ctx_s* ctx = g->ctx;
  const bool nido_tie = tie == NIDO_TIE_NIDO;
  const TierResident& R = g_resident[kMulti ? 1 : 0][kInts ? 1 : 0][nido_tie ? 1 : 0];
  const HubResident& H = g_hub_resident[kMulti ? 1 : 0][kInts ? 1 : 0];
  const cudaStream_t main_s = ctx->stream;
  NIDO_CUDA_TRY(cudaEventRecord(ctx->fork_ev, main_s));
  for (int i = 0; i < 2; ++i) NIDO_CUDA_TRY(cudaStreamWaitEvent(ctx->aux[i], ctx->fork_ev, 0));
  const int nb = g->nbatches;
  // edges staged in shared memory by bulk copies from this GPU's memory (a
  // tier option; never for edges kept in mapped host memory)
  const bool staged = g->cfg.staged_edges && !g->host_edges;
  for (int t = kNumTiers - 1; t >= 0; --t) {  // longest chains first
    const cudaStream_t s = t == kTierHub ? ctx->aux[0] : (t >= kTierCtaS ? ctx->aux[1] : main_s);
    const int64_t b0 = g->tier_off[(size_t)t * nb + batch], b1 = g->tier_off[(size_t)t * nb + batch + 1];
    const int64_t n = b1 - b0;
    if (n <= 0) continue;
    const int32_t* list = g->perm + b0;
    if (t != kTierHub) {
      if (nido_tie) NIDO_TRY((TierKernels<kMulti, kInts, true>::launch(R, t, list, n, p, staged, s)));
      else NIDO_TRY((TierKernels<kMulti, kInts, false>::launch(R, t, list, n, p, staged, s)));
      continue;
    }
        if constexpr (kInts) {
          // integer-weight phases with the smallest-id rule: hubs on
          // thread-block clusters when every hub of the phase fits one
          if (tie != NIDO_TIE_NIDO && g->cfg.hub_clusters && g->hub_cl_ok) {
            NIDO_TRY(launch_clusters<kMulti>(g, batch, p, s));
            continue;
          }
        }
        SliceResult* res = reinterpret_cast<SliceResult*>(g->hub_res);
        HubTable<kInts> tab;
        if constexpr (kInts) tab.slots = g->gpacked;  // integer phases are planned with packed tables
        else tab = HubTable<false>{g->gkeys, g->gvals};
        for (int64_t wv = g->hub_wave_off[batch]; wv < g->hub_wave_off[batch + 1]; ++wv) {
          const nido_graph_s::HubWave& w = g->hub_waves[wv];
          const int2* items = g->hub_items + w.i0;
          if (nido_tie) {
            k_move_hub<kMulti, kInts><<<grid_cap(w.i1 - w.i0, H.mv), kHubThreads, 0, s>>>(
                items, w.i1 - w.i0, g->hub_v, g->hub_toff, g->hub_capv, g->hub_nseg, g->hub_done, tab, p);
            NIDO_LAUNCH_CHECK();
            continue;
          }
          k_hub_insert<kInts><<<grid_cap(w.i1 - w.i0, H.ins), kHubThreads, 0, s>>>(
              items, w.i1 - w.i0, g->hub_v, g->hub_toff, g->hub_capv, tab, p);
          NIDO_LAUNCH_CHECK();
          k_hub_slices<kMulti, kInts><<<grid_cap(w.s1 - w.s0, H.sl), kHubThreads, 0, s>>>(
              g->hub_slices + w.s0, w.s1 - w.s0, g->hub_v, g->hub_toff, g->hub_capv, tab, p, res + w.s0);
          NIDO_LAUNCH_CHECK();
          k_hub_combine<kMulti><<<grid_cap((w.h1 - w.h0 + 7) / 8, kSMs * 4), 256, 0, s>>>(
              w.h1 - w.h0, g->hub_v + w.h0, g->hub_slice_first + w.h0, res, p);
          NIDO_LAUNCH_CHECK();
        }
  }
  for (int i = 0; i < 2; ++i) {
    NIDO_CUDA_TRY(cudaEventRecord(ctx->join_ev[i], ctx->aux[i]));
    NIDO_CUDA_TRY(cudaStreamWaitEvent(main_s, ctx->join_ev[i], 0));
  }
  return NIDO_OK;
}
}  // namespace

// attributes of the kernels of one graph (contexts) or many (batches)
int move_init_attributes(bool many) {
  if (many) {
    NIDO_TRY((init_mode<true, false>()));
    return init_mode<true, true>();
  }
  NIDO_TRY(cluster_init());
  NIDO_TRY((init_mode<false, false>()));
  return init_mode<false, true>();
}

MoveArgs move_args(nido_graph_s* g) {
  double zh = 0., zl = 0.;
  if (!g->gid && g->int_weights) mass_reciprocal(g->m, &zh, &zl);
  return MoveArgs{g->off, g->adj, g->w, g->k, g->comm, g->a, g->newc, g->m,
                  reinterpret_cast<unsigned long long*>(g->dcount + 1), g->gid, g->mg, zh, zl,
                  g->int_weights ? g->zg : nullptr,
                  g->int_weights ? 1 : 0, g->nv};
}

namespace {
int tiers_direct(nido_graph_s* g, int batch, int tie, const MoveArgs& p) {
  if (g->gid) return p.ints ? launch_tiers<true, true>(g, batch, tie, p) : launch_tiers<true, false>(g, batch, tie, p);
  return p.ints ? launch_tiers<false, true>(g, batch, tie, p) : launch_tiers<false, false>(g, batch, tie, p);
}
}  // namespace

// The tier kernels of one batch, enqueued directly (no events, no per-batch
// graph): what the device-resident loop captures.  The plan (tier lists, hub
// plan) must be valid.
int launch_move_tiers(nido_graph_s* g, int batch, int tie) {
  if (batch < 0 || batch >= g->nbatches)
    return nido_set_error(NIDO_E_INVALID, "louvain_update: batch %d out of range [0,%d)", batch, g->nbatches);
  return tiers_direct(g, batch, tie, move_args(g));
}

int check_bounded_wait(nido_ctx_s* ctx, int32_t* gave_up, int32_t* waited_ms) {
  int32_t* d = nullptr;
  NIDO_CUDA_TRY(cudaMalloc((void**)&d, 2 * sizeof(int32_t)));
  int32_t h[2] = {0, 0};
  k_check_bounded_wait<<<1, 32, 0, ctx->stream>>>(d);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  cudaFree(d);
  if (e != cudaSuccess) return nido_set_error(NIDO_E_CUDA, "bounded-wait check: %s", cudaGetErrorString(e));
  nido_count_launches(1);
  if (gave_up) *gave_up = h[0];
  if (waited_ms) *waited_ms = h[1];
  return NIDO_OK;
}

int launch_move(nido_graph_s* g, int batch, int tie, cudaEvent_t ev_start, cudaEvent_t ev_end) {
  if (batch < 0 || batch >= g->nbatches)
    return nido_set_error(NIDO_E_INVALID, "louvain_update: batch %d out of range [0,%d)", batch, g->nbatches);
  if (!g->bins_valid) NIDO_TRY(build_batches(g));
  cudaStream_t s = g->ctx->stream;
  const MoveArgs p = move_args(g);
  if (ev_start) NIDO_CUDA_TRY(cudaEventRecord(ev_start, s));
  auto direct = [&]() { return tiers_direct(g, batch, tie, p); };
  if (!g->use_graphs) {
    NIDO_TRY(direct());
  } else {
    // The launches of a batch are fixed for a phase: the first sweep runs them
    // directly, the second captures them into a CUDA graph, later sweeps
    // replay it (the arguments are all device pointers that live for the
    // phase).
    if (g->move_graphs.size() < (size_t)g->nbatches) g->move_graphs.resize(g->nbatches);
    nido_graph_s::MoveGraph& mg = g->move_graphs[batch];
    if (mg.epoch != g->plan_epoch || mg.tie != tie) {
      if (mg.exec) cudaGraphExecDestroy(mg.exec);
      mg = nido_graph_s::MoveGraph();
      mg.epoch = g->plan_epoch;
      mg.tie = tie;
    }
    if (mg.exec) {
      NIDO_CUDA_TRY(cudaGraphLaunch(mg.exec, s));
      nido_count_launches(mg.kernels);
    } else if (mg.uses++ == 0) {
      NIDO_TRY(direct());
    } else {
      const uint64_t l0 = nido_launch_count();
      cudaGraph_t graph = nullptr;
      NIDO_CUDA_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
      const int st = direct();
      const cudaError_t ce = cudaStreamEndCapture(s, &graph);
      if (st != NIDO_OK) {
        if (graph) cudaGraphDestroy(graph);
        return st;
      }
      if (ce != cudaSuccess) return nido_set_error(NIDO_E_CUDA, "move-sweep capture failed: %s", cudaGetErrorString(ce));
      mg.kernels = nido_launch_count() - l0;
      const cudaError_t ie = cudaGraphInstantiate(&mg.exec, graph, 0);
      cudaGraphDestroy(graph);
      if (ie != cudaSuccess) {
        mg.exec = nullptr;
        return nido_set_error(NIDO_E_CUDA, "move-sweep graph instantiation failed: %s", cudaGetErrorString(ie));
      }
      NIDO_CUDA_TRY(cudaGraphLaunch(mg.exec, s));
    }
  }
  if (ev_end) NIDO_CUDA_TRY(cudaEventRecord(ev_end, s));
  return NIDO_OK;
}

}  // namespace nido
