// phase_core.cuh -- device code of the commit and the modularity shared by the
// per-stage kernels (phase.cu) and the persistent phase loop (phase_loop.cuh).
// comm and a change while the phase loop runs, so no pointer to them is
// __restrict__ here.
#ifndef NIDO_PHASE_CORE_CUH_
#define NIDO_PHASE_CORE_CUH_
#include "common.cuh"

namespace nido {

// Movers subtract k_v from the old community and add it to the new one.  Movers
// of a warp with the same old (new) community add their k_v first (in lane
// order) and issue one atomic per community, which takes the contention off
// communities many vertices join.
__device__ __forceinline__ void warp_community_add(double* a, int c, double x, bool on) {
  const int lane = threadIdx.x & 31;
  const unsigned peers = __match_any_sync(NIDO_FULL_MASK, on ? c : -1);
  double s = 0.;
  unsigned rem = on ? peers : 0u;
  const int maxcnt = __reduce_max_sync(NIDO_FULL_MASK, (unsigned)__popc(rem));
  for (int it = 0; it < maxcnt; ++it) {
    const int src = rem ? __ffs(rem) - 1 : lane;
    const double y = __shfl_sync(NIDO_FULL_MASK, x, src);
    if (rem) { s += y; rem &= rem - 1; }
  }
  if (on && lane == __ffs(peers) - 1) atomicAdd(&a[c], s);
}

// Vertex v (in: this lane has one) moves from comm[v] to newc[v]; the ids are
// swapped, so that newc keeps the old one.  Warp-uniform.
__device__ __forceinline__ void commit_vertex(int64_t v, bool in, const double* k, int32_t* comm, int32_t* newc,
                                              double* a) {
  int32_t src = 0, dst = 0;
  double kv = 0.;
  if (in) {
    src = comm[v];
    dst = newc[v];
  }
  const bool mv = in && src != dst;
  if (mv) kv = k[v];
  if (__any_sync(NIDO_FULL_MASK, mv)) {
    warp_community_add(a, src, -kv, mv);
    warp_community_add(a, dst, kv, mv);
  }
  if (mv) {
    comm[v] = dst;
    newc[v] = src;
  }
}

// Sum of w[j] over j = j0, j0+step, ... < e with comm[adj[j]] == own, added in
// that order; four edges' loads (bounds-guarded) are issued before any is
// added, so four dependent gathers are in flight per lane at every degree.
__device__ __forceinline__ double own_weight(const int32_t* __restrict__ adj, const double* __restrict__ w,
                                             const int32_t* comm, int32_t own, int64_t j0,
                                             int64_t e, int step) {
  double x = 0.;
  for (int64_t j = j0; j < e; j += 4 * (int64_t)step) {
    int u[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int64_t jk = j + k * (int64_t)step;
      u[k] = jk < e ? adj[jk] : -1;
    }
    int c[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) c[k] = u[k] >= 0 ? comm[u[k]] : 0;
    // only in-community edges load their weight: a warp's 32-byte weight
    // sectors with no such edge are never fetched (most of them while the
    // communities are small); the sum and its order are unchanged
    bool in[4];
    double wt[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      in[k] = u[k] >= 0 && c[k] == own;
      wt[k] = in[k] ? w[j + k * (int64_t)step] : 0.;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (in[k]) x += wt[k];
  }
  return x;
}

// In-community weight (self-loops included) of the vertices of list[0, n) by
// groups of G lanes: lane l sums edges l, l+G, ... then a fixed tree.  This
// warp takes the sets of 32/G vertices warp, warp + nw, ...
template <int G>
__device__ __forceinline__ void q_self_list(const int32_t* __restrict__ list, int64_t n, int64_t warp, int64_t nw,
                                            const int64_t* __restrict__ off, const int32_t* __restrict__ adj,
                                            const double* __restrict__ w, const int32_t* comm, double* selfv) {
  constexpr int VPW = 32 / G;
  const int lane = threadIdx.x & 31, gl = lane & (G - 1), gid = lane / G;
  for (int64_t b = warp * VPW; b < n; b += nw * VPW) {
    const int64_t idx = b + gid;
    double x = 0.;
    int v = 0;
    if (idx < n) {
      v = list[idx];
      x = own_weight(adj, w, comm, comm[v], off[v] + gl, off[v + 1], G);
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) x += __shfl_down_sync(NIDO_FULL_MASK, x, o, G);
    if (gl == 0 && idx < n) selfv[v] = x;
  }
}

// Sum of the edges j0, j0 + T, ... < e in the community of v over a CTA of T
// threads (a fixed order: threads, lanes, warps); the result in thread 0.  ws:
// T/32 doubles, free again on return.
template <int T>
__device__ __forceinline__ double q_self_block(const int32_t* __restrict__ adj, const double* __restrict__ w,
                                               const int32_t* comm, int32_t own, int64_t e0, int64_t e1, double* ws) {
  double x = own_weight(adj, w, comm, own, e0 + threadIdx.x, e1, T);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(NIDO_FULL_MASK, x, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
  __syncthreads();
  double s = 0.;
  if (threadIdx.x == 0)
    for (int i = 0; i < T / 32; ++i) s += ws[i];
  __syncthreads();
  return s;
}

// A group's part of Q from its in-community weight s and ac = sum of a^2:
// self/(2m) - ac/(4m*m).
__device__ __forceinline__ double q_part(double s, double ac, double m) {
  double x = __ddiv_rn(s, __dmul_rn(2., m));
  x = __dsub_rn(x, __ddiv_rn(ac, __dmul_rn(__dmul_rn(4., m), m)));
  return __dadd_rn(0., x);
}

}  // namespace nido
#endif
