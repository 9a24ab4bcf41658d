// noalloc.cu -- modularity of a partition from caller-owned device arrays,
// with no memory allocation at all.
//
// Who needs this: code that runs where cudaMalloc is not allowed or not
// wanted -- while a CUDA stream is being captured into a graph, inside a
// custom device-memory allocator or a memory-pool callback, or in a serving
// process that has handed all of the GPU's memory to a fixed pool.  Such
// callers hold their graph and partition in device memory already and only
// need the number back.
//
// Design: the reference's reduction (compute_modularity_reduce_kernel<128,16>
// and reduce_vector_kernel, graph_cuda.cu:2078-2134, 1806-1835) writes one
// partial per 16-thread group into a buffer it cudaMallocs on every call
// (graph_gpu.cpp:872-875).  Here that buffer is a file-scope __device__
// array of the reference's maximum size, 65535 blocks * 128 / 16 = 524,280
// doubles (4 MiB), and the partial sums of vertex tiles whose edges are split
// over several blocks are two more (2 MiB); every GPU that loads this
// library holds them until the process exits.  Every partial that a kernel
// reads is written earlier in the same call, so nothing has to be cleared
// between calls.  All calls on a device share the arrays: calls that overlap
// on the GPU (for example on two streams at once) race and give wrong results.
#include <algorithm>

#include "common.cuh"

namespace {

constexpr int64_t kMaxGroups = 524280;  // 65535 * 128 / 16
constexpr int64_t kNoallocMaxVertices = ((int64_t)1 << 31) - 2;  // the library's vertex limit
// The in-community sums walk the edges in items of at most `chunk` edges of a
// tile of kTileV consecutive vertices.  A hub's edges are thus spread over
// many blocks, where one thread per vertex left the whole call waiting for the
// largest degree and read every row with a stride of its own.
constexpr int kTileV = 64;
constexpr int kTileG = kTileV / 16;      // 16-vertex groups of a tile
constexpr int kItemThreads = 256;
constexpr int kItemUnroll = 8;           // edges in flight per thread
constexpr int64_t kMinChunk = 4096;
constexpr int64_t kMaxChunks = 32768;    // the chunk grows so that the edges hold at most this many
constexpr int64_t kPassV = (int64_t)65535 * 128;  // vertices of one pass: one per thread slot

__device__ __align__(256) double g_group_partials[kMaxGroups];
// sums of the chunks of split tiles: chunk c of a tile starting in chunk f of
// the pass's edges is entry f + c, the tile's last chunk in g_split_last (the
// next tile may start in the same chunk)
__device__ double g_split[(kMaxChunks + 1) * kTileG];
__device__ double g_split_last[(kMaxChunks + 1) * kTileG];

__device__ __forceinline__ int64_t chunk_edges(int64_t e) {
  const int64_t c = (e + kMaxChunks - 1) / kMaxChunks;
  return c > kMinChunk ? c : kMinChunk;
}

// In-community weight of the 16-vertex groups of the vertices [vb, ve) (one
// pass).  Tile i of the pass starts at edge o_i of the pass and holds the
// items i + o_i / chunk up to the next tile's first: at least one, and enough
// for its edges.  A block finds the tile of an item by a search with a fan-out
// of its threads (two or three rounds), holds the tile's row offsets and
// communities in shared memory and takes the item's edges coalesced, eight
// in flight per thread; an edge finds its row by six shared-memory steps.
// Sums are added in a fixed order (threads, lanes, warps, chunks), so equal
// inputs give equal bits; integer weights are exact in any order.
// Bound: the streamed ids (8 bytes an edge) and the gathers of comm.  On
// R-MAT of 2^20 vertices and 31.4 M edges a call takes 0.35 ms (a thread per
// vertex: 10.6 ms, the longest row).
__global__ void __launch_bounds__(kItemThreads) k_noalloc_items(int64_t vb, int64_t ve, const int64_t* __restrict__ off,
                                                                const int64_t* __restrict__ adj,
                                                                const double* __restrict__ w,
                                                                const int64_t* __restrict__ comm, bool add) {
  __shared__ int rel[kTileV + 1];          // row starts relative to the item's first edge, clamped to the item
  __shared__ int64_t own[kTileV];
  __shared__ double red[kItemThreads / 32][kTileG];
  const int64_t nt = (ve - vb + kTileV - 1) / kTileV;
  const int64_t e0 = off[vb], ne = off[ve] - e0;
  const int64_t chunk = chunk_edges(ne);
  const int64_t items = nt + ne / chunk;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto first_item = [&](int64_t i) { return i + (off[min(vb + i * kTileV, ve)] - e0) / chunk; };
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    int64_t lo = 0, hi = nt;               // first_item(lo) <= it < first_item(hi)
    while (hi - lo > 1) {
      const int64_t step = (hi - lo + kItemThreads - 1) / kItemThreads;
      const int64_t i = lo + threadIdx.x * step;
      const int n = __syncthreads_count(i < hi && first_item(i) <= it);
      lo += (int64_t)(n - 1) * step;
      hi = min(lo + step, hi);
    }
    const int64_t v0 = vb + lo * kTileV, v1 = min(v0 + kTileV, ve);
    const int64_t o0 = off[v0], o1 = off[v1];
    const int64_t f0 = (o0 - e0) / chunk, f1 = (o1 - e0) / chunk;
    const int64_t c = it - (lo + f0);
    const int64_t eb = o0 + c * chunk;
    const int len = (int)max((int64_t)0, min(chunk, o1 - eb));
    if (threadIdx.x <= kTileV)
      rel[threadIdx.x] = (int)min(max(off[min(v0 + threadIdx.x, v1)] - eb, (int64_t)0), (int64_t)len);
    if (threadIdx.x < kTileV) own[threadIdx.x] = v0 + threadIdx.x < v1 ? comm[v0 + threadIdx.x] : -1;
    __syncthreads();
    double s[kTileG] = {};
    for (int b = 0; b < len; b += kItemUnroll * kItemThreads) {
      int64_t u[kItemUnroll];
#pragma unroll
      for (int k = 0; k < kItemUnroll; ++k) {
        const int j = b + k * kItemThreads + threadIdx.x;
        u[k] = j < len ? adj[eb + j] : -1;
      }
#pragma unroll
      for (int k = 0; k < kItemUnroll; ++k) u[k] = u[k] >= 0 ? comm[u[k]] : -1;
#pragma unroll
      for (int k = 0; k < kItemUnroll; ++k) {
        const int j = b + k * kItemThreads + threadIdx.x;
        if (j >= len) continue;
        int r = 0;                         // last row starting at or before j
#pragma unroll
        for (int d = kTileV / 2; d >= 1; d >>= 1)
          if (rel[r + d] <= j) r += d;
        if (u[k] == own[r]) {
          const double x = w[eb + j];
#pragma unroll
          for (int q = 0; q < kTileG; ++q)
            if (q == r >> 4) s[q] += x;
        }
      }
    }
#pragma unroll
    for (int q = 0; q < kTileG; ++q) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_down_sync(NIDO_FULL_MASK, s[q], o);
      if (lane == 0) red[wid][q] = s[q];
    }
    __syncthreads();
    if (threadIdx.x < kTileG) {
      double x = 0.;
      for (int i = 0; i < kItemThreads / 32; ++i) x += red[i][threadIdx.x];
      const int64_t g = lo * kTileG + threadIdx.x;
      if (f0 == f1) {                      // the whole tile is this item
        if (v0 + 16 * threadIdx.x < v1) g_group_partials[g] = add ? g_group_partials[g] + x : x;
      } else if (c == f1 - f0) {
        g_split_last[f1 * kTileG + threadIdx.x] = x;
      } else {
        g_split[(f0 + c) * kTileG + threadIdx.x] = x;
      }
    }
    __syncthreads();                       // rel, own and red are read
  }
}

// Groups of split tiles: their chunks added in order.  After the last pass
// the group's sum becomes its part of Q: thread slot t folds
// ac = fma(a_v, a_v, ac) over the vertices t, t+S, ..., 16-lane shuffle trees
// add the slots, and lane 0 writes self/(2m) - ac/(4m*m).
__global__ void k_noalloc_groups(int64_t vb, int64_t ve, bool add, bool last, int64_t nv, int64_t S, int64_t ngroups,
                                 const int64_t* __restrict__ off, const double* __restrict__ a, double m) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t g = t >> 4;
  double s = 0., ac = 0.;
  if (g < ngroups && (t & 15) == 0) {
    s = g_group_partials[g];
    const int64_t v0 = vb + (g / kTileG) * kTileV, q = g % kTileG;
    if (v0 + 16 * q < ve) {
      const int64_t e0 = off[vb], chunk = chunk_edges(off[ve] - e0);
      const int64_t f0 = (off[v0] - e0) / chunk, f1 = (off[min(v0 + kTileV, ve)] - e0) / chunk;
      if (f0 != f1) {
        double x = 0.;
        for (int64_t f = f0; f < f1; ++f) x += g_split[f * kTileG + q];
        x += g_split_last[f1 * kTileG + q];
        s = add ? s + x : x;
        if (!last) g_group_partials[g] = s;
      }
    }
  }
  if (!last) return;
  if (g < ngroups)
    for (int64_t v = t; v < nv; v += S) ac = fma(a[v], a[v], ac);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) ac += __shfl_down_sync(NIDO_FULL_MASK, ac, o, 16);
  if ((t & 15) == 0 && g < ngroups) {
    double x = __ddiv_rn(s, __dmul_rn(2., m));
    x = __dsub_rn(x, __ddiv_rn(ac, __dmul_rn(__dmul_rn(4., m), m)));
    g_group_partials[g] = __dadd_rn(0., x);
  }
}

// One block of 1024 threads: strided fold (sixteen loads in flight, added in
// order), then warp trees.
__global__ void __launch_bounds__(1024) k_noalloc_reduce(int64_t n, double* __restrict__ q) {
  __shared__ double ws[32];
  double s = 0.;
  for (int64_t b = threadIdx.x; b < n; b += 16 * 1024) {
    double x[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) x[k] = b + k * 1024 < n ? g_group_partials[b + k * 1024] : 0.;
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (b + k * 1024 < n) s += x[k];
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(NIDO_FULL_MASK, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = ws[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(NIDO_FULL_MASK, s, o);
    if (threadIdx.x == 0) *q = s;
  }
}

}  // namespace

extern "C" int nido_modularity_noalloc(void* stream, int64_t nv, const int64_t* d_off, const int64_t* d_adj,
                                       const double* d_w, const int64_t* d_comm, const double* d_a, double m,
                                       double* d_q) {
  // every array the kernels may read must be given once there are vertices;
  // a caller whose graph has no edges passes any non-null d_adj and d_w
  if (nv < 0 || !d_q || (nv > 0 && (!d_off || !d_adj || !d_w || !d_comm || !d_a)))
    return nido_set_error(NIDO_E_INVALID, "nido_modularity_noalloc: bad arguments");
  if (nv > kNoallocMaxVertices)
    return nido_set_error(NIDO_E_TOO_LARGE, "nido_modularity_noalloc: %lld vertices exceed the limit of %lld",
                          (long long)nv, (long long)kNoallocMaxVertices);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t grid = (nv + 7) / 8;
  if (grid > 65535) grid = 65535;
  if (grid < 1) grid = 1;
  const int64_t S = 128 * grid;
  const int64_t nslots = nv < S ? nv : S;
  const int64_t ngroups = (nslots + 15) / 16;  // <= kMaxGroups for every nv
  if (ngroups > kMaxGroups) return nido_set_error(NIDO_E_TOO_LARGE, "too many groups");
  // a pass covers at most one vertex per thread slot (all of them below 8.4 M vertices)
  for (int64_t vb = 0; vb < nv; vb += kPassV) {
    const int64_t ve = std::min<int64_t>(nv, vb + kPassV);
    const int64_t tiles = (ve - vb + kTileV - 1) / kTileV;
    // hubs make more items than tiles: small graphs get some more blocks than tiles
    k_noalloc_items<<<(unsigned)std::min<int64_t>(2 * tiles, nido::kSMs * 8), kItemThreads, 0, s>>>(
        vb, ve, d_off, d_adj, d_w, d_comm, vb > 0);
    NIDO_LAUNCH_CHECK();
    k_noalloc_groups<<<(unsigned)((ngroups * 16 + 255) / 256), 256, 0, s>>>(vb, ve, vb > 0, ve == nv, nv, S, ngroups,
                                                                           d_off, d_a, m);
    NIDO_LAUNCH_CHECK();
  }
  k_noalloc_reduce<<<1, 1024, 0, s>>>(ngroups, d_q);
  NIDO_LAUNCH_CHECK();
  return NIDO_OK;
}
