// move_tiers.cuh -- the move kernels of the degree tiers below the hubs.  They
// are instantiated per mode (one graph / many graphs, FP64 / integer tables,
// tie rule) in tiers_*.cu, one file per graph mode and table kind.
#ifndef NIDO_MOVE_TIERS_CUH_
#define NIDO_MOVE_TIERS_CUH_
#include <algorithm>

#include "common.cuh"
#include "engine.cuh"
#include "move_core.cuh"

namespace nido {

// CTAs of every tier kernel that fit on the GPU at once (SMs x resident CTAs
// per SM, from the occupancy calculator): grid-stride kernels launched with
// more would leave a partial wave at the end.
struct TierResident {
  int64_t g4 = kSMs, g8 = kSMs, g16 = kSMs, g32 = kSMs, warp = kSMs, ctas = kSMs, ctam = kSMs, ctal = kSMs,
          ctaxa = kSMs, ctax = kSMs, ctas_st = kSMs, ctam_st = kSMs;
};

template <typename K>
int64_t resident_ctas(K kernel, int threads, size_t smem, int sms) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess) {
    cudaGetLastError();
    per_sm = 1;
  }
  return (int64_t)std::max(per_sm, 1) * sms;
}

template <bool kMulti, bool kInts, bool kTie>
struct TierKernels {
  // shared-memory attributes and resident CTAs of the mode's kernels
  static int init(int sms, TierResident* R);
  // the kernel of tier t (not the hubs) over list[0, n); staged: CTA-S and
  // CTA-M with their edges staged by bulk copies
  static int launch(const TierResident& R, int t, const int32_t* list, int64_t n, const MoveArgs& p, bool staged,
                    cudaStream_t s);
};

// ---- bounded waits on an mbarrier --------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void* ptr) { return (unsigned)__cvta_generic_to_shared(ptr); }

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred P;\n mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n selp.u32 %0, 1, 0, P;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// bounded wait: gives up (false) after kMbarTries attempts or about a second,
// whichever comes first, instead of spinning forever; the caller counts the
// failure in p.err
constexpr int kMbarTries = 1 << 20;
constexpr unsigned long long kMbarWaitNs = 1000000000ull;
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
  const unsigned long long t0 = gtimer_ns();
  for (int i = 0; i < kMbarTries; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255) == 255 && gtimer_ns() - t0 > kMbarWaitNs) return false;
  }
  return false;
}

#ifdef NIDO_TIER_KERNELS
// ---- degree <= 32: lane groups, registers ------------------------------------------
// Six 256-thread blocks an SM (at most 40 registers a thread): the tier waits
// on its gathers, and more resident warps hide more of them.
template <int G, bool kMulti, bool kTie>
__global__ void __launch_bounds__(256, 6) k_move_group(const int32_t* __restrict__ list, int64_t n, MoveArgs p) {
  __shared__ int fold[256];
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  group_list<G, kMulti, kTie>(list, n, warp, nw, p, fold + (threadIdx.x & ~31));
}

// ---- 32 < degree <= 192: one warp per vertex, table in shared memory ----------------
constexpr int kWarpChunks = 6;  // 32-edge chunks of a vertex (degree <= 192)

template <int kCap, bool kMulti, bool kInts, bool kTie>
__global__ void __launch_bounds__(256, 5) k_move_warp(const int32_t* __restrict__ list, int64_t n, MoveArgs p) {
  extern __shared__ __align__(128) double smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  SharedTable<kInts> t;
  t.place(reinterpret_cast<char*>(smem) + wid * table_bytes(kCap, kInts), kCap);
  for (int i = lane; i < kCap; i += 32) t.clear(i);
  __syncwarp();
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  warp_list<kCap, kWarpChunks, kMulti, kInts, kTie>(list, n, warp, nw, p, t);
}

// ---- staged adjacency: 1-D bulk copies (TMA) of a vertex's edge ranges --------
// One thread copies the next vertex's ids and weights from this GPU's global
// memory into shared memory with cp.async.bulk, completed on an mbarrier,
// while the block still evaluates the current vertex; the block then reads
// the edges from shared memory.  Copies start and end on 16-byte boundaries:
// the id range is widened to multiples of 4 ids and the weight range to
// multiples of 2 weights (the edge arrays carry 4 spare entries so the widened
// end stays inside them).  No multicast.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// shared memory of one staged vertex of degree <= kDeg: ids then weights
template <int kDeg>
struct Stage {
  static constexpr int kIds = kDeg + 8;     // widened by up to 3 ids each side
  static constexpr int kWts = kDeg + 4;     // widened by up to 1 weight each side
  static constexpr size_t kBytes = (size_t)kIds * 4 + (size_t)kWts * 8;
};

// Thread 0: copy the edges [s, e) into the stage (ids at sadj, weights at
// sw) on bar; *a0 / *w0 receive the first id / weight index held.
__device__ __forceinline__ void stage_edges(const MoveArgs& p, int64_t s, int64_t e, int32_t* sadj, double* sw,
                                            unsigned long long* bar, int64_t* a0, int64_t* w0) {
  const int64_t ia = s & ~(int64_t)3, ib = (e + 3) & ~(int64_t)3;
  const int64_t wa = s & ~(int64_t)1, wb = (e + 1) & ~(int64_t)1;
  const unsigned bi = (unsigned)(4 * (ib - ia)), bw = (unsigned)(8 * (wb - wa));
  *a0 = ia;
  *w0 = wa;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // earlier reads of the stage come first
  mbar_arrive_expect_tx(bar, bi + bw);
  if (bi) bulk_g2s(sadj, p.adj + ia, bi, bar);
  if (bw) bulk_g2s(sw, p.w + wa, bw, bar);
}

// ---- 192 < degree <= 12288: one CTA per vertex, table in shared memory --------------
// kChunks edges of a vertex per thread at most.  kStageDeg > 0: the tier's
// vertices (degree <= kStageDeg) have their edges staged in shared memory
// behind the table (see stage_edges), one vertex ahead: the copy of vertex i+1
// runs while vertex i is evaluated.
// Resident CTAs an SM: ten of 128 threads or five of 256 (at most 48 registers
// a thread), else the 64-register fill of 1024 threads.
template <int kThreads, int kCap, int kChunks, bool kMulti, bool kInts, bool kTie, int kStageDeg = 0>
__global__ void __launch_bounds__(kThreads, kThreads == 128 ? 10 : (kThreads == 256 && kChunks == 6 ? 5 : 1024 / kThreads))
    k_move_cta(const int32_t* __restrict__ list, int64_t n, MoveArgs p) {
  constexpr bool kStaged = kStageDeg > 0;
  extern __shared__ __align__(128) double smem[];
  __shared__ CtaShared sh;
  __shared__ unsigned long long stage_bar;
  __shared__ long long stage_off[2];  // first id and weight index held by the stage
  int32_t* sadj = nullptr;
  double* sw = nullptr;
  if constexpr (kStaged) {
    char* st = reinterpret_cast<char*>(smem) + table_bytes(kCap, kInts);
    sadj = reinterpret_cast<int32_t*>(st);
    sw = reinterpret_cast<double*>(st + (size_t)Stage<kStageDeg>::kIds * 4);
    if (threadIdx.x == 0) {
      mbar_init(&stage_bar, 1);
      if (blockIdx.x < n) {  // the first vertex's edges start on their way at once
        const int v0 = list[blockIdx.x];
        int64_t a0, w0;
        stage_edges(p, p.off[v0], p.off[v0 + 1], sadj, sw, &stage_bar, &a0, &w0);
        stage_off[0] = a0;
        stage_off[1] = w0;
      }
    }
  }
  unsigned stage_parity = 0;
  SharedTable<kInts> t;
  t.place(smem, kCap);
  for (int i = threadIdx.x; i < kCap; i += kThreads) t.clear(i);
  if (threadIdx.x == 0) sh.eown = 0.;
  __syncthreads();
  // The next vertex's header (id, offsets, community, k, a_own) is loaded
  // while the current one is evaluated, so its dependent round trips overlap.
  int64_t task = blockIdx.x;
  int v = 0, own = 0;
  int64_t s = 0, eend = 0;
  double ki = 0., aown = 0.;
  if (task < n) {
    v = list[task];
    s = p.off[v];
    eend = p.off[v + 1];
    own = p.comm[v];
    ki = p.k[v];
    aown = p.a[own];
  }
  for (; task < n; task += gridDim.x) {
    const int64_t nt = task + gridDim.x;
    const int vn = nt < n ? list[nt] : 0;
    int64_t sn = 0, en = 0;
    if (nt < n) {
      sn = p.off[vn];
      en = p.off[vn + 1];
    }
    int ownn = 0;
    double kin = 0., aownn = 0.;
    const int32_t* ap = p.adj + s;
    const double* wp = p.w + s;
    if constexpr (kStaged) {
      if (!mbar_wait(&stage_bar, stage_parity)) atomicAdd(p.err, 1ull);
      stage_parity ^= 1u;
      ap = sadj + (s - stage_off[0]);
      wp = sw + (s - stage_off[1]);
    }
    cta_vertex<kThreads, kCap, kChunks, kInts, kTie, kStaged>(
        p, vertex_mass<kMulti>(p, v), v, ap, wp, (int)(eend - s), own, ki, aown, t, sh, [&]() {
          if constexpr (kStaged) {
            // every thread has read the stage (and stage_off): the next vertex's
            // edges go into it while this one is evaluated
            if (threadIdx.x == 0 && nt < n) {
              int64_t a0, w0;
              stage_edges(p, sn, en, sadj, sw, &stage_bar, &a0, &w0);
              stage_off[0] = a0;
              stage_off[1] = w0;
            }
          }
          if (nt < n) {
            ownn = p.comm[vn];
            kin = p.k[vn];
            aownn = p.a[ownn];
          }
        });
    v = vn;
    s = sn;
    eend = en;
    own = ownn;
    ki = kin;
    aown = aownn;
  }
}

constexpr int kWarpCap = 256;     // warp tier: degree <= 192
// threads per CTA and table slots of the CTA tiers
constexpr int kCtaSThreads = 128;
constexpr int kCtaMThreads = 256;
constexpr int kCtaLThreads = 256;
constexpr int kCtaSCap = 1024;
constexpr int kCtaMCap = 2048;
constexpr int kCtaLCap = 4096;
// CTA-S and CTA-M with staged edges: table plus one vertex's widened ranges
constexpr size_t smem_s_staged(bool ints) { return table_bytes(kCtaSCap, ints) + Stage<kCtaSMaxDeg>::kBytes; }
constexpr size_t smem_m_staged(bool ints) { return table_bytes(kCtaMCap, ints) + Stage<kCtaMMaxDeg>::kBytes; }
constexpr int kCtaXAThreads = 512;
// edges of a vertex per thread, at most
constexpr int kCtaSChunks = kCtaSMaxDeg / kCtaSThreads;
constexpr int kCtaMChunks = kCtaMMaxDeg / kCtaMThreads;
constexpr int kCtaLChunks = kCtaLMaxDeg / kCtaLThreads;
constexpr int kCtaXAChunks = kCtaXAMaxDeg / kCtaXAThreads;
constexpr int kCtaXChunks = kCtaXMaxDeg / 1024;
constexpr int kCtaXACap = 8192;   // 512-thread CTA-XA tier, two CTAs an SM
constexpr int kCtaXCap = 16384;   // 1024-thread CTA-XL tier

template <typename K>
int set_smem(K kernel, size_t bytes) {
  NIDO_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return NIDO_OK;
}

template <bool kMulti, bool kInts, bool kTie>
int TierKernels<kMulti, kInts, kTie>::init(int sms, TierResident* R) {
  R->g4 = resident_ctas(k_move_group<4, kMulti, kTie>, 256, 0, sms);
  R->g8 = resident_ctas(k_move_group<8, kMulti, kTie>, 256, 0, sms);
  R->g16 = resident_ctas(k_move_group<16, kMulti, kTie>, 256, 0, sms);
  R->g32 = resident_ctas(k_move_group<32, kMulti, kTie>, 256, 0, sms);
  auto set = [sms](auto kernel, int threads, size_t smem, int64_t* out) -> int {
    NIDO_TRY(set_smem(kernel, smem));
    *out = resident_ctas(kernel, threads, smem, sms);
    return NIDO_OK;
  };
  NIDO_TRY(set(k_move_warp<kWarpCap, kMulti, kInts, kTie>, 256, 8 * table_bytes(kWarpCap, kInts), &R->warp));
  NIDO_TRY(set(k_move_cta<kCtaSThreads, kCtaSCap, kCtaSChunks, kMulti, kInts, kTie>, kCtaSThreads,
               table_bytes(kCtaSCap, kInts), &R->ctas));
  NIDO_TRY(set(k_move_cta<kCtaMThreads, kCtaMCap, kCtaMChunks, kMulti, kInts, kTie>, kCtaMThreads,
               table_bytes(kCtaMCap, kInts), &R->ctam));
  NIDO_TRY(set(k_move_cta<kCtaSThreads, kCtaSCap, kCtaSChunks, kMulti, kInts, kTie, kCtaSMaxDeg>, kCtaSThreads,
               smem_s_staged(kInts), &R->ctas_st));
  NIDO_TRY(set(k_move_cta<kCtaMThreads, kCtaMCap, kCtaMChunks, kMulti, kInts, kTie, kCtaMMaxDeg>, kCtaMThreads,
               smem_m_staged(kInts), &R->ctam_st));
  NIDO_TRY(set(k_move_cta<kCtaLThreads, kCtaLCap, kCtaLChunks, kMulti, kInts, kTie>, kCtaLThreads,
               table_bytes(kCtaLCap, kInts), &R->ctal));
  NIDO_TRY(set(k_move_cta<kCtaXAThreads, kCtaXACap, kCtaXAChunks, kMulti, kInts, kTie>, kCtaXAThreads,
               table_bytes(kCtaXACap, kInts), &R->ctaxa));
  return set(k_move_cta<1024, kCtaXCap, kCtaXChunks, kMulti, kInts, kTie>, 1024, table_bytes(kCtaXCap, kInts),
             &R->ctax);
}

template <bool kMulti, bool kInts, bool kTie>
int TierKernels<kMulti, kInts, kTie>::launch(const TierResident& R, int t, const int32_t* list, int64_t n,
                                             const MoveArgs& p, bool staged, cudaStream_t s) {
  auto grid = [](int64_t blocks, int64_t cap) { return (unsigned)std::min<int64_t>(std::max<int64_t>(blocks, 1), cap); };
  switch (t) {
    case kTierG4: k_move_group<4, kMulti, kTie><<<grid((n + 63) / 64, R.g4), 256, 0, s>>>(list, n, p); break;
    case kTierG8: k_move_group<8, kMulti, kTie><<<grid((n + 31) / 32, R.g8), 256, 0, s>>>(list, n, p); break;
    case kTierG16: k_move_group<16, kMulti, kTie><<<grid((n + 15) / 16, R.g16), 256, 0, s>>>(list, n, p); break;
    case kTierG32: k_move_group<32, kMulti, kTie><<<grid((n + 7) / 8, R.g32), 256, 0, s>>>(list, n, p); break;
    case kTierWarp:
      k_move_warp<kWarpCap, kMulti, kInts, kTie>
          <<<grid((n + 7) / 8, R.warp), 256, 8 * table_bytes(kWarpCap, kInts), s>>>(list, n, p);
      break;
    case kTierCtaS:
      if (staged)
        k_move_cta<kCtaSThreads, kCtaSCap, kCtaSChunks, kMulti, kInts, kTie, kCtaSMaxDeg>
            <<<grid(n, R.ctas_st), kCtaSThreads, smem_s_staged(kInts), s>>>(list, n, p);
      else
        k_move_cta<kCtaSThreads, kCtaSCap, kCtaSChunks, kMulti, kInts, kTie>
            <<<grid(n, R.ctas), kCtaSThreads, table_bytes(kCtaSCap, kInts), s>>>(list, n, p);
      break;
    case kTierCtaM:
      if (staged)
        k_move_cta<kCtaMThreads, kCtaMCap, kCtaMChunks, kMulti, kInts, kTie, kCtaMMaxDeg>
            <<<grid(n, R.ctam_st), kCtaMThreads, smem_m_staged(kInts), s>>>(list, n, p);
      else
        k_move_cta<kCtaMThreads, kCtaMCap, kCtaMChunks, kMulti, kInts, kTie>
            <<<grid(n, R.ctam), kCtaMThreads, table_bytes(kCtaMCap, kInts), s>>>(list, n, p);
      break;
    case kTierCtaL:
      k_move_cta<kCtaLThreads, kCtaLCap, kCtaLChunks, kMulti, kInts, kTie>
          <<<grid(n, R.ctal), kCtaLThreads, table_bytes(kCtaLCap, kInts), s>>>(list, n, p);
      break;
    case kTierCtaXA:
      k_move_cta<kCtaXAThreads, kCtaXACap, kCtaXAChunks, kMulti, kInts, kTie>
          <<<grid(n, R.ctaxa), kCtaXAThreads, table_bytes(kCtaXACap, kInts), s>>>(list, n, p);
      break;
    default:
      k_move_cta<1024, kCtaXCap, kCtaXChunks, kMulti, kInts, kTie>
          <<<grid(n, R.ctax), 1024, table_bytes(kCtaXCap, kInts), s>>>(list, n, p);
      break;
  }
  NIDO_LAUNCH_CHECK();
  return NIDO_OK;
}
#endif  // NIDO_TIER_KERNELS

}  // namespace nido
#endif
