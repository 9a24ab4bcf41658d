// phase_loop.cu -- host side of the persistent phase loop (phase_loop.cuh).
#include "phase_loop.cuh"

#include <string.h>

#include <algorithm>
#include <mutex>
#include <vector>

namespace nido {
namespace {

int64_t g_loop_resident[2][2][2];  // [many graphs][integer tables][reference tie rule]

// One block's share of a batch's edges: small phases take fewer blocks, whose
// barriers are cheaper, but each vertex waits for a chain of gathers, so a
// warp should get few.  Sweeps of a 1,000-vertex / 20,011-vertex graph: 50 / 65
// us with 64 to 256 edges a block, 65 / 75 us with 1024, 150 / 130 us with 4096.
constexpr int64_t kLoopBlockEdges = 128;

template <bool kMulti, bool kInts>
int run_loop(nido_graph_s* g, int tie, double tau, int64_t max_iter, const LoopGraphs* many, PhaseLoop* r,
             int64_t log_cap, bool* unsupported) {
  cudaStream_t s = g->ctx->stream;
  const int nb = g->nbatches;
  const int64_t nv = g->nv;
  const int64_t nt = (int64_t)kNumTiers * nb + 1;
  LoopArgs<kInts> A;
  memset(&A, 0, sizeof(A));
  A.p = move_args(g);
  A.comm = g->comm;
  A.newc = g->newc;
  A.a = g->a;
  A.perm = g->perm;
  A.nb = nb;
  A.nv = nv;
  int64_t grid = std::min<int64_t>((nv + 7) / 8, 65535);
  A.S = 128 * grid;
  A.ngroups = (std::min<int64_t>(A.S, nv) + 15) / 16;
  A.tau = tau;
  A.max_iter = max_iter;
  // list offsets, cuts and hub ranges in one copy
  std::vector<int64_t> plan(g->tier_off.begin(), g->tier_off.begin() + nt);
  const bool ranges = !g->gid && !g->color_mode;
  if (ranges) plan.insert(plan.end(), g->cuts.begin(), g->cuts.begin() + nb + 1);
  const size_t hub_at = plan.size();
  if (g->nhubs > 0)
    for (int b = 0; b < nb; ++b) {
      int64_t w4[4] = {0, 0, 0, 0};
      if (g->hub_wave_off[b + 1] - g->hub_wave_off[b] > 1) { *unsupported = true; return NIDO_OK; }
      if (g->hub_wave_off[b + 1] > g->hub_wave_off[b]) {
        const nido_graph_s::HubWave& w = g->hub_waves[g->hub_wave_off[b]];
        w4[0] = w.i0; w4[1] = w.i1; w4[2] = w.s0; w4[3] = w.s1;
      }
      plan.insert(plan.end(), w4, w4 + 4);
    }
  Arena ar(g->scratch, g->scratch_bytes);
  int64_t* dplan = ar.take<int64_t>((int64_t)plan.size());
  A.ctl = ar.take<PhaseCtl>(1);
  A.selfv = ar.take<double>(nv);
  A.modv = many ? many->modv : ar.take<double>(A.ngroups);
  A.log = log_cap > 0 ? ar.take<double>(2 * log_cap) : nullptr;
  A.log_cap = log_cap;
  if (!dplan || !A.ctl || !A.selfv || !A.modv || (log_cap > 0 && !A.log)) { *unsupported = true; return NIDO_OK; }
  NIDO_CUDA_TRY(cudaMemcpyAsync(dplan, plan.data(), sizeof(int64_t) * plan.size(), cudaMemcpyHostToDevice, s));
  A.tier_off = dplan;
  A.cuts = ranges ? dplan + nt : nullptr;
  A.nhubs = g->nhubs;
  if (g->nhubs > 0) {
    A.hub_rng = dplan + hub_at;
    A.nitems = g->hub_nitems;
    A.items = g->hub_items;
    A.slices = g->hub_slices;
    A.slice_first = g->hub_slice_first;
    A.item_first = g->hub_item_first;
    A.hub_v = g->hub_v;
    A.hub_toff = g->hub_toff;
    A.hub_cap = g->hub_capv;
    A.hub_done = g->hub_done;
    A.res = reinterpret_cast<SliceResult*>(g->hub_res);
    A.part = g->hub_part;
    if constexpr (kInts) A.tab.slots = g->gpacked;
    else A.tab = HubTable<false>{g->gkeys, g->gvals};
  }
  if (many) {
    A.gl = many->gl;
    A.qoff = many->qoff;
    A.nl = many->nl;
    A.nbig = many->nbig;
    A.gbase = g->gbase;
    A.gq = many->q;
    A.gq_old = many->q_old;
    A.loops_phase = many->loops_phase;
    A.loops_total = many->loops_total;
    A.giter = many->giter;
    A.grest = many->grest;
    A.relist_below = many->relist_below;
  }
  // vertices in no tier list (no edges) have no in-community weight
  NIDO_CUDA_TRY(cudaMemsetAsync(A.selfv, 0, sizeof(double) * nv, s));
  NIDO_CUDA_TRY(cudaMemsetAsync(A.ctl, 0, sizeof(PhaseCtl), s));
  const int64_t resident = g_loop_resident[kMulti ? 1 : 0][kInts ? 1 : 0][tie == NIDO_TIE_NIDO ? 1 : 0];
  const int64_t blocks = std::max<int64_t>(1, std::min(resident, (many && g->plan_ne >= 0 ? g->plan_ne : g->ne) / nb / kLoopBlockEdges));
  NIDO_TRY((PhaseLoopKernel<kMulti, kInts>::launch(A, tie == NIDO_TIE_NIDO, blocks, s)));
  PhaseCtl hc;
  NIDO_CUDA_TRY(cudaMemcpyAsync(&hc, A.ctl, sizeof(hc), cudaMemcpyDeviceToHost, s));
  r->log.clear();
  if (log_cap > 0) {
    r->log.resize(2 * (size_t)log_cap);
    NIDO_CUDA_TRY(cudaMemcpyAsync(r->log.data(), A.log, sizeof(double) * r->log.size(), cudaMemcpyDeviceToHost, s));
  }
  NIDO_CUDA_TRY(cudaStreamSynchronize(s));
  if (hc.fail) return nido_set_error(NIDO_E_TIMEOUT, "the phase loop's grid barrier gave up");
  r->q_old = hc.q_old;
  r->q = hc.q;
  r->loops = hc.loops;
  r->move_ms = hc.move_ns * 1e-6;
  r->q_ms = hc.q_ns * 1e-6;
  for (int i = 0; i < 4; ++i) r->counters[i] = hc.counters[i];
  if (log_cap > 0) r->log.resize(2 * (size_t)std::min<int64_t>(hc.loops, log_cap));
  return NIDO_OK;
}

}  // namespace

int phase_loop_init(bool many) {
  int dev = 0, sms = kSMs;
  NIDO_CUDA_TRY(cudaGetDevice(&dev));
  NIDO_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  static std::mutex mu;  // contexts may be created from several threads
  std::lock_guard<std::mutex> lk(mu);
  if (many) {
    NIDO_TRY((PhaseLoopKernel<true, false>::init(sms, g_loop_resident[1][0])));
    return PhaseLoopKernel<true, true>::init(sms, g_loop_resident[1][1]);
  }
  NIDO_TRY((PhaseLoopKernel<false, false>::init(sms, g_loop_resident[0][0])));
  return PhaseLoopKernel<false, true>::init(sms, g_loop_resident[0][1]);
}

// The iteration loop of the prepared phase on the persistent kernel; many:
// the per-graph state of a many-graph phase.  *unsupported is set (and nothing
// has run) when the phase's plan does not fit it.
int persistent_phase_loop(nido_graph_s* g, int tie, double tau, int64_t max_iter, bool want_log, const LoopGraphs* many,
                          PhaseLoop* r, bool* unsupported) {
  *unsupported = false;
  if (!g->bins_valid) NIDO_TRY(build_batches(g));
  if (!g->loop_plan || g->nv == 0) { *unsupported = true; return NIDO_OK; }
  const int64_t log_cap = want_log ? std::min<int64_t>(max_iter, kLoopLogCap) : 0;
  if (many)
    return g->int_weights ? run_loop<true, true>(g, tie, tau, max_iter, many, r, log_cap, unsupported)
                          : run_loop<true, false>(g, tie, tau, max_iter, many, r, log_cap, unsupported);
  return g->int_weights ? run_loop<false, true>(g, tie, tau, max_iter, nullptr, r, log_cap, unsupported)
                        : run_loop<false, false>(g, tie, tau, max_iter, nullptr, r, log_cap, unsupported);
}

}  // namespace nido
