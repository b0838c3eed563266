// Plans and launches of the wave's register-tile passes.
#include <string.h>

#include "wave_rt.cuh"

namespace pde {

RTPlan rt_wave_plan(const WaveRun& J, bool fwd, bool adj, int nsteps, int k_req, int tile_x, int tile_y) {
  const int BX = J.X - 2 * (J.g + 1), BY = J.Y - 2 * (J.g + 1);
  RTPlan no;
  no.ok = false;
  if (BX < 8 || BY < 8 || (long long)J.X * J.Y >= (1LL << 30)) return no;
  RTCost cost = {};
  const double chains = fwd && adj ? 2.0 : 1.0;
  cost.ops[0] = 18.0 * chains; cost.ops[1] = 16.0; cost.ops[2] = 16.0;
  cost.latency = 250.0 * (fwd && adj ? 1.4 : 1.0);
  cost.chain = 10.0 * chains;
  cost.barrier = 6.0;
  cost.relaunch = 4200.0;
  cost.cell = 200.0 * chains;
  cost.even = true;
  cost.shapes = adj ? 1 : 7;  // the adjoint holds seven values a cell: 8 cells a thread
  for (int i = 0; i < 4; ++i) cost.max_warps[i] = RT_WARPS;
  return rt_plan(cost, BX, BY, 0, BX, 1, nsteps, k_req, false, tile_x, tile_y, sm_count());
}

namespace {

template <bool F, bool A, int C, int RPT>
int wave_launch(const RTPlan& L, const RWParams& P, bool pairs, cudaStream_t st) {
  const size_t smem = (size_t)(F && A ? 2 : 1) * rt_rows_floats<1, C>(L.threads / 32) * sizeof(float);
  return pairs ? launch_pdl(wave_rt_kernel<F, A, true, C, RPT>, L.tiles, L.threads, smem, st, P)
               : launch_pdl(wave_rt_kernel<F, A, false, C, RPT>, L.tiles, L.threads, smem, st, P);
}

int wave_launch_shape(const RTPlan& L, const RWParams& P, bool pairs, cudaStream_t st) {
  switch (L.shape) {
    case 0: return wave_launch<true, false, 2, 4>(L, P, pairs, st);
    case 1: return wave_launch<true, false, 4, 4>(L, P, pairs, st);
    default: return wave_launch<true, false, 2, 8>(L, P, pairs, st);
  }
}

}  // namespace

int rt_wave_pass(const RTPlan& L, const WaveRun& J, const WaveFwd* f, const WaveAdj* a, cudaStream_t st) {
  RWParams P;
  memset(&P, 0, sizeof(P));
  P.W = L.W;
  P.X = J.X;
  P.Y = J.Y;
  P.pad = J.g + 1;
  P.w[0] = J.w[0];
  P.w[1] = J.w[1];
  P.negzero = -0.0f;
  P.K = J.K;
  P.srcx = P.srcy = -1;
  uintptr_t bits = reinterpret_cast<uintptr_t>(J.K);
  auto see = [&](const void* p) { bits |= reinterpret_cast<uintptr_t>(p); };
  if (f) {
    P.kf = f->k;
    P.um_in = f->um;
    P.u0_in = f->u0;
    P.um_out = f->um_out;
    P.u0_out = f->u0_out;
    P.lst = f->lst;
    P.src = f->src;
    if (J.srcx >= 0 && f->src) {
      P.srcx = J.srcx - P.pad;
      P.srcy = J.srcy - P.pad;
      // a source on a node or ghost cell never enters the state
      if (P.srcx < 0 || P.srcx >= L.W.BX || P.srcy < 0 || P.srcy >= L.W.BY) P.srcx = -1;
    }
    see(f->um); see(f->u0); see(f->um_out); see(f->u0_out); see(f->lst);
  }
  if (a) {
    P.ka = a->k;
    P.m1_in = a->m1;
    P.m2_in = a->m2;
    P.m1_out = a->m1_out;
    P.m2_out = a->m2_out;
    P.lsts = a->lsts;
    P.gK = a->gK;
    see(a->m1); see(a->m2); see(a->m1_out); see(a->m2_out); see(a->lsts); see(a->gK);
  }
  // windows start at even columns: 0, a multiple of the (even) tile minus the halo,
  // or the box's end minus the window
  const RTGeom& W = L.W;
  const bool one = W.TBY >= W.BY;
  const bool pairs = (bits & 7u) == 0 && ((P.Y | P.pad | W.BY | W.NC) & 1) == 0 && (one || ((W.TBY | W.H) & 1) == 0);
  if (f && a) return wave_launch<true, true, 2, 4>(L, P, pairs, st);
  return f ? wave_launch_shape(L, P, pairs, st) : wave_launch<false, true, 2, 4>(L, P, pairs, st);
}

}  // namespace pde
