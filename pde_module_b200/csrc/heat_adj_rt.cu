// Plans and launches of the differentiable heat rollout's register-tile passes.
#include <string.h>

#include "heat_adj_rt.cuh"

namespace pde {

RTPlan rt_heat_field_plan(const Geo& G, const PdeBCRules& rules, bool adjoint, int nsteps, int k_req, int tile_x,
                          int tile_y) {
  RTPlan no;
  no.ok = false;
  if (G.order != 2 || !rt_heat_shape(G, 1, &rules)) return no;
  RTCost cost = {};
  cost.ops[0] = adjoint ? 24.0 : 19.0;
  cost.ops[1] = cost.ops[2] = 17.0;
  cost.latency = adjoint ? 300.0 : 270.0;
  cost.chain = adjoint ? 14.0 : 11.0;
  cost.barrier = 6.0;
  cost.relaunch = 4200.0;
  cost.cell = adjoint ? 300.0 : 180.0;
  cost.shapes = adjoint ? 1 : 7;
  for (int i = 0; i < 4; ++i) cost.max_warps[i] = RT_WARPS;
  return rt_plan(cost, (int)G.ext[0], (int)G.ext[1], 0, (int)G.ext[0], 1, nsteps, k_req, false, tile_x, tile_y,
                 sm_count());
}

int rt_heat_field_pass(const RTPlan& L, const HeatFieldPass& H, const PdeBCRules& rules, cudaStream_t st) {
  RGParams P;
  memset(&P, 0, sizeof(P));
  P.W = L.W;
  P.X = H.X;
  P.Y = H.Y;
  P.g = H.g;
  P.k = H.k;
  P.w[0] = H.w[0];
  P.w[1] = H.w[1];
  P.dt = H.dt;
  P.negzero = -0.0f;
  P.alpha = H.alpha;
  P.in = H.in;
  P.out = H.out;
  P.lst = H.lst;
  P.lsts = H.lsts;
  P.galpha = H.galpha;
  P.t0 = H.t0;
  P.tstep = H.tstep;
  P.n0 = H.n0;
  const int nw = L.threads / 32;
  if (H.galpha)
    return launch_pdl(heat2d_adj_rt_kernel, L.tiles, L.threads, rt_rows_floats<1, 2>(nw) * sizeof(float), st, P, rules);
  switch (L.shape) {
    case 0:
      return launch_pdl(heat2d_field_rt_kernel<2, 4>, L.tiles, L.threads, rt_rows_floats<1, 2>(nw) * sizeof(float), st, P, rules);
    case 1:
      return launch_pdl(heat2d_field_rt_kernel<4, 4>, L.tiles, L.threads, rt_rows_floats<1, 4>(nw) * sizeof(float), st, P, rules);
    default:
      return launch_pdl(heat2d_field_rt_kernel<2, 8>, L.tiles, L.threads, rt_rows_floats<1, 2>(nw) * sizeof(float), st, P, rules);
  }
}

}  // namespace pde
