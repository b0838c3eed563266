// Launch planning of the register-tile kernels (regtile.cuh): window shape, tile
// and pass depth from the array's size, and the launches of a rollout.
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include "regtile.cuh"
#include "regtile_host.h"

namespace pde {

namespace {

// Window and tile along one axis for nt tiles: the rows (columns) the window
// needs, a multiple of `unit` and at most n, or 0 when it does not fit in `cap`.
// `hold`: the cells the window may use; n < hold (a slab's rows): halo on both sides.
int axis_window(int n, int hold, int nt, int H, int unit, int cap) {
  const int tile = (n + nt - 1) / nt;
  const int most = hold / unit * unit;
  const int need = n < hold ? tile + 2 * H : nt == 1 ? n : nt == 2 ? tile + H : tile + 2 * H;
  int win = (need + unit - 1) / unit * unit;
  if (win > most) win = most;
  if (win < need || win > cap || (long long)(nt - 1) * tile >= n) return 0;
  return win;
}

// Fewest tiles along an axis of n whose windows of at most cap hold tile and halo.
int fewest(int n, int hold, int H, int unit, int cap) {
  if (n == hold && n <= cap && n % unit == 0) return 1;
  const int two = (n + 1) / 2 + H;
  if (n == hold && two <= cap / unit * unit && two <= n / unit * unit) return 2;
  const int room = cap / unit * unit - 2 * H;
  return room < 1 ? 0 : (n + room - 1) / room;
}

}  // namespace

bool rt_grid_tiles(int BX, int BY, int H, int C, int RPT, int cap_x, int cap_y, int tile_x, int tile_y, RTGeom* W) {
  const int nx = tile_x > 0 ? (BX + tile_x - 1) / tile_x : fewest(BX, BX, H, RPT, cap_x);
  const int ny = tile_y > 0 ? (BY + tile_y - 1) / tile_y : fewest(BY, BY, H, C, cap_y);
  if (nx < 1 || ny < 1) return false;
  const int nr = axis_window(BX, BX, nx, H, RPT, cap_x), nc = axis_window(BY, BY, ny, H, C, cap_y);
  if (nr < 2 * RPT || nc < 2 * C) return false;
  const int tbx = (BX + nx - 1) / nx, tby = (BY + ny - 1) / ny;
  if ((nx > 1 && H > tbx) || (ny > 1 && H > tby)) return false;
  *W = RTGeom{BX, BY, 0, BX, true, true, tbx, tby, ny, H, nr, nc};
  return true;
}

// The shape with the least estimated time per step, over the four strips (C, RPT),
// the pass depths, and per axis the largest windows or as many tiles as fill the
// SMs once or twice.  A step of a block costs its
// arithmetic (active strips x cells x operations over the SM's 128 lanes, at the
// share of that rate the kernels reach) or, when there is little of it, the
// latency of publish, barrier, read and the dependent sums; a pass of k steps costs
// a dependent launch and the loads and stores of its windows.
RTPlan rt_plan(const RTCost& cost, int BX, int Y, int X0, int X1, int R, int nsteps, int k_req, bool k_only,
               int tile_x, int tile_y, int sms) {
  const int X = X1 - X0;
  RTPlan best;
  best.ok = false;
  best.cycles = 1e30;
  auto consider = [&](int ci, int C, int RPT, int k, int nx, int ny) {
    const int H = k * R;
    const int nr = axis_window(X, BX, nx, H, RPT, cost.max_warps[ci] * RPT);
    int nc = axis_window(Y, Y, ny, H, C, 32 * C);
    if (nr < 2 * RPT || nc < 2 * C) return;
    const long long tiles = (long long)nx * ny;
    const int tbx = (X + nx - 1) / nx;
    int tby = (Y + ny - 1) / ny;
    if (cost.even && ny > 1 && (tby & 1) && (ny - 1) * (tby + 1) < Y) {
      const int wide = (tby + 1 + (ny == 2 ? 1 : 2) * H + C - 1) / C * C;
      if (wide <= 32 * C && wide <= Y) {
        ++tby;
        nc = wide > nc ? wide : nc;
      }
    }
    const double act = fmin((double)nr, tbx + 1.4 * H + RPT);  // strips rest as the reach shrinks
    const double per_sm = (double)((tiles + sms - 1) / sms);
    const double arith = act * 32.0 * C * cost.ops[ci] / 128.0 * per_sm;
    const double step = fmax(arith, cost.latency + RPT * C * cost.chain) + cost.barrier * (nr / RPT);
    const double pass = cost.relaunch + RPT * C * cost.cell * per_sm;
    const double t = step + pass * ((nsteps + k - 1) / k) / nsteps;
    if (t >= best.cycles) return;
    best.ok = true;
    best.cycles = t;
    best.shape = ci;
    best.C = C;
    best.RPT = RPT;
    best.k = k;
    best.W = RTGeom{BX, Y, X0, X1, true, true, tbx, tby, ny, H, nr, nc};
    best.tiles = (int)tiles;
    best.threads = nr / RPT * 32;
  };
  static const int depths[] = {1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 16, 17, 20, 24, 25};
  for (int ci = 0; ci < 4; ++ci) {
    if (!((cost.shapes >> ci) & 1)) continue;
    const int C = ci & 1 ? 4 : 2, RPT = ci & 2 ? 8 : 4;
    for (int d : depths) {
      const int k = k_only ? k_req : d;
      if (cost.even && (k & 1) && k != nsteps && k != k_req && k > 1) continue;
      if (k > nsteps || (k_req > 0 && k > k_req)) break;
      int ny = tile_y > 0 ? (Y + tile_y - 1) / tile_y : fewest(Y, Y, k * R, C, 32 * C);
      if (ny < 1) break;
      for (int more = 0; more < 3; ++more, ++ny) {
        if (tile_x > 0) {
          consider(ci, C, RPT, k, (X + tile_x - 1) / tile_x, ny);
        } else {
          // the largest windows, and as many tiles as fill the SMs once or twice
          const int lo = fewest(X, BX, k * R, RPT, cost.max_warps[ci] * RPT);
          if (lo < 1) break;
          consider(ci, C, RPT, k, lo, ny);
          for (int m = 1; m <= 2; ++m) {
            const int nx = m * sms / ny;
            if (nx > lo && X / nx >= 4) consider(ci, C, RPT, k, nx, ny);
          }
        }
        if (tile_y > 0) break;
      }
      if (k_only) break;
    }
  }
  return best;
}

namespace {

template <int R, int C, int RPT>
int heat_launch(const RTPlan& L, const RHParams& P, const PdeBCRules& rules, cudaStream_t st) {
  auto kern = heat2d_rt_kernel<R, C, RPT>;
  const size_t smem = rt_rows_floats<R, C>(L.threads / 32) * sizeof(float);
  if (smem > 48 * 1024 - 4096)
    PDE_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return launch_pdl(kern, L.tiles, L.threads, smem, st, P, rules);
}

template <int R>
int heat_launch_shape(const RTPlan& L, const RHParams& P, const PdeBCRules& rules, cudaStream_t st) {
  switch (L.shape) {
    case 0: return heat_launch<R, 2, 4>(L, P, rules, st);
    case 1: return heat_launch<R, 4, 4>(L, P, rules, st);
    case 2: return heat_launch<R, 2, 8>(L, P, rules, st);
    default:
      if constexpr (R == 1) return heat_launch<R, 4, 8>(L, P, rules, st);
      else return PDE_ERR_UNSUPPORTED;  // order 4 with 32 cells a thread does not fit the registers: never planned
  }
}

}  // namespace

// Scalar 2D grids of at least 8 x 8 interior cells whose first ghost layer is filled
// on every face (the fill replaces the stored ghosts).  Others run the
// shared-memory kernels.
bool rt_heat_shape(const Geo& G, int ncomp, const PdeBCRules* rules) {
  if (ncomp != 1 || G.ndims != 2 || G.n[2] != 1 || G.g < G.order / 2 || G.ext[0] < 8 || G.ext[1] < 8 ||
      G.n[0] * G.n[1] >= (1LL << 30))
    return false;
  return !rules || rt_fills_all_faces(*rules);
}

// Every ghost next to the box is filled by some group (2D, component 0).
bool rt_fills_all_faces(const PdeBCRules& rules) {
  for (int K = 0; K < 27; ++K)
    for (int a = 0; a < 2; ++a) {
      const int k[3] = {K / 9, (K / 3) % 3, K % 3};
      if (k[2] == 1 && k[a] != 1 && rules.ghost_group[K][a][0] < 0) return false;
    }
  return true;
}

RTPlan rt_heat_plan(const Geo& G, int nsteps, int k_req, int tile_x, int tile_y) {
  const int R = G.order / 2;
  RTCost cost = {};
  // Fitted to timings of every shape and depth on 13 grids (66^2 .. 2050^2, both
  // orders): the plan is within 12% of the fastest of them on each.  Small strips
  // pay more per cell (row exchange and shuffles), large ones need large grids:
  // 256^2 runs (2, 4) at k = 16, 1024^2 (4, 8) at k = 10.
  if (R == 1) {
    cost.ops[0] = 17.0; cost.ops[1] = 14.5; cost.ops[2] = 16.5; cost.ops[3] = 12.5;
  } else {
    cost.ops[0] = 36.0; cost.ops[1] = 40.0; cost.ops[2] = 40.0;
  }
  cost.latency = R == 1 ? 250.0 : 350.0;
  cost.chain = R == 1 ? 10.0 : 20.0;
  cost.barrier = 6.0;
  cost.relaunch = 4200.0;
  cost.cell = 130.0;
  cost.shapes = R == 1 ? 15 : 7;
  for (int i = 0; i < 4; ++i) cost.max_warps[i] = rt_heat_warps(i & 1 ? 4 : 2, i & 2 ? 8 : 4);
  return rt_plan(cost, (int)G.ext[0], (int)G.ext[1], 0, (int)G.ext[0], R, nsteps, k_req, false, tile_x, tile_y, sm_count());
}

int rt_heat_run(const RTPlan& L, const float* u_in, float* u_out, float* work, const Geo& G,
                const Weights& W, const PdeBCRules& rules, float alpha, float dt, int nsteps, double t0, double tstep,
                int n0, cudaStream_t st) {
  RHParams P;
  memset(&P, 0, sizeof(P));
  P.W = L.W;
  P.X = (int)G.n[0];
  P.Y = (int)G.n[1];
  P.g = G.g;
  for (int t = 0; t <= W.radius; ++t) P.w[t] = W.w[t];
  P.alpha = alpha;
  P.dt = dt;
  P.negzero = -0.0f;
  P.t0 = t0;
  P.tstep = tstep;
  const int R = W.radius;
  const int npasses = (nsteps + L.k - 1) / L.k;
  const float* src = u_in;
  float* dst = (u_out == u_in || npasses % 2 == 0) ? work : u_out;
  for (int done = 0; done < nsteps; done += P.k) {
    P.k = nsteps - done < L.k ? nsteps - done : L.k;
    P.n0 = n0 + done;
    P.in = src;
    P.out = dst;
    const int rc = R == 1 ? heat_launch_shape<1>(L, P, rules, st) : heat_launch_shape<2>(L, P, rules, st);
    if (rc) return rc;
    src = dst;
    dst = dst == work ? u_out : work;
  }
  if (src != u_out) {
    const size_t bytes = (size_t)(G.n[0] * G.n[1]) * sizeof(float);
    PDE_CUDA_CHECK(cudaMemcpyAsync(u_out, src, bytes, cudaMemcpyDeviceToDevice, st));
  }
  return PDE_OK;
}

namespace {

template <int C, int RPT>
int jacobi_launch(const RTPlan& L, const RJParams& P, const PdeBCRules& rules, cudaStream_t st) {
  const size_t smem = rt_rows_floats<1, C>(L.threads / 32) * sizeof(float);
  return launch_pdl(jacobi2d_rt_kernel<C, RPT>, L.tiles, L.threads, smem, st, P, rules);
}

}  // namespace

RTPlan rt_jacobi_plan(const JacobiRun& J, int nsweeps, int k_req, bool k_only, int tile_x, int tile_y) {
  RTPlan no;
  no.ok = false;
  const int lo = J.held_lo > J.g ? J.held_lo : J.g, hi = J.held_hi < J.X - J.g ? J.held_hi : J.X - J.g;
  const int o0 = J.own_lo > J.g ? J.own_lo : J.g, o1 = J.own_hi < J.X - J.g ? J.own_hi : J.X - J.g;
  if (hi - lo < 8 || o1 - o0 < 1 || J.Y - 2 * J.g < 8) return no;
  RTCost cost = {};
  cost.ops[0] = 10.0; cost.ops[1] = 8.0; cost.ops[2] = 9.0; cost.ops[3] = 7.0;
  cost.latency = 220.0;
  cost.chain = 8.0;
  cost.barrier = 6.0;
  cost.relaunch = 4200.0;
  cost.cell = 180.0;
  cost.shapes = 15;
  for (int i = 0; i < 4; ++i) cost.max_warps[i] = RT_WARPS;
  RTPlan L = rt_plan(cost, hi - lo, J.Y - 2 * J.g, o0 - lo, o1 - lo, 1, nsweeps, k_req, k_only, tile_x, tile_y, sm_count());
  L.W.xlo = lo == J.g;
  L.W.xhi = hi == J.X - J.g;
  return L;
}

int rt_jacobi_pass(const RTPlan& L, const JacobiRun& J, const float* pin, float* pout, const float* rhs, float* resid,
                   int k, bool last, const PdeBCRules& rules, cudaStream_t st) {
  RJParams P;
  memset(&P, 0, sizeof(P));
  P.W = L.W;
  P.X = J.X;
  P.Y = J.Y;
  P.g = J.g;
  P.x0 = J.held_lo > J.g ? J.held_lo : J.g;
  P.own_lo = J.own_lo;
  P.own_hi = J.own_hi;
  P.k = k;
  P.h2 = J.h2;
  P.negzero = -0.0f;
  P.in = pin;
  P.out = pout;
  P.rhs = rhs;
  P.resid = last ? resid : nullptr;
  switch (L.shape) {
    case 0: return jacobi_launch<2, 4>(L, P, rules, st);
    case 1: return jacobi_launch<4, 4>(L, P, rules, st);
    case 2: return jacobi_launch<2, 8>(L, P, rules, st);
    default: return jacobi_launch<4, 8>(L, P, rules, st);
  }
}

}  // namespace pde
