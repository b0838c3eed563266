// Host side of the register-tile kernels: launch plans and rollouts.
#pragma once
#include "common.cuh"

namespace pde {

struct RTGeom {
  int BX, BY;          // the box the windows lie in
  int X0, X1;          // rows the tiles cover (a slab: its own rows; else 0, BX)
  bool xlo, xhi;       // the box's first (last) row is a boundary node row (a slab: not at a cut side)
  int TBX, TBY;        // tile
  int tiles_y;
  int H;               // halo (cells)
  int NR, NC;          // window rows (a multiple of RPT) and columns (a multiple of C)
};

// Most warps of a block: 128 registers a thread; the heat step with 32 cells a thread takes 168.
constexpr int RT_WARPS = 16;
constexpr int rt_heat_warps(int C, int RPT) { return C * RPT >= 32 ? 12 : RT_WARPS; }

struct RTCost {
  double ops[4];       // issue cost of a cell and step in lane operations, by shape
  double latency;      // cycles of a step with little arithmetic ...
  double chain;        // ... and per cell of a thread
  double barrier;      // cycles of a barrier per warp
  double relaunch;     // cycles of a pass besides its steps: the dependent launch ...
  double cell;         // ... and per cell of a thread, its load and store
  int max_warps[4];    // of a block, by shape
  bool even;           // even depths and tile widths (column pairs that stay together)
  int shapes;          // bit per (C, RPT) pair: (2,4), (4,4), (2,8), (4,8)
};

struct RTPlan {
  bool ok;
  int shape, C, RPT, k, tiles, threads;
  double cycles;
  RTGeom W;
};

// Tiles and windows of a box for windows of at most cap_x x cap_y cells, strips of
// RPT rows and lanes of C columns; false when a window would not fit in the box or
// its halo would reach past a neighbouring tile.
bool rt_grid_tiles(int BX, int BY, int H, int C, int RPT, int cap_x, int cap_y, int tile_x, int tile_y, RTGeom* W);

// Box of BX x BY cells, tiles over rows [X0, X1).  k_req: deepest pass allowed (0:
// any); k_only: exactly that depth.
RTPlan rt_plan(const RTCost& cost, int BX, int BY, int X0, int X1, int R, int nsteps, int k_req, bool k_only,
               int tile_x, int tile_y, int sms);

bool rt_heat_shape(const Geo& G, int ncomp, const PdeBCRules* rules);
RTPlan rt_heat_plan(const Geo& G, int nsteps, int k_req, int tile_x, int tile_y);
int rt_heat_run(const RTPlan& L, const float* u_in, float* u_out, float* work, const Geo& G, const Weights& W,
                const PdeBCRules& rules, float alpha, float dt, int nsteps, double t0, double tstep, int n0,
                cudaStream_t st);

// Jacobi sweeps of the cavity's pressure on rows [own_lo, own_hi) of a domain of
// X x Y cells, arrays holding rows [held_lo, held_hi) (all four in global rows).
struct JacobiRun {
  int X, Y, g, own_lo, own_hi, held_lo, held_hi;
  float h2;
};
bool rt_fills_all_faces(const PdeBCRules& rules);
RTPlan rt_jacobi_plan(const JacobiRun& J, int nsweeps, int k_req, bool k_only, int tile_x, int tile_y);
// One pass of k sweeps; `last`: add the squared updates of the last sweep to *resid.
int rt_jacobi_pass(const RTPlan& L, const JacobiRun& J, const float* pin, float* pout, const float* rhs, float* resid,
                   int k, bool last, const PdeBCRules& rules, cudaStream_t st);

// Wave passes (wave_rt.cuh): forward, adjoint, or both of equal depth in one launch.
struct WaveRun {
  int X, Y, g;
  float w[2];
  const float* K;
  int srcx, srcy;  // array coordinates, -1: none
};
struct WaveFwd {
  int k;
  const float *um, *u0;
  float *um_out, *u0_out, *lst;
  const float* src;
};
struct WaveAdj {
  int k;
  const float *m1, *m2;
  float *m1_out, *m2_out;
  const float* lsts;
  float* gK;
};
RTPlan rt_wave_plan(const WaveRun& J, bool fwd, bool adj, int nsteps, int k_req, int tile_x, int tile_y);
int rt_wave_pass(const RTPlan& L, const WaveRun& J, const WaveFwd* f, const WaveAdj* a, cudaStream_t st);

// Passes of the differentiable heat rollout of order 2 (heat_adj_rt.cuh).
struct HeatFieldPass {
  int X, Y, g, k;
  float w[2], dt;
  const float *alpha, *in;
  float *out, *lst;
  const float* lsts;
  float* galpha;  // set: an adjoint pass
  double t0, tstep;
  int n0;
};
RTPlan rt_heat_field_plan(const Geo& G, const PdeBCRules& rules, bool adjoint, int nsteps, int k_req, int tile_x,
                          int tile_y);
int rt_heat_field_pass(const RTPlan& L, const HeatFieldPass& H, const PdeBCRules& rules, cudaStream_t st);

}  // namespace pde
