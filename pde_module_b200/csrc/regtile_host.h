// Host side of the register-tile kernels: launch plans and rollouts.
#pragma once
#include "common.cuh"

namespace pde {

struct RTGeom {
  int BX, BY;          // the box the tiles cover
  int TBX, TBY;        // tile
  int tiles_y;
  int H;               // halo (cells)
  int NR, NC;          // window rows (a multiple of RPT) and columns (a multiple of C)
};

// Warps of a block: 168 registers a thread for 32 cells, 128 for 8 and 16.
constexpr int rt_max_warps(int C, int RPT) { return C * RPT >= 32 ? 12 : 16; }

struct RTCost {
  double ops[4];       // issue cost of a cell and step in lane operations, by shape
  double latency;      // cycles of a step with little arithmetic ...
  double chain;        // ... and per cell of a thread
  double barrier;      // cycles of a barrier per warp
  double relaunch;     // cycles of a pass besides its steps: the dependent launch ...
  double cell;         // ... and per cell of a thread, its load and store
  int shapes;          // bit per (C, RPT) pair: (2,4), (4,4), (2,8), (4,8)
};

struct RTPlan {
  bool ok;
  int shape, C, RPT, k, tiles, threads;
  double cycles;
  RTGeom W;
};

RTPlan rt_plan(const RTCost& cost, int X, int Y, int R, int nsteps, int k_req, int tile_x, int tile_y, int sms);

bool rt_heat_shape(const Geo& G, int ncomp, const PdeBCRules* rules);
RTPlan rt_heat_plan(const Geo& G, int nsteps, int k_req, int tile_x, int tile_y);
int rt_heat_run(const RTPlan& L, const float* u_in, float* u_out, float* work, const Geo& G, const Weights& W,
                const PdeBCRules& rules, float alpha, float dt, int nsteps, double t0, double tstep, int n0,
                cudaStream_t st);

}  // namespace pde
