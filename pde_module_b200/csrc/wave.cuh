// Differentiable 2D wave equation (new: the reference's wave examples step a
// first-order (u, v) pair with forward Euler, tests/FDM/test_WaveStanding.py:71-76).
//
// State on the cells strictly inside the Dirichlet node ring (x, y in
// [g+1, n-g-2]); nodes and ghosts stay 0.  With K = dt^2 c^2 (a field) and L the
// reference's 5-point Laplacian (FDM/kernel/laplacian.py:40-46 order, alpha 1):
//
//   forward  u^{n+1} = 2 u^n - u^{n-1} + K o L(u^n) + s^n e_src
//   adjoint  mu^n    = 2 mu^{n+1} - mu^{n+2} + L(K o mu^{n+1})      (mu^{N+1} = 0)
//   gradient dJ/dK  += mu^{n+1} o L(u^n)      for n = N-1 .. 0, one add per step
//
// Both directions advance k steps per launch out of shared-memory tiles
// (halo k cells; cells outside the node ring are constant zeros, so only the
// region's cut edges lose one valid cell per step).  Regions are loaded with
// cp.async (every copy of a thread in flight at once; cells outside the ring
// zero-filled), and each step computes only the rectangle of cells that change.  Every product and sum is
// rounded on its own.  The forward can store L(u^n), the Laplacian it has just
// formed, for the adjoint's gradient term; the adjoint keeps K o mu in shared
// memory (each product formed once per cell and step, the same value every
// neighbour reads) and accumulates dJ/dK of its tile in shared memory, in the
// order n = N-1 .. 0, so the result does not depend on k or the tile.
#pragma once
#include <type_traits>

#include "common.cuh"

namespace pde {


struct WaveParams {
  int X, Y, g;
  int k;                 // steps in this pass
  int TBX, TBY, tiles_y;
  int RC;                // region capacity (cells)
  float w[3];            // Laplacian weights
  int srcx, srcy;        // source cell (forward), -1 for none
  const float* src;      // per-step source amplitude s^n (forward)
  int n0;                // forward: index n of u^n (the input "current" field)
  float* lst;            // forward: if set, L(u^{n0+s}) is stored at lst + s*cells
  long long cells;       // X*Y
  const float* lsts;     // adjoint: L(u^n) at lsts + n*cells
  int ntop;              // adjoint: the pass handles n = ntop, ntop-1, ..., ntop-k+1
  float* gK;             // adjoint: dJ/dK accumulated in place
};

__device__ __forceinline__ bool wave_inside(const WaveParams& P, int x, int y) {
  return x > P.g && x < P.X - 1 - P.g && y > P.g && y < P.Y - 1 - P.g;
}

// Region of a tile: the tile grown by the halo H, clipped to the array.
struct WaveRegion {
  int bx0, by0, rx0, ry0, RX, RY, OX, OY;
  __device__ WaveRegion(const WaveParams& P, int H) {
    const int tx = blockIdx.x / P.tiles_y, ty = blockIdx.x % P.tiles_y;
    bx0 = tx * P.TBX;
    by0 = ty * P.TBY;
    rx0 = max(bx0 - H, 0);
    ry0 = max(by0 - H, 0);
    RX = min(bx0 + P.TBX + H, P.X) - rx0;
    RY = min(by0 + P.TBY + H, P.Y) - ry0;
    OX = min(P.TBX, P.X - bx0);
    OY = min(P.TBY, P.Y - by0);
  }
};

// Rectangle of region cells a step computes: inside the node ring and one cell
// away from the region's edges (region indices [cx0, cx1) x [cy0, cy1)).  Cells
// outside the ring hold 0 in every buffer; region-edge cells are never
// rewritten, so their values go stale and, as cut edges do, invalidate one more
// cell inward per step.  Tile cells inside the ring are at least k cells from
// any cut edge, so they always lie in the rectangle.
struct WaveRect {
  int cx0, cy0, W, NR, count;  // NR rows of W cells
  __device__ WaveRect(const WaveParams& P, const WaveRegion& Rg) {
    cx0 = max(P.g + 1, Rg.rx0 + 1) - Rg.rx0;
    const int cx1 = min(P.X - 1 - P.g, Rg.rx0 + Rg.RX - 1) - Rg.rx0;
    cy0 = max(P.g + 1, Rg.ry0 + 1) - Rg.ry0;
    const int cy1 = min(P.Y - 1 - P.g, Rg.ry0 + Rg.RY - 1) - Rg.ry0;
    W = max(cy1 - cy0, 0);
    NR = max(cx1 - cx0, 0);
    count = NR * W;
  }
};

// Load a region row-major (RX x RY) with fn(region index, array x, array y).
template <class F>
__device__ __forceinline__ void for_region(const WaveRegion& Rg, F fn) {
  RectWalk wk(Rg.RY, (int)blockDim.x);
  for (int i = threadIdx.x; i < Rg.RX * Rg.RY; i += blockDim.x, wk.next()) fn(i, Rg.rx0 + wk.row, Rg.ry0 + wk.col);
}

// Tile cells (OX x OY) with fn(tile index, region index, global index).
template <class F>
__device__ __forceinline__ void for_tile(const WaveRegion& Rg, int Y, F fn) {
  RectWalk wk(Rg.OY, (int)blockDim.x);
  for (int t = threadIdx.x; t < Rg.OX * Rg.OY; t += blockDim.x, wk.next())
    fn(t, (Rg.bx0 - Rg.rx0 + wk.row) * Rg.RY + (Rg.by0 - Rg.ry0 + wk.col),
       (size_t)(Rg.bx0 + wk.row) * Y + Rg.by0 + wk.col);
}

// ---- shared-memory layout ---------------------------------------------------
// A region's cells are interleaved, NB floats per cell, so a cell's time levels
// and K sit at fixed offsets from one base: every access of a step is the cell's
// base plus a constant (neighbours: +-NB along y, +-NB*RY along x).  Leapfrog
// keeps two levels per field: step n overwrites u^{n-1}, which only its own cell
// reads, with u^{n+1}, so the two levels swap roles every step (parity
// p = s & 1) and the step loop runs two steps per iteration with p a
// compile-time constant.  The adjoint does the same with mu^{n+2} and keeps two
// levels of K o mu (its neighbours are read while the next level is written).
//   forward  (NB 3): 0, 1 levels of u (u^n in 1 - p, u^{n-1} in p), 2 K
//   adjoint  (NB 5): 0, 1 levels of mu (mu^{n+1} in 1 - p), 2, 3 levels of K o mu
//                    (K o mu^{n+1} in 3 - p), 4 K
//   paired   (NB 7): 0, 1 u; 2, 3 mu; 4, 5 K o mu; 6 K
// Laplacian (alpha 1) around the interleaved element c: rows rs floats apart,
// neighbours along y NB floats apart; the reference's term order.
template <int NB>
__device__ __forceinline__ float lap5n(const float* c, int rs, const float* w) {
  float acc = 0.0f;
  acc = add(acc, mul(w[0], c[-rs]));
  acc = add(acc, mul(w[1], c[0]));
  acc = add(acc, mul(w[2], c[rs]));
  acc = add(acc, mul(w[0], c[-NB]));
  acc = add(acc, mul(w[1], c[0]));
  acc = add(acc, mul(w[2], c[NB]));
  return acc;
}

__device__ __forceinline__ int wave_src_index(const WaveParams& P, const WaveRegion& Rg) {
  return (P.srcx >= 0 && P.srcx >= Rg.rx0 && P.srcx < Rg.rx0 + Rg.RX && P.srcy >= Rg.ry0 &&
          P.srcy < Rg.ry0 + Rg.RY)
             ? (P.srcx - Rg.rx0) * Rg.RY + (P.srcy - Rg.ry0)
             : -1;
}

// k forward steps: u^{n+1} = 2 u^n - u^{n-1} + K o L(u^n) (+ source), written over u^{n-1}.
template <bool STORE>
__device__ __forceinline__ void wave_fwd_steps(const WaveParams& P, const WaveRegion& Rg, float* sm) {
  constexpr int NB = 3;
  const int RY = Rg.RY, rs = NB * RY;
  const WaveRect Rt(P, Rg);
  const int srci = wave_src_index(P, Rg);
  // the tile in rectangle coordinates (for the stored Laplacians)
  const int nt = (int)blockDim.x;
  const int tx0 = Rg.bx0 - Rg.rx0 - Rt.cx0, ty0 = Rg.by0 - Rg.ry0 - Rt.cy0;
  for (int s = 0; s < P.k; ++s) {
    const int p = s & 1;
    const float sn = (srci >= 0) ? P.src[P.n0 + s] : 0.0f;
    float* Ls = STORE ? P.lst + (size_t)s * P.cells : nullptr;
    RectWalk wk(Rt.W, nt);
    for (int q = threadIdx.x; q < Rt.count; q += nt, wk.next()) {
      const int i = (Rt.cx0 + wk.row) * RY + Rt.cy0 + wk.col;
      float* pc = sm + NB * i;
      const float lap = lap5n<NB>(pc + (1 - p), rs, P.w);
      float v = sub(mul(2.0f, pc[1 - p]), pc[p]);
      v = add(v, mul(pc[2], lap));
      if (i == srci) v = add(v, sn);
      pc[p] = v;
      if (STORE) {
        const int ox = wk.row - tx0, oy = wk.col - ty0;
        if (ox >= 0 && ox < Rg.OX && oy >= 0 && oy < Rg.OY)
          Ls[(size_t)(Rg.bx0 + ox) * P.Y + Rg.by0 + oy] = lap;
      }
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(1024) wave_fwd_tb_kernel(const float* __restrict__ um_in,
                                                            const float* __restrict__ u0_in,
                                                            const float* __restrict__ Kf, float* __restrict__ um_out,
                                                            float* __restrict__ u0_out, const WaveParams P) {
  extern __shared__ __align__(16) float sm[];
  constexpr int NB = 3;
  const WaveRegion Rg(P, P.k);
  for_region(Rg, [&](int i, int x, int y) {
    const size_t gi = (size_t)x * P.Y + y;
    const bool in = wave_inside(P, x, y);  // the state is zero outside the node ring
    cp_async4(sm + NB * i, um_in + gi, in);
    cp_async4(sm + NB * i + 1, u0_in + gi, in);
    cp_async4(sm + NB * i + 2, Kf + gi, true);
  });
  cp_async_wait_all();
  __syncthreads();
  if (P.lst) wave_fwd_steps<true>(P, Rg, sm);
  else wave_fwd_steps<false>(P, Rg, sm);
  const int nw = (P.k & 1) ? 0 : 1;  // level the last step wrote
  for_tile(Rg, P.Y, [&](int t, int ri, size_t gi) {
    um_out[gi] = sm[NB * ri + (1 - nw)];
    u0_out[gi] = sm[NB * ri + nw];
  });
}

__global__ void __launch_bounds__(1024) wave_adj_tb_kernel(const float* __restrict__ m1_in,
                                                            const float* __restrict__ m2_in,
                                                            const float* __restrict__ Kf, float* __restrict__ m1_out,
                                                            float* __restrict__ m2_out, const WaveParams P) {
  extern __shared__ __align__(16) float sm[];
  constexpr int NB = 5;
  const WaveRegion Rg(P, P.k);
  const int RY = Rg.RY, rs = NB * RY;
  const int oga = NB * P.RC;  // dJ/dK of the tile
  for_region(Rg, [&](int i, int x, int y) {
    const size_t gi = (size_t)x * P.Y + y;
    const bool in = wave_inside(P, x, y);
    cp_async4(sm + NB * i, m2_in + gi, in);      // mu^{n+2}
    cp_async4(sm + NB * i + 1, m1_in + gi, in);  // mu^{n+1}
    cp_async4(sm + NB * i + 4, Kf + gi, true);
    sm[NB * i + 2] = 0.0f;
  });
  for_tile(Rg, P.Y, [&](int t, int ri, size_t gi) { cp_async4(sm + oga + t, P.gK + gi, true); });
  cp_async_wait_all();
  // K o mu^{n+1} of the cells this thread copied (its own copies are complete)
  for_region(Rg, [&](int i, int x, int y) { sm[NB * i + 3] = mul(sm[NB * i + 4], sm[NB * i + 1]); });
  __syncthreads();
  const WaveRect Rt(P, Rg);
  const int nt = (int)blockDim.x;
  const int tx0 = Rg.bx0 - Rg.rx0 - Rt.cx0, ty0 = Rg.by0 - Rg.ry0 - Rt.cy0;
  for (int s = 0; s < P.k; ++s) {
    const int p = s & 1;
    const float* Ln = P.lsts + (size_t)(P.ntop - s) * P.cells;
    RectWalk wk(Rt.W, nt);
    for (int q = threadIdx.x; q < Rt.count; q += nt, wk.next()) {
      const int i = (Rt.cx0 + wk.row) * RY + Rt.cy0 + wk.col;
      float* pc = sm + NB * i;
      const float m1 = pc[1 - p];
      {  // gradient term of step n on the tile: dJ/dK += mu^{n+1} o L(u^n)
        const int ox = wk.row - tx0, oy = wk.col - ty0;
        if (ox >= 0 && ox < Rg.OX && oy >= 0 && oy < Rg.OY) {
          const int t = oga + ox * Rg.OY + oy;
          sm[t] = add(sm[t], mul(m1, __ldg(Ln + (size_t)(Rg.bx0 + ox) * P.Y + Rg.by0 + oy)));
        }
      }
      // mu^n = 2 mu^{n+1} - mu^{n+2} + L(K o mu^{n+1})
      const float acc = lap5n<NB>(pc + (3 - p), rs, P.w);
      const float v = add(sub(mul(2.0f, m1), pc[p]), acc);
      pc[p] = v;
      pc[2 + p] = mul(pc[4], v);
    }
    __syncthreads();
  }
  for_tile(Rg, P.Y, [&](int t, int ri, size_t gi) { P.gK[gi] = sm[oga + t]; });
  const int nw = (P.k & 1) ? 0 : 1;  // level the last step wrote
  for_tile(Rg, P.Y, [&](int t, int ri, size_t gi) {
    m1_out[gi] = sm[NB * ri + nw];
    m2_out[gi] = sm[NB * ri + (1 - nw)];
  });
}

// ---- paired launch: forward recomputation beside the adjoint --------------
// One launch advances the same tile through up to k forward steps of one
// segment (storing L(u^n) of the tile, as wave_fwd_tb_kernel with lst set) and
// up to k adjoint steps of another segment (as wave_adj_tb_kernel).  The two
// are independent, so each warp interleaves two dependency chains and a step
// of both costs one barrier.  Arithmetic and per-cell operation order are
// those of the two kernels above.  Shared memory: the NB = 7 interleaved
// region, then the gradient tile. 
__global__ void __launch_bounds__(1024) wave_pair_tb_kernel(const float* __restrict__ um_in,
                                                             const float* __restrict__ u0_in,
                                                             float* __restrict__ um_out, float* __restrict__ u0_out,
                                                             const float* __restrict__ m1_in,
                                                             const float* __restrict__ m2_in,
                                                             float* __restrict__ m1_out, float* __restrict__ m2_out,
                                                             const float* __restrict__ Kf, const WaveParams Pf,
                                                             const WaveParams Pa) {
  extern __shared__ __align__(16) float sm[];
  constexpr int NB = 7;
  const int H = max(Pf.k, Pa.k);
  const WaveRegion Rg(Pa, H);  // Pf and Pa share the grid, tile and region capacity
  const int RY = Rg.RY, rs = NB * RY;
  const int oga = NB * Pa.RC;
  const bool fwd = Pf.k > 0, adj = Pa.k > 0;
  for_region(Rg, [&](int i, int x, int y) {
    const size_t gi = (size_t)x * Pa.Y + y;
    const bool in = wave_inside(Pa, x, y);  // the states are zero outside the node ring
    float* pc = sm + NB * i;
    cp_async4(pc + 6, Kf + gi, true);
    if (fwd) {
      cp_async4(pc, um_in + gi, in);
      cp_async4(pc + 1, u0_in + gi, in);
    }
    if (adj) {
      cp_async4(pc + 2, m2_in + gi, in);
      cp_async4(pc + 3, m1_in + gi, in);
      pc[4] = 0.0f;
    }
  });
  if (adj) for_tile(Rg, Pa.Y, [&](int t, int ri, size_t gi) { cp_async4(sm + oga + t, Pa.gK + gi, true); });
  cp_async_wait_all();
  if (adj) for_region(Rg, [&](int i, int x, int y) { sm[NB * i + 5] = mul(sm[NB * i + 6], sm[NB * i + 3]); });
  __syncthreads();
  const WaveRect Rt(Pa, Rg);
  const int srci = wave_src_index(Pf, Rg);
  const int nt = (int)blockDim.x;
  const int tx0 = Rg.bx0 - Rg.rx0 - Rt.cx0, ty0 = Rg.by0 - Rg.ry0 - Rt.cy0;
  for (int s = 0; s < H; ++s) {
    const int p = s & 1;
    const bool fs = s < Pf.k, as = s < Pa.k;
    const float sn = (fs && srci >= 0) ? Pf.src[Pf.n0 + s] : 0.0f;
    float* Ls = fs ? Pf.lst + (size_t)s * Pf.cells : nullptr;
    const float* Ln = as ? Pa.lsts + (size_t)(Pa.ntop - s) * Pa.cells : nullptr;
    RectWalk wk(Rt.W, nt);
    for (int q = threadIdx.x; q < Rt.count; q += nt, wk.next()) {
      const int i = (Rt.cx0 + wk.row) * RY + Rt.cy0 + wk.col;
      float* pc = sm + NB * i;
      const int ox = wk.row - tx0, oy = wk.col - ty0;
      const bool tile = ox >= 0 && ox < Rg.OX && oy >= 0 && oy < Rg.OY;
      if (fs) {  // u^{n+1} = 2 u^n - u^{n-1} + K o L(u^n) (+ source)
        const float lap = lap5n<NB>(pc + (1 - p), rs, Pf.w);
        float v = sub(mul(2.0f, pc[1 - p]), pc[p]);
        v = add(v, mul(pc[6], lap));
        if (i == srci) v = add(v, sn);
        pc[p] = v;
        if (tile) Ls[(size_t)(Rg.bx0 + ox) * Pf.Y + Rg.by0 + oy] = lap;
      }
      if (as) {
        const float m1 = pc[3 - p];
        if (tile) {  // dJ/dK += mu^{n+1} o L(u^n)
          const int t = oga + ox * Rg.OY + oy;
          sm[t] = add(sm[t], mul(m1, __ldg(Ln + (size_t)(Rg.bx0 + ox) * Pa.Y + Rg.by0 + oy)));
        }
        // mu^n = 2 mu^{n+1} - mu^{n+2} + L(K o mu^{n+1})
        const float acc = lap5n<NB>(pc + (5 - p), rs, Pa.w);
        const float v = add(sub(mul(2.0f, m1), pc[2 + p]), acc);
        pc[2 + p] = v;
        pc[4 + p] = mul(pc[6], v);
      }
    }
    __syncthreads();
  }
  if (adj) for_tile(Rg, Pa.Y, [&](int t, int ri, size_t gi) { Pa.gK[gi] = sm[oga + t]; });
  const int fw = (Pf.k & 1) ? 0 : 1, aw = (Pa.k & 1) ? 0 : 1;  // levels the last steps wrote
  for_tile(Rg, Pa.Y, [&](int t, int ri, size_t gi) {
    const float* pc = sm + NB * ri;
    if (fwd) {
      um_out[gi] = pc[1 - fw];
      u0_out[gi] = pc[fw];
    }
    if (adj) {
      m1_out[gi] = pc[2 + aw];
      m2_out[gi] = pc[3 - aw];
    }
  });
}

}  // namespace pde
