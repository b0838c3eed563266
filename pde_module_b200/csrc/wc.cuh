// Weakly compressible flow, one RK2 (midpoint) step per launch (new: the
// reference composes the step from ~40 module launches, examples/LDC/LDC_RK2.py).
//
// Fields: momentum m (X, Y, 1, 2) and density rho (X, Y, 1, 1).  With the
// reference's operators (every product and sum rounded on its own, in their order):
//
//   bc(m, rho):  u = m / rho;  u = BC_u(u);  rho = BC_rho(rho);  m = rho * u
//   f(m, rho):   u = m / rho
//                m_div  = Div(m, -1)                        (divergence.py, vec -> scalar)
//                u_diff = Lap(u, nu)
//                u_conv = Div(outer(m, u), 1)               (elementWiseOps.py, divergence of a matrix)
//                u_damp = Lap(u_diff, eps)                  (biharmonic damping)
//                dp     = Grad(c2 * (rho - rho0), -1)
//                k_m    = ((dp - u_conv) + u_diff) + u_damp;  k_rho = m_div
//   step (time_step/rungeKatta.py:123-174):
//                y0 = bc(y);  y1 = bc(y0 + (dt/2) f(y0));  y' = y0 + dt f(y1)
//
// The operators' outputs are 0 outside the array interior (their launch domain),
// so f is 0 on ghost cells and y' keeps y0's boundary-filled ghosts there.
// A block owns a tile and works on the tile grown by 4 cells (clipped to the
// array) in shared memory: each f consumes 2 cells of the region's cut edges
// (Lap of Lap), the boundary fills read inward only, so the tile's result is exact.
#pragma once
#include "common.cuh"
#include "fused.cuh"

namespace pde {

struct WCParams {
  int X, Y, g;
  int TBX, TBY, tiles_y, RC;  // tile, tiles along Y, region capacity (cells)
  float wl[3];                // Laplacian weights (1, -2, 1) / dx^2
  float wd[3];                // first-derivative weights (-1, 0, 1) / (2 dx)
  float nu, eps, c2, rho0;
  float dt_half, dt;          // fp32 of dt/2 and of dt, each rounded from the caller's double
};

constexpr int WC_HALO = 4;

template <class F>
__device__ __forceinline__ void wc_region(int RC, int RY, F fn) {
  RectWalk wk(RY, (int)blockDim.x);
  for (int i = threadIdx.x; i < RC; i += blockDim.x, wk.next()) fn(i, wk.row, wk.col);
}

// Boundary fill of velocity and density together: the ghosts of both, barrier, the
// nodes of both, barrier (the order of bc_fill_planned for each).
template <int E>
__device__ __forceinline__ void wc_fill(float2* U, float* Rh, const BcPlan<E>& pl, const H2Params& hp,
                                        const PdeBCRules& Ru, const PdeBCRules& Rr, int rx0, int RX, int ry0, int RY) {
  float* Uf = reinterpret_cast<float*>(U);
  if (pl.mode == 2) {
    bc_fill_region<2, 2>(Uf, hp, Ru, rx0, RX, ry0, RY, Ru.dx32);
    bc_fill_region<1, 1>(Rh, hp, Rr, rx0, RX, ry0, RY, Rr.dx32);
    return;
  }
#pragma unroll
  for (int i = 0; i < E; ++i) {
    if (pl.gh[i] == ~0u) continue;
    const int dst = (int)(pl.gh[i] & 0xffffu), src = (int)(pl.gh[i] >> 16);
    const int K = pl.gm[i] & 31, ax = (pl.gm[i] >> 5) & 1, inc = ((pl.gm[i] >> 6) & 1) ? 1 : -1;
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int gi = Ru.ghost_group[K][ax][v];
      if (gi >= 0) Uf[dst * 2 + v] = ghost_value(Ru, gi, inc, Uf[src * 2 + v], Ru.dx32);
    }
    const int gi = Rr.ghost_group[K][ax][0];
    if (gi >= 0) Rh[dst] = ghost_value(Rr, gi, inc, Rh[src], Rr.dx32);
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < E; ++i) {
    if (pl.nd[i] == ~0u) continue;
    const int dst = (int)(pl.nd[i] & 0xffffu), K = (int)(pl.nd[i] >> 16);
    const int gu = Ru.node_group[K], gr = Rr.node_group[K];
    if (gu >= 0) {
#pragma unroll
      for (int v = 0; v < 2; ++v)
        if ((Ru.group[gu].comp_mask >> v) & 1u) Uf[dst * 2 + v] = Ru.group[gu].value;
    }
    if (gr >= 0 && (Rr.group[gr].comp_mask & 1u)) Rh[dst] = Rr.group[gr].value;
  }
  __syncthreads();
}

// Cell-wise arithmetic on both components, each rounded on its own.
__device__ __forceinline__ float2 wc_mul(float s, float2 a) { return make_float2(mul(s, a.x), mul(s, a.y)); }
__device__ __forceinline__ float2 wc_add(float2 a, float2 b) { return make_float2(add(a.x, b.x), add(a.y, b.y)); }
__device__ __forceinline__ float2 wc_div(float2 a, float s) { return make_float2(__fdiv_rn(a.x, s), __fdiv_rn(a.y, s)); }

// Phases of a stage: u of a cell, the fill of an edge tile, (rho u, u) of a cell,
// Lap(u), f.  Where there is nothing to fill the phases before and after the fill are
// one, so an interior tile meets five barriers a step and an edge tile eleven (14 and
// 22 when every operator was its own phase).  Both components of a vector move in one
// 8-byte access: a cell's f takes 19 shared-memory loads instead of 34 with two-way
// bank conflicts.  Latency bounds a step on small grids (201^2 nodes, calls of 100 steps:
// 10.2 -> 6.5 us a step), the loads and the arithmetic on large ones (1025^2: 73.7 ->
// 61.7 us).  An array
// of its own for y1's velocity saves one more barrier but 1.5% only, and costs a block
// per SM.
// WC_REGS: 3 blocks of 512 threads per SM.
constexpr int WC_THREADS = 640;
constexpr int WC_REGS = 40;

__global__ void __maxnreg__(WC_REGS) wc_rk2_kernel(const float* m_in, const float* r_in, float* m_out, float* r_out,
                                                   const WCParams P, const __grid_constant__ PdeBCRules Ru,
                                                   const __grid_constant__ PdeBCRules Rr) {
  extern __shared__ __align__(16) float sm[];
  const int X = P.X, Y = P.Y, g = P.g;
  const int tx = blockIdx.x / P.tiles_y, ty = blockIdx.x % P.tiles_y;
  const int bx0 = tx * P.TBX, by0 = ty * P.TBY;
  const int rx0 = max(bx0 - WC_HALO, 0), rx1 = min(bx0 + P.TBX + WC_HALO, X);
  const int ry0 = max(by0 - WC_HALO, 0), ry1 = min(by0 + P.TBY + WC_HALO, Y);
  const int RX = rx1 - rx0, RY = ry1 - ry0, RC = RX * RY;
  float2* M0 = reinterpret_cast<float2*>(sm);  // y0: momentum, density
  float2* U = M0 + P.RC;                       // velocity (of y0, then of y1)
  float2* D = U + P.RC;                        // Lap(u, nu)
  float2* M1 = D + P.RC;                       // y1
  float* R0 = reinterpret_cast<float*>(M1 + P.RC);
  float* R1 = R0 + P.RC;
  H2Params hp;  // the boundary fill reads the array shape and ghost width only
  hp.X = X;
  hp.Y = Y;
  hp.g = g;
  BcPlan<2> bp;  // one region for both fields and both fills
  bc_plan(bp, hp, rx0, RX, ry0, RY);
  const bool fill = bp.mode != 0;  // the same for the whole block
  const float* wl = P.wl;
  const float* wd = P.wd;

  // inside the array's interior, with all neighbours in the region
  auto active = [&](int lx, int ly) {
    const int x = rx0 + lx, y = ry0 + ly;
    return x >= g && x < X - g && y >= g && y < Y - g && lx >= 1 && lx < RX - 1 && ly >= 1 && ly < RY - 1;
  };
  // m = rho u, and u = m / rho as f forms it
  auto after = [&](float2* M, float2* V, int i, float2 u, float rh) {
    const float2 m = wc_mul(rh, u);
    M[i] = m;
    V[i] = wc_div(m, rh);
  };
  // a state's cell: its velocity goes to the fill, or straight on
  auto before = [&](float2* M, float2* V, float* Rh, int i, float2 m, float rh) {
    Rh[i] = rh;
    const float2 u = wc_div(m, rh);
    if (fill) V[i] = u;
    else after(M, V, i, u, rh);
  };
  auto fill_phase = [&](float2* M, float2* V, float* Rh) {
    if (!fill) return;
    wc_fill(V, Rh, bp, hp, Ru, Rr, rx0, RX, ry0, RY);
    for (int i = threadIdx.x; i < RC; i += blockDim.x) after(M, V, i, V[i], Rh[i]);
    __syncthreads();
  };
  // weighted sum over axes and taps, in the operators' order
  auto lap = [&](const float2* A, int i) {
    float2 acc = make_float2(0.0f, 0.0f);
    const float2 c = A[i];
    acc = wc_add(acc, wc_mul(wl[0], A[i - RY]));
    acc = wc_add(acc, wc_mul(wl[1], c));
    acc = wc_add(acc, wc_mul(wl[2], A[i + RY]));
    acc = wc_add(acc, wc_mul(wl[0], A[i - 1]));
    acc = wc_add(acc, wc_mul(wl[1], c));
    acc = wc_add(acc, wc_mul(wl[2], A[i + 1]));
    return acc;
  };
  // D = Lap(u, nu)
  auto lap_phase = [&](const float2* V) {
    wc_region(RC, RY, [&](int i, int lx, int ly) {
      D[i] = active(lx, ly) ? wc_mul(P.nu, lap(V, i)) : make_float2(0.0f, 0.0f);
    });
    __syncthreads();
  };
  // f at region cell i of (M, Rh) (velocity V and D prepared): (k_m, k_rho)
  auto f_at = [&](const float2* M, const float2* V, const float* Rh, int i, float2& km, float& kr) {
    float div = 0.0f;                       // m_div = Div(m, -1)
    float2 conv = make_float2(0.0f, 0.0f);  // u_conv[v] = sum over axes a, taps of w * (m_v u_a)
    float gp[2];                            // Grad(c2 * (rho - rho0)) along each axis
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      float s = 0.0f;
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        const int j = i + (t - 1) * (a == 0 ? RY : 1);
        const float2 m = M[j], u = V[j];
        div = add(div, mul(wd[t], a == 0 ? m.x : m.y));
        conv = wc_add(conv, wc_mul(wd[t], wc_mul(a == 0 ? u.x : u.y, m)));
        s = add(s, mul(wd[t], mul(P.c2, sub(Rh[j], P.rho0))));
      }
      gp[a] = s;
    }
    kr = mul(-1.0f, div);
    const float2 damp = wc_mul(P.eps, lap(D, i)), diff = D[i];
    km.x = add(add(sub(mul(-1.0f, gp[0]), conv.x), diff.x), damp.x);
    km.y = add(add(sub(mul(-1.0f, gp[1]), conv.y), diff.y), damp.y);
  };

  // The previous step is complete before its output is read; only then may the next
  // step's blocks start (their plans overlap this step), so no block can hold cached
  // lines of a buffer that an earlier step still writes.
  pdl_wait();
  pdl_launch_dependents();
  // ---- stage 1: y0 = bc(y); y1 = y0 + dt/2 f(y0) ----
  wc_region(RC, RY, [&](int i, int lx, int ly) {
    const size_t c = (size_t)(rx0 + lx) * Y + ry0 + ly;
    before(M0, U, R0, i, make_float2(m_in[2 * c], m_in[2 * c + 1]), r_in[c]);
  });
  __syncthreads();
  fill_phase(M0, U, R0);
  lap_phase(U);
  wc_region(RC, RY, [&](int i, int lx, int ly) {
    float2 km = make_float2(0.0f, 0.0f);
    float kr = 0.0f;
    if (active(lx, ly)) f_at(M0, U, R0, i, km, kr);
    M1[i] = wc_add(M0[i], wc_mul(P.dt_half, km));
    R1[i] = add(R0[i], mul(P.dt_half, kr));
  });
  __syncthreads();  // every f is formed: U may be overwritten
  // ---- stage 2: y' = y0 + dt f(bc(y1)) on the tile ----
  for (int i = threadIdx.x; i < RC; i += blockDim.x) before(M1, U, R1, i, M1[i], R1[i]);
  __syncthreads();
  fill_phase(M1, U, R1);
  lap_phase(U);
  const int ox1 = min(bx0 + P.TBX, X), oy1 = min(by0 + P.TBY, Y);
  const int OY = oy1 - by0, OC = (ox1 - bx0) * OY;
  RectWalk wo(OY, (int)blockDim.x);
  for (int o = threadIdx.x; o < OC; o += blockDim.x, wo.next()) {
    const int i = (bx0 - rx0 + wo.row) * RY + by0 - ry0 + wo.col;
    const int x = bx0 + wo.row, y = by0 + wo.col;
    float2 km = make_float2(0.0f, 0.0f);
    float kr = 0.0f;
    // tile cells are 4 cells from any cut
    if (x >= g && x < X - g && y >= g && y < Y - g) f_at(M1, U, R1, i, km, kr);
    const size_t c = (size_t)x * Y + y;
    const float2 m = wc_add(M0[i], wc_mul(P.dt, km));
    m_out[2 * c] = m.x;  // the caller's array is 4-byte aligned
    m_out[2 * c + 1] = m.y;
    r_out[c] = add(R0[i], mul(P.dt, kr));
  }
}

}  // namespace pde
