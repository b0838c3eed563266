// Fractional-step (projection) solver for the 2D lid-driven cavity, composed
// from the operators of the reference's LDC examples (examples/LDC/*.py:
// GridBoundary, Laplacian, Grad, Divergence, ForwardEuler) with a Jacobi
// pressure-Poisson sweep, which the reference does not have (it uses
// artificial compressibility).  Each kernel evaluates exactly the float32
// operations of that module composition, one rounding per product and sum:
//
//   u2   = BC_u(u)
//   u*   = u2 + dt * (nu*Lap(u2) - Grad(u2) u2)        (predictor)
//   rhs  = (1/dt) * Div(BC_u(u*))                        (divergence)
//   p    <- 0.25 * (pW + pE + pS + pN - dx^2 * rhs)      (Jacobi, p_bc = BC_p(p)), 50 sweeps
//   u    = BC_u(u*) + dt * (-Grad(BC_p(p)))              (projection)
#pragma once
#include <type_traits>

#include "common.cuh"
#include "fused.cuh"

namespace pde {

struct LdcConst {
  float wl[3];    // Laplacian weights
  float wd[3];    // first-derivative weights
  float nu, dt, inv_dt, h2;
};

// The predictor, divergence and projection work on shared-memory tiles: a block
// loads its tile grown by a halo (clipped to the rows held), fills the boundary
// there once (bc_fill_region), and every cell reads plain neighbours.  Evaluating
// the boundary-filled value per neighbour instead, one thread per cell on global
// memory, took 56 us a step for the three kernels on 1024^2 and 23 us on 100^2 (the
// chain of rule look-ups of a boundary cell); these take 25 and 11.5.  Row indices are those of the whole domain; a
// slab passes pointers shifted to them.
constexpr int LDC_TX = 16, LDC_TY = 64, LDC_THREADS = 256;

struct LdcRows {
  int X, Y, g;
  int own_lo, own_hi;    // rows written
  int held_lo, held_hi;  // rows that may be read
  bool pairs;            // the velocity arrays are 8-byte aligned
};

// Both components of a cell.
__device__ __forceinline__ float2 ldc_ld2(const float* p, size_t cell, bool pairs) {
  if (pairs) return reinterpret_cast<const float2*>(p)[cell];
  return make_float2(p[2 * cell], p[2 * cell + 1]);
}
__device__ __forceinline__ void ldc_st2(float* p, size_t cell, float2 v, bool pairs) {
  if (pairs) {
    reinterpret_cast<float2*>(p)[cell] = v;
  } else {
    p[2 * cell] = v.x;
    p[2 * cell + 1] = v.y;
  }
}

// Region accessor: N floats per cell, cells addressed by array indices.
template <int N>
struct Reg2 {
  const float* s;
  int rx0, ry0, RY;
  __device__ __forceinline__ float operator()(int i, int j, int v) const {
    return s[((i - rx0) * RY + (j - ry0)) * N + v];
  }
};

// A block's tile and region (tile + halo, within the array and the held rows).  A
// tile's ghosts are filled in its region from the cell two steps inward, so a tile that
// begins at the high ghosts, or ends at the low ones, takes two cells on that side
// whatever the halo: at most one more row and one more column than tile and halos.
__host__ __device__ constexpr int ldc_cap(int halo) {
  const int most = halo < 2 ? 2 : halo;
  return (LDC_TX + halo + most) * (LDC_TY + halo + most);
}
struct LdcTile {
  int bx0, by0, bx1, by1, rx0, ry0, RX, RY;
  __device__ LdcTile(const LdcRows& D, int halo) {
    bx0 = D.own_lo + (int)blockIdx.y * LDC_TX;
    by0 = (int)blockIdx.x * LDC_TY;
    bx1 = min(bx0 + LDC_TX, D.own_hi);
    by1 = min(by0 + LDC_TY, D.Y);
    const int most = max(halo, 2);
    rx0 = max(bx0 - (bx0 == D.X - D.g ? most : halo), D.held_lo);
    ry0 = max(by0 - (by0 == D.Y - D.g ? most : halo), 0);
    RX = min(bx1 + (bx1 == D.g ? most : halo), D.held_hi) - rx0;
    RY = min(by1 + (by1 == D.g ? most : halo), D.Y) - ry0;
  }
  // fn(region index, x, y) over the region's cells / the tile's cells
  template <class F>
  __device__ __forceinline__ void region(F fn) const {
    RectWalk wk(RY, LDC_THREADS);
    for (int i = threadIdx.x; i < RX * RY; i += LDC_THREADS, wk.next()) fn(i, rx0 + wk.row, ry0 + wk.col);
  }
  template <class F>
  __device__ __forceinline__ void tile(F fn) const {
    const int W = by1 - by0, n = (bx1 - bx0) * W;
    RectWalk wk(W, LDC_THREADS);
    for (int i = threadIdx.x; i < n; i += LDC_THREADS, wk.next()) fn(bx0 + wk.row, by0 + wk.col);
  }
};

__device__ __forceinline__ bool ldc_stencil(const LdcRows& D, int i, int j) {
  return i >= D.g && i < D.X - D.g && j >= D.g && j < D.Y - D.g;
}
__device__ __forceinline__ H2Params ldc_shape(const LdcRows& D) {
  H2Params H;
  H.X = D.X; H.Y = D.Y; H.g = D.g; H.N = 1;
  return H;
}

// Predictor of one stencil cell: u* = u2 + dt * (nu*Lap(u2) - Grad(u2) u2), with u2 = BC_u(u).
template <class Get>
__device__ __forceinline__ void ldc_predict_cell(const Get& at, int i, int j, const LdcConst& K, float* res) {
  const float uc[2] = {at(i, j, 0), at(i, j, 1)};
  float nb[2][2][3];  // [axis][comp][tap]
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    nb[0][c][1] = uc[c];
    nb[1][c][1] = uc[c];
    nb[0][c][0] = at(i - 1, j, c);
    nb[0][c][2] = at(i + 1, j, c);
    nb[1][c][0] = at(i, j - 1, c);
    nb[1][c][2] = at(i, j + 1, c);
  }
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float acc = 0.0f;  // Laplacian, FDM/kernel/laplacian.py:40-46 order
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int t = 0; t < 3; ++t) acc = add(acc, mul(K.wl[t], nb[a][c][t]));
    const float lap = mul(K.nu, acc);
    float gr[2];  // Grad(u2, 1.0): row c of the 2x2 matrix
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      float g = 0.0f;
#pragma unroll
      for (int t = 0; t < 3; ++t) g = add(g, mul(K.wd[t], nb[a][c][t]));
      gr[a] = mul(1.0f, g);
    }
    const float conv = add(mul(gr[0], uc[0]), mul(gr[1], uc[1]));
    res[c] = add(uc[c], mul(K.dt, sub(lap, conv)));
  }
}

// rhs = (1/dt) * Div(BC_u(u*)) on stencil cells (ghosts of rhs are never read).
template <class Get>
__device__ __forceinline__ float ldc_div_cell(const Get& at, int i, int j, const LdcConst& K) {
  float acc = 0.0f;  // FDM/kernel/divergence.py:85-106: axis 0 on component 0, axis 1 on component 1
#pragma unroll
  for (int t = 0; t < 3; ++t) acc = add(acc, mul(K.wd[t], at(i + t - 1, j, 0)));
#pragma unroll
  for (int t = 0; t < 3; ++t) acc = add(acc, mul(K.wd[t], at(i, j + t - 1, 1)));
  return mul(K.inv_dt, acc);
}

// PREDICT: u -> u*.  DIVERGE: u* -> rhs.  Both: u* of the tile and one cell around it
// stays in shared memory for the divergence (a slab runs them one by one: u* rows
// of the neighbouring slab come between).
template <bool PREDICT, bool DIVERGE>
__global__ void __launch_bounds__(LDC_THREADS) ldc_velocity_kernel(const float* u, float* us, float* rhs, const LdcRows D,
                                                                   const PdeBCRules Ru, const LdcConst K) {
  pdl_launch_dependents();
  constexpr int HALO = PREDICT && DIVERGE ? 2 : 1;
  constexpr int CAP = ldc_cap(HALO);
  __shared__ float2 A[PREDICT ? CAP : 1], B[DIVERGE ? CAP : 1];
  const LdcTile T(D, HALO);
  const H2Params HP = ldc_shape(D);
  pdl_wait();
  const float* src = PREDICT ? u : us;
  float2* first = PREDICT ? A : B;
  T.region([&](int i, int x, int y) { first[i] = ldc_ld2(src, (size_t)x * D.Y + y, D.pairs); });
  __syncthreads();
  if constexpr (PREDICT) {
    bc_fill_region<2>(reinterpret_cast<float*>(A), HP, Ru, T.rx0, T.RX, T.ry0, T.RY, Ru.dx32);
    __syncthreads();
    const Reg2<2> at{reinterpret_cast<const float*>(A), T.rx0, T.ry0, T.RY};
    auto value = [&](int x, int y) {
      float res[2] = {at(x, y, 0), at(x, y, 1)};
      if (ldc_stencil(D, x, y)) ldc_predict_cell(at, x, y, K, res);
      return make_float2(res[0], res[1]);
    };
    if constexpr (!DIVERGE) {
      T.tile([&](int x, int y) { ldc_st2(us, (size_t)x * D.Y + y, value(x, y), D.pairs); });
      return;
    } else {
      T.region([&](int i, int x, int y) {
        // the region's outer ring has no complete neighbourhood and is not read
        const bool ring = (x == T.rx0 && x > 0) || (x == T.rx0 + T.RX - 1 && x < D.X - 1) || (y == T.ry0 && y > 0) ||
                          (y == T.ry0 + T.RY - 1 && y < D.Y - 1);
        const float2 v = ring ? A[i] : value(x, y);
        B[i] = v;
        if (x >= T.bx0 && x < T.bx1 && y >= T.by0 && y < T.by1)
          ldc_st2(us, (size_t)x * D.Y + y, v, D.pairs);
      });
      __syncthreads();
    }
  }
  if constexpr (DIVERGE) {
    bc_fill_region<2>(reinterpret_cast<float*>(B), HP, Ru, T.rx0, T.RX, T.ry0, T.RY, Ru.dx32);
    __syncthreads();
    const Reg2<2> at{reinterpret_cast<const float*>(B), T.rx0, T.ry0, T.RY};
    T.tile([&](int x, int y) {
      rhs[(size_t)x * D.Y + y] = ldc_stencil(D, x, y) ? ldc_div_cell(at, x, y, K) : 0.0f;
    });
  }
}

// u = BC_u(u*) + dt * Grad(BC_p(p), -1)
template <class GetU, class GetP>
__device__ __forceinline__ void ldc_project_cell(const GetU& au, const GetP& ap, int i, int j, const LdcConst& K,
                                                 float* res) {
  const float a0 = au(i, j, 0), a1 = au(i, j, 1);
  float gx = 0.0f, gy = 0.0f;
#pragma unroll
  for (int t = 0; t < 3; ++t) gx = add(gx, mul(K.wd[t], ap(i + t - 1, j, 0)));
#pragma unroll
  for (int t = 0; t < 3; ++t) gy = add(gy, mul(K.wd[t], ap(i, j + t - 1, 0)));
  res[0] = add(a0, mul(K.dt, mul(-1.0f, gx)));
  res[1] = add(a1, mul(K.dt, mul(-1.0f, gy)));
}

__global__ void __launch_bounds__(LDC_THREADS) ldc_project_kernel(const float* us, const float* p, float* u,
                                                                   const LdcRows D, const PdeBCRules Ru,
                                                                   const PdeBCRules Rp, const LdcConst K) {
  pdl_launch_dependents();
  constexpr int CAP = ldc_cap(1);
  __shared__ float2 A[CAP];
  __shared__ float Pr[CAP];
  const LdcTile T(D, 1);
  const H2Params HP = ldc_shape(D);
  pdl_wait();
  T.region([&](int i, int x, int y) {
    const size_t c = (size_t)x * D.Y + y;
    A[i] = ldc_ld2(us, c, D.pairs);
    Pr[i] = p[c];
  });
  __syncthreads();
  bc_fill_region<2>(reinterpret_cast<float*>(A), HP, Ru, T.rx0, T.RX, T.ry0, T.RY, Ru.dx32);
  bc_fill_region<1>(Pr, HP, Rp, T.rx0, T.RX, T.ry0, T.RY, Rp.dx32);
  __syncthreads();
  const Reg2<2> au{reinterpret_cast<const float*>(A), T.rx0, T.ry0, T.RY};
  const Reg2<1> ap{Pr, T.rx0, T.ry0, T.RY};
  T.tile([&](int x, int y) {
    float res[2] = {au(x, y, 0), au(x, y, 1)};
    if (ldc_stencil(D, x, y)) ldc_project_cell(au, ap, x, y, K, res);
    ldc_st2(u, (size_t)x * D.Y + y, make_float2(res[0], res[1]), D.pairs);
  });
}

// k Jacobi sweeps per pass on shared-memory tiles (halo k + 1, as in
// heat2d_tb_kernel), Neumann ghosts refilled in shared memory every sweep.
// On the pass's last sweep the squared update of the tile's stencil cells is
// reduced (warp shuffles, then one atomic per block) into *resid.
struct J2Params {
  int X, Y, g;            // X: rows of the whole domain (a slab's arrays are addressed by global row)
  int own_lo, own_hi;     // rows whose results this launch writes
  int held_lo, held_hi;   // rows the arrays hold (owned rows plus halo rows on a slab's cut sides)
  int k;
  int TBX, TBY, tiles_y;
  int RXM, RYM;
  float h2;
  int last;  // this pass ends the step's sweeps: accumulate the residual
};

__global__ void __launch_bounds__(1024) jacobi2d_tb_kernel(const float* __restrict__ pin, float* __restrict__ pout,
                                                           const float* __restrict__ rhs, float* __restrict__ resid,
                                                           const J2Params P, const PdeBCRules Rp) {
  extern __shared__ __align__(16) float sm[];
  const int tx = blockIdx.x / P.tiles_y, ty = blockIdx.x % P.tiles_y;
  const int bx0 = P.own_lo + tx * P.TBX, by0 = ty * P.TBY;
  const int H = P.k + 1;
  const int rx0 = max(bx0 - H, P.held_lo), rx1 = min(bx0 + P.TBX + H, P.held_hi);
  const int ry0 = max(by0 - H, 0), ry1 = min(by0 + P.TBY + H, P.Y);
  const int RX = rx1 - rx0, RY = ry1 - ry0, RC = RX * RY;
  const int cap = P.RXM * P.RYM;
  float* A = sm;
  float* B = sm + cap;
  float* Rh = sm + 2 * cap;
  const int nt = (int)blockDim.x;
  // Both level buffers start with the region (cp.async, every copy of a thread
  // in flight at once); a sweep writes only its stencil rectangle, so the other
  // cells keep their loaded or last boundary-filled value.
  {
    RectWalk wk(RY, nt);
    for (int i = threadIdx.x; i < RC; i += nt, wk.next()) {
      const size_t gi = (size_t)(rx0 + wk.row) * P.Y + ry0 + wk.col;
      cp_async4(A + i, pin + gi, true);
      cp_async4(B + i, pin + gi, true);
      cp_async4(Rh + i, rhs + gi, true);
    }
  }
  cp_async_wait_all();
  __syncthreads();
  H2Params HP;
  HP.X = P.X; HP.Y = P.Y; HP.g = P.g; HP.N = 1;
  const int g = P.g;
  // stencil rectangle: cells of [g, n-g) whose four neighbours are inside the region
  const int sx0 = max(g, rx0 + 1) - rx0, sx1 = min(P.X - g, rx0 + RX - 1) - rx0;
  const int sy0 = max(g, ry0 + 1) - ry0, sy1 = min(P.Y - g, ry0 + RY - 1) - ry0;
  const int tw = min(bx0 + P.TBX, P.own_hi) - bx0, th = min(by0 + P.TBY, P.Y) - by0;
  float sq = 0.0f;
  for (int s = 0; s < P.k; ++s) {
    bc_fill_region<1>(A, HP, Rp, rx0, RX, ry0, RY, Rp.dx32);
    const bool acc_res = P.last && s == P.k - 1;
    // Sweep s only has to update the stencil cells within (k - 1 - s) + 1 of the
    // tile (the boundary fills read inward): the stencil rectangle cut to that box.
    const int reach = P.k - s;
    const int qx0 = max(sx0, bx0 - rx0 - reach), qx1 = min(sx1, bx0 - rx0 + tw + reach);
    const int qy0 = max(sy0, by0 - ry0 - reach), qy1 = min(sy1, by0 - ry0 + th + reach);
    const int SW = max(qy1 - qy0, 1), SC = max(qx1 - qx0, 0) * max(qy1 - qy0, 0);
    const int dq = nt / SW, dr = nt - dq * SW;
    // the tile in box coordinates (residual cells)
    const int tx0 = bx0 - rx0 - qx0, ty0 = by0 - ry0 - qy0;
    int lx = (int)threadIdx.x / SW, ly = (int)threadIdx.x - lx * SW;
    for (int c = threadIdx.x; c < SC; c += nt) {
      const int i = (qx0 + lx) * RY + qy0 + ly;
      const float old = A[i];
      const float sum = add(add(add(A[i - RY], A[i + RY]), A[i - 1]), A[i + 1]);
      const float res = mul(0.25f, sub(sum, mul(P.h2, Rh[i])));
      B[i] = res;
      if (acc_res) {
        const int ox = lx - tx0, oy = ly - ty0;
        if (ox >= 0 && ox < tw && oy >= 0 && oy < th) {
          const float d = res - old;
          sq = fmaf(d, d, sq);
        }
      }
      lx += dq;
      ly += dr;
      if (ly >= SW) { ly -= SW; ++lx; }
    }
    __syncthreads();
    float* t = A;
    A = B;
    B = t;
  }
  // output: stencil cells from the newest level, the others as last filled (B)
  RectWalk wo(th, nt);
  for (int i = threadIdx.x; i < tw * th; i += nt, wo.next()) {
    const int x = bx0 + wo.row, y = by0 + wo.col;
    const int ri = (x - rx0) * RY + (y - ry0);
    const bool st = x >= g && x < P.X - g && y >= g && y < P.Y - g;
    pout[(size_t)x * P.Y + y] = st ? A[ri] : B[ri];  // (equal when k = 0: both hold the loaded values)
  }
  if (P.last && resid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    __shared__ float wsum[32];
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      float b = 0.0f;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) b += wsum[w];
      atomicAdd(resid, b);
    }
  }
}

}  // namespace pde
