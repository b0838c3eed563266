// The differentiable 2D heat rollout of order 2 on register tiles: the forward with a
// diffusivity field and its adjoint (heat_adj.cuh states the scheme and the order of
// operations).  Tiles cover the stencil box.  In the adjoint the transposed boundary
// fill stays inside a thread: a ghost's mu is its lambda plus the weighted z of the
// node next to it, and folds into the partner one cell further in, all three in the
// same thread's rows or columns; the fill leaves every ghost's lambda 0, so only the
// first step of a pass has any.  256^2 x 1000 steps, forward and gradients, on one
// B200: 4.57 -> 1.82 ms against the shared-memory regions (five to nine words read a
// cell and step, up to four barriers); bound by issue and by the launch and the window
// loads of a pass.
#pragma once
#include "regtile.cuh"

namespace pde {

struct RGParams {
  RTGeom W;
  int X, Y, g;
  int k;
  float w[2];          // Laplacian weights: neighbour, centre
  float dt, negzero;
  const float* alpha;
  const float* in;
  float* out;
  float* lst;          // forward, if set: S of step s at lst + s * X * Y
  const float* lsts;   // adjoint: S of the pass's first (highest) step; the next ones X * Y before
  float* galpha;       // adjoint: dJ/dalpha, accumulated in place
  double t0, tstep;    // forward ramps
  int n0;
};

template <int C, int RPT>
__global__ void __launch_bounds__(RT_WARPS * 32) heat2d_field_rt_kernel(const RGParams P, const PdeBCRules Rl) {
  constexpr int HP = RPT / 2;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float rows[];
  __shared__ RTBc T;
  __shared__ PdeBCRules SR;  // ramps: the rules with the current step's group values
  const RTView<C, RPT> V(P.W, blockIdx.x);
  const int tid = (int)threadIdx.x, nt = (int)blockDim.x;
  if (Rl.has_ramp) {
    if (tid == 0) SR = Rl;
  } else {
    for (int i = tid; i < 21; i += nt) rt_bc_entry(T, Rl, Rl.dx32, i);
  }
  __syncthreads();
  RTGhosts<C, RPT> gh;
  RTEdge E;
  if (!Rl.has_ramp) E.load(T, V);
  float* const own = rt_own_row<1, C>(rows, V.warp, V.lane);
  const int flip = (int)rt_buf_floats<1, C>(V.nw);
  const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
  const float2 nz = rt_pair(P.negzero), w0 = rt_pair(P.w[0]), w1 = rt_pair(P.w[1]), dt = rt_pair(P.dt);
  auto M = [&](float2 a, float2 b) { return __ffma2_rn(a, b, nz); };
  const size_t first = (size_t)(P.g + V.r0) * P.Y + P.g + V.c0, cells = (size_t)P.X * P.Y;
  pdl_wait();
  float2 u[HP][C], al[HP][C];
  rt_load<C, RPT>(u, P.in + first, P.Y, V.on);
  rt_load<C, RPT>(al, P.alpha + first, P.Y, V.on);
  int par = 0;
  auto run = [&](auto Yc) {
    constexpr int YE = decltype(Yc)::value;
    for (int reach = P.k - 1; reach >= 0; --reach) {
      const int s = P.k - 1 - reach;
      if (Rl.has_ramp) {
        // every read of the table in the previous step came before its barrier
        if (tid < Rl.ngroups && Rl.group[tid].func == PDE_BC_FUNC_RAMP) {
          const float t = step_time(P.t0, P.tstep, P.n0 + s);
          SR.group[tid].value = bc_value(PDE_BC_FUNC_RAMP, Rl.group[tid].value, Rl.group[tid].t_max, &t);
        }
        __syncthreads();
        for (int i = tid; i < 21; i += nt) rt_bc_entry(T, SR, Rl.dx32, i);
        __syncthreads();
        E.load(T, V);
      }
      const bool live = V.dist <= reach + 1;
      if (live) rt_bc_fill<YE, C, RPT>(u, V, E, gh);
      RTRows<C> e;
      rt_rows_put<C, RPT>(u, own + par, w0, nz, live, e);
      __syncthreads();
      if (V.dist <= reach) {
        float2 lap[HP][C];
        rt_rows_sum<YE, false, C, RPT>(u, V, own + par, w0, nz, e, gh, [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
          const float2 mid = M(w1, u[i][j]);
          float2 acc = __fadd2_rn(a, mid);
          acc = __fadd2_rn(acc, b);
          acc = __fadd2_rn(acc, l);
          acc = __fadd2_rn(acc, mid);
          acc = __fadd2_rn(acc, r);
          lap[i][j] = acc;
          u[i][j] = __fadd2_rn(u[i][j], M(dt, M(al[i][j], acc)));
        });
        if (P.lst) rt_store<C, RPT>(lap, P.lst + first + (size_t)s * cells, P.Y, V);
      }
      par = flip - par;
    }
  };
  if (ye == 0) run(std::integral_constant<int, 0>{});
  else if (ye == 1) run(std::integral_constant<int, 1>{});
  else if (ye == 2) run(std::integral_constant<int, 2>{});
  else run(std::integral_constant<int, 3>{});
  rt_store_all<C, RPT>(u, gh, V, P.out + first, P.Y);
  rt_copy_outer(P.in, P.out, P.X, P.Y, P.g, 0, P.X);
}

// The adjoint step's boundary roles of a thread: how a ghost's mu folds into its
// partner (+1, -1: the ghost's coefficient of its partner; every face is filled) and
// which nodes the fill overwrites, for first, middle and last row (at a y edge) and
// column (at an x edge).
struct RTFold {
  float rf, rm, rl, cf, cm, cl;
  bool nrf, nrm, nrl, ncf, ncm, ncl;
  template <int C, int RPT>
  __device__ __forceinline__ void load(const RTBc& T, const RTView<C, RPT>& V) {
    RTEdge E;
    E.load(T, V);
    rf = E.rf.x; rm = E.rm.x; rl = E.rl.x;
    cf = E.cf.x; cm = E.cm.x; cl = E.cl.x;
    nrf = E.nrf; nrm = E.nrm; nrl = E.nrl;
    ncf = E.ncf; ncm = E.ncm; ncl = E.ncl;
  }
};

__global__ void __launch_bounds__(RT_WARPS * 32) heat2d_adj_rt_kernel(const RGParams P, const PdeBCRules Rl) {
  constexpr int C = 2, RPT = 4, HP = RPT / 2;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float rows[];
  __shared__ RTBc T;
  const RTView<C, RPT> V(P.W, blockIdx.x);
  const int tid = (int)threadIdx.x;
  for (int i = tid; i < 21; i += (int)blockDim.x) rt_bc_entry(T, Rl, Rl.dx32, i);
  __syncthreads();
  RTFold B;
  B.load(T, V);
  float* const own = rt_own_row<1, C>(rows, V.warp, V.lane);
  const int flip = (int)rt_buf_floats<1, C>(V.nw);
  const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
  const float2 nz = rt_pair(P.negzero), w0 = rt_pair(P.w[0]), w1 = rt_pair(P.w[1]), dt = rt_pair(P.dt);
  auto M = [&](float2 a, float2 b) { return __ffma2_rn(a, b, nz); };
  const size_t first = (size_t)(P.g + V.r0) * P.Y + P.g + V.c0, cells = (size_t)P.X * P.Y;
  bool in[C];
#pragma unroll
  for (int j = 0; j < C; ++j) in[j] = V.col_in(j);
  pdl_wait();
  float2 lam[HP][C], al[HP][C], ga[HP][C], sv[HP][C];
  rt_load<C, RPT>(lam, P.in + first, P.Y, V.on);
  rt_load<C, RPT>(al, P.alpha + first, P.Y, V.on);
  auto fetch = [&](float2 (&v)[HP][C], const float* p) {  // the tile's cells
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int j = 0; j < C; ++j)
        if (V.row_in(r) && in[j]) rt_at<C, RPT>(v, r, j) = p[(size_t)r * P.Y + j];
  };
#pragma unroll
  for (int i = 0; i < HP; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) ga[i][j] = sv[i][j] = rt_pair(0.0f);
  fetch(ga, P.galpha + first);
  const float* lsrc = P.lsts + first;
  fetch(sv, lsrc);
  // the ghosts' lambda as the pass begins (0 after its first step)
  float2 gcol[HP];
  float grow[C];
#pragma unroll
  for (int i = 0; i < HP; ++i) {
    const float* q = P.in + first + (V.llo ? -1 : C);
    gcol[i] = (V.llo || V.lhi) ? make_float2(q[(size_t)i * P.Y], q[(size_t)(i + HP) * P.Y]) : rt_pair(0.0f);
  }
#pragma unroll
  for (int j = 0; j < C; ++j) {
    const float* q = V.wlo ? P.in + first - P.Y : P.in + first + (size_t)RPT * P.Y;
    grow[j] = V.xe && V.on ? q[j] : 0.0f;
  }
  const RTGhosts<C, RPT> none{};  // not read: z is 0 beyond the box
  int par = 0;
  auto run = [&](auto Yc) {
    constexpr int YE = decltype(Yc)::value;
    for (int reach = P.k - 1; reach >= 0; --reach) {
      float2 z[HP][C];
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) z[i][j] = M(dt, M(al[i][j], lam[i][j]));
      RTRows<C> e;
      rt_rows_put<C, RPT>(z, own + par, w0, nz, V.dist <= reach + 1, e);
      __syncthreads();
      if (V.dist <= reach) {
#pragma unroll
        for (int i = 0; i < HP; ++i)
#pragma unroll
          for (int j = 0; j < C; ++j) ga[i][j] = __fadd2_rn(ga[i][j], M(lam[i][j], M(dt, sv[i][j])));
        if (reach > 0) fetch(sv, lsrc - (size_t)(P.k - reach) * cells);
        // mu, over lambda
        rt_rows_sum<YE, true, C, RPT>(z, V, own + par, w0, nz, e, none, [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
          const float2 mid = M(w1, z[i][j]);
          float2 acc = __fadd2_rn(a, mid);
          acc = __fadd2_rn(acc, b);
          acc = __fadd2_rn(acc, l);
          acc = __fadd2_rn(acc, mid);
          acc = __fadd2_rn(acc, r);
          lam[i][j] = __fadd2_rn(lam[i][j], acc);
        });
        // the transposed fill: overwritten nodes to 0, then the ghosts' mu into their
        // partners, x before y; the ghosts' lambda becomes 0
        if (V.xe) {
#pragma unroll
          for (int j = 0; j < C; ++j) {
            const bool n = j == 0 ? B.ncf : B.ncl;
            rt_at<C, RPT>(lam, 0, j) = V.wlo && n ? 0.0f : rt_at<C, RPT>(lam, 0, j);
            rt_at<C, RPT>(lam, RPT - 1, j) = V.whi && n ? 0.0f : rt_at<C, RPT>(lam, RPT - 1, j);
          }
        }
        if constexpr (YE != 0) {
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            const bool n = r == 0 ? B.nrf : r == RPT - 1 ? B.nrl : B.nrm;
            if constexpr ((YE & 1) != 0) rt_at<C, RPT>(lam, r, 0) = V.llo && n ? 0.0f : rt_at<C, RPT>(lam, r, 0);
            if constexpr ((YE & 2) != 0)
              rt_at<C, RPT>(lam, r, C - 1) = V.lhi && n ? 0.0f : rt_at<C, RPT>(lam, r, C - 1);
          }
        }
        if (V.xe) {
#pragma unroll
          for (int j = 0; j < C; ++j) {
            const float m = add(grow[j], V.wlo ? e.first[j].x : e.last[j].y);
            const float c = j == 0 ? B.cf : B.cl;
            float& lo = rt_at<C, RPT>(lam, 1, j);
            float& hi = rt_at<C, RPT>(lam, RPT - 2, j);
            lo = V.wlo ? fmaf(c, m, lo) : lo;  // c is +-1: one rounding
            hi = V.whi ? fmaf(c, m, hi) : hi;
            grow[j] = 0.0f;
          }
        }
        if constexpr (YE != 0) {
#pragma unroll
          for (int i = 0; i < HP; ++i) {
            const float2 node = YE == 1 ? z[i][0] : YE == 2 ? z[i][C - 1] : rt_sel(V.lhi, z[i][C - 1], z[i][0]);
            const float2 m = __fadd2_rn(gcol[i], M(w0, node));
            const float2 c = make_float2(i == 0 ? B.rf : B.rm, i == HP - 1 ? B.rl : B.rm);
            if constexpr ((YE & 1) != 0) lam[i][1] = rt_sel(V.llo, __ffma2_rn(c, m, lam[i][1]), lam[i][1]);
            if constexpr ((YE & 2) != 0) lam[i][C - 2] = rt_sel(V.lhi, __ffma2_rn(c, m, lam[i][C - 2]), lam[i][C - 2]);
            gcol[i] = rt_pair(0.0f);
          }
        }
      }
      par = flip - par;
    }
  };
  if (ye == 0) run(std::integral_constant<int, 0>{});
  else if (ye == 1) run(std::integral_constant<int, 1>{});
  else if (ye == 2) run(std::integral_constant<int, 2>{});
  else run(std::integral_constant<int, 3>{});
  rt_store<C, RPT>(ga, P.galpha + first, P.Y, V);
  RTGhosts<C, RPT> zero;
#pragma unroll
  for (int i = 0; i < HP; ++i) zero.col[i] = rt_pair(0.0f);
#pragma unroll
  for (int j = 0; j < C; ++j) zero.row[j] = 0.0f;
  rt_store_all<C, RPT>(lam, zero, V, P.out + first, P.Y);
  rt_copy_outer(P.in, P.out, P.X, P.Y, P.g, 0, P.X);
}

}  // namespace pde
