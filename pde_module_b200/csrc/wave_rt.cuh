// The differentiable 2D wave on register tiles: the leapfrog forward, its discrete
// adjoint, and both in one launch (wave.cuh states the scheme and the order of
// operations).  Against the interleaved shared-memory regions (three to seven words a
// cell, read five times a step), 512^2 x 2000 steps on one B200: forward 2.3 -> 1.3
// ms, recomputation and adjoint 4.2 -> 3.6 ms.  Bound by the latency of a step (37-43% of
// the issue slots used) and by what a pass spends besides its steps (launch, loading and
// storing seven fields' windows); the forward takes up to 16 steps a pass, both together
// 8.  Tiles cover the cells inside the node ring, outside of which every state is 0.
#pragma once
#include "regtile.cuh"

namespace pde {

struct RWParams {
  RTGeom W;
  int X, Y, pad;        // array extents; cells before the box (g + 1)
  float w[2];           // Laplacian weights: neighbour, centre
  float negzero;
  const float* K;
  // forward: kf steps from (um, u0) = (u^{n-1}, u^n)
  int kf;
  const float* um_in;
  const float* u0_in;
  float* um_out;
  float* u0_out;
  float* lst;           // if set: L(u^n) of step s at lst + s * X * Y
  int srcx, srcy;       // source cell (box coordinates), -1: none
  const float* src;     // its amplitude per step, from this pass's first
  // adjoint: ka steps from (m1, m2) = (mu^{n+1}, mu^{n+2})
  int ka;
  const float* m1_in;
  const float* m2_in;
  float* m1_out;
  float* m2_out;
  const float* lsts;    // L(u^n) of the pass's first (highest) step; the next ones X * Y before
  float* gK;            // dJ/dK, accumulated in place
};

// The cells outside the box are 0 in every state.
__device__ __forceinline__ void rw_zero_outer(float* a, float* b, int X, int Y, int pad) {
  const int band = pad * Y, side = (X - 2 * pad) * pad, total = 2 * band + 2 * side;
  for (int i = blockIdx.x * (int)blockDim.x + (int)threadIdx.x; i < total; i += (int)(gridDim.x * blockDim.x)) {
    int x, y;
    if (i < 2 * band) {
      const int b_ = i % band;
      x = b_ / Y + (i < band ? 0 : X - pad);
      y = b_ % Y;
    } else {
      const int b_ = (i - 2 * band) % side;
      x = pad + b_ / pad;
      y = b_ % pad + (i - 2 * band < side ? 0 : Y - pad);
    }
    a[(size_t)x * Y + y] = 0.0f;
    b[(size_t)x * Y + y] = 0.0f;
  }
}

// F: forward steps; A: adjoint steps (with both, step s of one and of the other
// between two barriers: independent chains that fill each other's latency).
// PAIRS: two neighbouring columns of a lane always form an aligned 8-byte word that
// is inside or outside the tile as a whole (a template parameter: both forms of
// every access in one kernel cost 5-10% of a pass).
template <bool F, bool A, bool PAIRS, int C, int RPT>
__global__ void __launch_bounds__(RT_WARPS * 32) wave_rt_kernel(const RWParams P) {
  constexpr int HP = RPT / 2;
  pdl_launch_dependents();
  extern __shared__ __align__(16) float rows[];
  const RTView<C, RPT> V(P.W, blockIdx.x);
  const int flip = (int)rt_buf_floats<1, C>(V.nw);
  float* const ownf = rt_own_row<1, C>(rows, V.warp, V.lane);
  float* const owna = ownf + (F ? 2 * flip : 0);
  const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
  const float2 nz = rt_pair(P.negzero), w0 = rt_pair(P.w[0]), w1 = rt_pair(P.w[1]), two = rt_pair(2.0f);
  auto M = [&](float2 a, float2 b) { return __ffma2_rn(a, b, nz); };
  const size_t first = (size_t)(P.pad + V.r0) * P.Y + P.pad + V.c0, cells = (size_t)P.X * P.Y;
  // the source cell, if this thread holds it
  const int sr = P.srcx - V.r0, sj = P.srcy - V.c0;
  const bool src_here = F && P.srcx >= 0 && V.on && sr >= 0 && sr < RPT && sj >= 0 && sj < C;
  const bool src_warp = F && __any_sync(0xffffffffu, src_here);
  auto load = [&](float2 (&v)[HP][C], const float* p) {  // the whole strip
    if constexpr (PAIRS) {
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) v[i][j] = rt_pair(0.0f);
      if (V.on) {
#pragma unroll
        for (int q = 0; q < RPT * C; q += 2) {
          const float2 t = *reinterpret_cast<const float2*>(p + (size_t)(q / C) * P.Y + q % C);
          rt_at<C, RPT>(v, q / C, q % C) = t.x;
          rt_at<C, RPT>(v, q / C, q % C + 1) = t.y;
        }
      }
    } else {
      rt_load<C, RPT>(v, p, P.Y, V.on);
    }
  };
  pdl_wait();
  float2 K[HP][C];
  load(K, P.K + first);
  float2 u[F ? HP : 1][C], um[F ? HP : 1][C];  // the two levels, in turn
  if constexpr (F) {
    if (P.kf > 0) {
      load(u, P.u0_in + first);
      load(um, P.um_in + first);
    }
  }
  float2 m1[A ? HP : 1][C], m2[A ? HP : 1][C], ga[A ? HP : 1][C], lv[A ? HP : 1][C];
  unsigned tmask = 0;  // bit r * C + j: the cell is in the tile
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int j = 0; j < C; ++j)
      if (V.row_in(r) && V.col_in(j)) tmask |= 1u << (r * C + j);
  constexpr int S = PAIRS ? 2 : 1;
  auto fetch = [&](float2 (&v)[HP][C], const float* p) {  // the tile's cells
#pragma unroll
    for (int q = 0; q < RPT * C; q += S)
      if (tmask & (1u << q)) {
        const float* c = p + (size_t)(q / C) * P.Y + q % C;
        if constexpr (PAIRS) {
          const float2 t = *reinterpret_cast<const float2*>(c);
          rt_at<C, RPT>(v, q / C, q % C) = t.x;
          rt_at<C, RPT>(v, q / C, q % C + 1) = t.y;
        } else {
          rt_at<C, RPT>(v, q / C, q % C) = *c;
        }
      }
  };
  auto store = [&](float2 (&v)[HP][C], float* p) {
#pragma unroll
    for (int q = 0; q < RPT * C; q += S)
      if (tmask & (1u << q)) {
        float* c = p + (size_t)(q / C) * P.Y + q % C;
        if constexpr (PAIRS)
          *reinterpret_cast<float2*>(c) = make_float2(rt_at<C, RPT>(v, q / C, q % C), rt_at<C, RPT>(v, q / C, q % C + 1));
        else
          *c = rt_at<C, RPT>(v, q / C, q % C);
      }
  };
  const float* lsrc = P.lsts + first;
  if constexpr (A) {
    if (P.ka > 0) {
      load(m1, P.m1_in + first);
      load(m2, P.m2_in + first);
    }
#pragma unroll
    for (int i = 0; i < HP; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) ga[i][j] = lv[i][j] = rt_pair(0.0f);
    if (P.ka > 0) {
      fetch(ga, P.gK + first);
      fetch(lv, lsrc);
    }
  }
  const RTGhosts<C, RPT> gh{};  // not read: 0 beyond the ring
  int par = 0;
  auto run = [&](auto Yc) {
    constexpr int YE = decltype(Yc)::value;
    // step s: the new levels over the old ones, so the two arrays of a chain take turns
    auto step = [&](auto Odd, int s) {
      constexpr bool odd = decltype(Odd)::value;
      auto& now = odd ? um : u;
      auto& old = odd ? u : um;
      auto& mu1 = odd ? m2 : m1;
      auto& mu2 = odd ? m1 : m2;
      const int fr = P.kf - 1 - s, ar = P.ka - 1 - s;  // negative past a chain's last step
      float* const bf = ownf + par;
      float* const ba = owna + par;
      RTRows<C> ef, ea;
      float2 z[A ? HP : 1][C];  // K o mu^{n+1}
      if constexpr (F) rt_rows_put<C, RPT>(now, bf, w0, nz, fr >= 0 && V.dist <= fr + 1, ef);
      if constexpr (A) {
#pragma unroll
        for (int i = 0; i < HP; ++i)
#pragma unroll
          for (int j = 0; j < C; ++j) z[i][j] = M(K[i][j], mu1[i][j]);
        rt_rows_put<C, RPT>(z, ba, w0, nz, ar >= 0 && V.dist <= ar + 1, ea);
      }
      const float sn = F && src_warp && fr >= 0 ? P.src[s] : 0.0f;
      __syncthreads();
      if constexpr (F) {
        if (V.dist <= fr) {  // u^{n+1} = 2 u^n - u^{n-1} + K o L(u^n) (+ source)
          float2 lap[HP][C];
          rt_rows_sum<YE, true, C, RPT>(now, V, bf, w0, nz, ef, gh, [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
            const float2 mid = M(w1, now[i][j]);
            float2 acc = __fadd2_rn(a, mid);
            acc = __fadd2_rn(acc, b);
            acc = __fadd2_rn(acc, l);
            acc = __fadd2_rn(acc, mid);
            acc = __fadd2_rn(acc, r);
            lap[i][j] = acc;
            // 2 u - u_prev in one rounding, as 2 u is exact (|u| under 1.7e38), then K L(u).
            // Both signs turned (u_prev - 2 u, subtracted) would need no negation, but
            // turns the sign of a zero: 512^2 x 2000 steps with gradient 4.97 against 4.98 ms.
            const float2 v = __ffma2_rn(two, now[i][j], make_float2(-old[i][j].x, -old[i][j].y));
            old[i][j] = __fadd2_rn(v, M(K[i][j], acc));
          });
          if (src_warp) {
#pragma unroll
            for (int r = 0; r < RPT; ++r)
#pragma unroll
              for (int j = 0; j < C; ++j) {
                float& q = rt_at<C, RPT>(old, r, j);
                q = src_here && r == sr && j == sj ? add(q, sn) : q;
              }
          }
          if (P.lst) store(lap, P.lst + first + (size_t)s * cells);
        }
      }
      if constexpr (A) {
        if (V.dist <= ar) {  // mu^n = 2 mu^{n+1} - mu^{n+2} + L(K o mu^{n+1}); dJ/dK += mu^{n+1} o L(u^n)
#pragma unroll
          for (int i = 0; i < HP; ++i)
#pragma unroll
            for (int j = 0; j < C; ++j) ga[i][j] = __fadd2_rn(ga[i][j], M(mu1[i][j], lv[i][j]));
          if (ar > 0) fetch(lv, lsrc - (size_t)(s + 1) * cells);
          rt_rows_sum<YE, true, C, RPT>(z, V, ba, w0, nz, ea, gh, [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
            const float2 mid = M(w1, z[i][j]);
            float2 acc = __fadd2_rn(a, mid);
            acc = __fadd2_rn(acc, b);
            acc = __fadd2_rn(acc, l);
            acc = __fadd2_rn(acc, mid);
            acc = __fadd2_rn(acc, r);
            const float2 v = __ffma2_rn(two, mu1[i][j], make_float2(-mu2[i][j].x, -mu2[i][j].y));
            mu2[i][j] = __fadd2_rn(v, acc);
          });
        }
      }
      par = flip - par;
    };
    const int n = F && A ? max(P.kf, P.ka) : F ? P.kf : P.ka;
    for (int s = 0; s < n; s += 2) {
      step(std::false_type{}, s);
      if (s + 1 < n) step(std::true_type{}, s + 1);
    }
  };
  if (ye == 0) run(std::integral_constant<int, 0>{});
  else if (ye == 1) run(std::integral_constant<int, 1>{});
  else if (ye == 2) run(std::integral_constant<int, 2>{});
  else run(std::integral_constant<int, 3>{});
  if constexpr (F) {
    if (P.kf > 0) {  // an odd count of steps leaves u^{n+1} in um
      store(u, ((P.kf & 1) ? P.um_out : P.u0_out) + first);
      store(um, ((P.kf & 1) ? P.u0_out : P.um_out) + first);
      rw_zero_outer(P.um_out, P.u0_out, P.X, P.Y, P.pad);
    }
  }
  if constexpr (A) {
    if (P.ka > 0) {
      store(m1, ((P.ka & 1) ? P.m2_out : P.m1_out) + first);
      store(m2, ((P.ka & 1) ? P.m1_out : P.m2_out) + first);
      store(ga, P.gK + first);
      rw_zero_outer(P.m1_out, P.m2_out, P.X, P.Y, P.pad);
    }
  }
}

}  // namespace pde
