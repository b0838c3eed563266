// Batched rollouts on register tiles: the work queue of batched.cuh (time block,
// grid, tile items, progress words, bounded waits), each item a window held in
// registers (regtile.cuh) instead of shared memory.  Heat of order 2 and wave; tiles
// cover each grid's stencil box (wave: the cells inside the node ring, outside of
// which the state is 0), sized per grid so that its windows are filled.  A block of
// 8 warps with 4 x 8 cells a thread (a 64 x 128 window) takes 128 registers a
// thread: two blocks per SM, one loading or waiting while the other steps.  Half the
// issue slots are used (barriers, dependent sums, window loads).  On one B200, against the shared-memory items, depth 10 the fastest of 4..16
// for both: 64 heat grids of 64..1024 a side x 100 steps 5.48 -> 2.04 ms, 24 wave
// grids x 200 steps 3.02 -> 1.28 ms.
#pragma once
#include "batched.cuh"
#include "regtile.cuh"

namespace pde {

constexpr int BRT_C = 4, BRT_RPT = 8, BRT_WARPS = 8;
constexpr int BRT_ROWS = BRT_WARPS * BRT_RPT, BRT_COLS = 32 * BRT_C;

// Rows of a strip with everything beyond H cells of the tile left out (nothing
// valid depends on those cells, and other blocks may be writing them).
__device__ __forceinline__ void brt_load(float2 (&u)[BRT_RPT / 2][BRT_C], const float* p, int pitch,
                                         const RTView<BRT_C, BRT_RPT>& V, int H) {
  bool need[BRT_C];
#pragma unroll
  for (int j = 0; j < BRT_C; ++j) need[j] = V.on && V.c0 + j >= V.by0 - H && V.c0 + j < V.by1 + H;
#pragma unroll
  for (int r = 0; r < BRT_RPT; ++r) {
    const bool row = V.r0 + r >= V.bx0 - H && V.r0 + r < V.bx1 + H;  // the same for the whole warp
#pragma unroll
    for (int j = 0; j < BRT_C; ++j) rt_at<BRT_C, BRT_RPT>(u, r, j) = 0.0f;
    if (row) {
#pragma unroll
      for (int j = 0; j < BRT_C; ++j)
        if (need[j]) rt_at<BRT_C, BRT_RPT>(u, r, j) = p[(size_t)r * pitch + j];
    }
  }
}

// One step: fill (boundary, if any), row exchange, sums through put.
template <int YE, bool ZERO, class Fill, class Put>
__device__ __forceinline__ void brt_step(float2 (&u)[BRT_RPT / 2][BRT_C], const RTView<BRT_C, BRT_RPT>& V, float* buf,
                                         float2 w0, float2 nz, int reach, const RTGhosts<BRT_C, BRT_RPT>& gh,
                                         Fill fill, Put put) {
  const bool live = V.dist <= reach + 1;
  if (live) fill();
  RTRows<BRT_C> e;
  rt_rows_put<BRT_C, BRT_RPT>(u, buf, w0, nz, live, e);
  __syncthreads();
  if (V.dist <= reach) rt_rows_sum<YE, ZERO, BRT_C, BRT_RPT>(u, V, buf, w0, nz, e, gh, put);
}

template <int OP>
__global__ void __launch_bounds__(BRT_WARPS * 32, 2) batched_rt_kernel(const BatchParams P, const PdeBCRules Rl,
                                                                       const float negzero) {
  constexpr int C = BRT_C, RPT = BRT_RPT, HP = RPT / 2;
  __shared__ __align__(16) float rows[rt_rows_floats<1, C>(BRT_WARPS)];
  __shared__ int s_item;
  __shared__ RTBc T;
  __shared__ PdeBCRules SR;  // ramps: the rules with the current step's group values
  const int tid = (int)threadIdx.x;
  if (OP == BATCH_HEAT && P.ramp && tid == 0) SR = Rl;
  const unsigned total_items = (unsigned)P.total_tiles * (unsigned)P.ntb;
  const int q = P.nsteps / P.ntb, rmd = P.nsteps % P.ntb;
  const float2 nz = rt_pair(negzero);
  auto M = [&](float2 a, float2 b) { return __ffma2_rn(a, b, nz); };
  bool timed_out = false;
  for (;;) {
    if (tid == 0) s_item = (int)atomicAdd(P.counter, 1u);
    __syncthreads();
    const unsigned item = (unsigned)s_item;
    if (item >= total_items) break;
    const int tb = (int)(item / (unsigned)P.total_tiles);
    const int gt = (int)(item - (unsigned)tb * (unsigned)P.total_tiles);
    int lo = 0, hi = P.ngrids - 1;  // the last grid whose tile_base <= gt
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (P.grids[mid].tile_base <= gt) lo = mid; else hi = mid - 1;
    }
    const BatchGridDev& Gd = P.grids[lo];
    const RTGeom W = Gd.W;
    const int lt = gt - Gd.tile_base;
    if (tb > 0 && tid < 9) {
      const int tx = lt / W.tiles_y, ty = lt - tx * W.tiles_y;
      const int nx = tx + tid / 3 - 1, ny = ty + tid % 3 - 1;
      if (nx >= 0 && nx < Gd.ntiles / W.tiles_y && ny >= 0 && ny < W.tiles_y && !timed_out) {
        if (!wait_at_least(P.progress + Gd.tile_base + nx * W.tiles_y + ny, (unsigned)tb, P.wait_ns)) {
          timed_out = true;
          flag_error(PDE_ERR_TIMEOUT);
        }
      }
      __threadfence();
    }
    if (OP == BATCH_HEAT && !P.ramp && tid >= 32 && tid < 53) rt_bc_entry(T, Rl, Gd.dx32, tid - 32);
    __syncthreads();
    const RTView<C, RPT> V(W, lt);
    const bool strip = V.warp < V.nw;  // small windows leave warps without rows
    const int ks = q + (tb < rmd ? 1 : 0);
    const bool odd = (tb & 1) != 0;
    const int pad = OP == BATCH_HEAT ? P.g : P.g + 1;  // array cells before the box
    const size_t first = (size_t)(pad + V.r0) * Gd.Y + pad + V.c0;
    const float2 w0 = rt_pair(Gd.w[0]), w1 = rt_pair(Gd.w[1]), coef = rt_pair(Gd.coef);
    float* const own = rt_own_row<1, C>(rows, V.warp, V.lane);
    const int flip = (int)rt_buf_floats<1, C>(BRT_WARPS);
    const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
    auto by_edge = [&](auto f) {
      if (ye == 0) f(std::integral_constant<int, 0>{});
      else if (ye == 1) f(std::integral_constant<int, 1>{});
      else if (ye == 2) f(std::integral_constant<int, 2>{});
      else f(std::integral_constant<int, 3>{});
    };
    int par = 0;
    if constexpr (OP == BATCH_HEAT) {
      const float* in = odd ? Gd.b0 : Gd.a0;
      float* out = odd ? Gd.a0 : Gd.b0;
      float2 u[HP][C];
      RTGhosts<C, RPT> gh;
      if (strip) brt_load(u, in + first, Gd.Y, V, W.H);
      const float2 dt = rt_pair(Gd.dt);
      const int n_first = tb * q + min(tb, rmd);  // rollout step of the block's first step
      by_edge([&](auto Y) {
        constexpr int YE = decltype(Y)::value;
        for (int reach = ks - 1; reach >= 0; --reach) {
          if (P.ramp) {  // this step's ramp values (the previous step's reads are behind its barrier)
            if (tid < Rl.ngroups && Rl.group[tid].func == PDE_BC_FUNC_RAMP) {
              const float t = step_time(P.t0, (double)Gd.dt, n_first + ks - 1 - reach);
              SR.group[tid].value = bc_value(PDE_BC_FUNC_RAMP, Rl.group[tid].value, Rl.group[tid].t_max, &t);
            }
            __syncthreads();
            if (tid < 21) rt_bc_entry(T, SR, Gd.dx32, tid);
            __syncthreads();
          }
          if (!strip) {
            __syncthreads();
            continue;
          }
          brt_step<YE, false>(
              u, V, own + par, w0, nz, reach, gh,
              [&]() {
                if (YE != 0 || V.xe) {
                  RTEdge E;
                  E.load(T, V);
                  rt_bc_fill<YE, C, RPT>(u, V, E, gh);
                }
              },
              [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
                const float2 mid = M(w1, u[i][j]);
                float2 acc = __fadd2_rn(a, mid);
                acc = __fadd2_rn(acc, b);
                acc = __fadd2_rn(acc, l);
                acc = __fadd2_rn(acc, mid);
                acc = __fadd2_rn(acc, r);
                u[i][j] = __fadd2_rn(u[i][j], M(dt, M(coef, acc)));
              });
          par = flip - par;
        }
      });
      if (strip && ks > 0) rt_store_all<C, RPT>(u, gh, V, out + first, Gd.Y);
      if (ks == 0) {  // no step: the tile and the ghosts next to it go on as they are
        const int x0 = V.bx0 + P.g - (V.bx0 == 0), x1 = V.bx1 + P.g + (V.bx1 == W.BX);
        const int y0 = V.by0 + P.g - (V.by0 == 0), y1 = V.by1 + P.g + (V.by1 == W.BY);
        RectWalk wk(y1 - y0, (int)blockDim.x);
        for (int i = tid; i < (x1 - x0) * (y1 - y0); i += (int)blockDim.x, wk.next()) {
          const int x = x0 + wk.row, y = y0 + wk.col;
          const bool xin = x >= P.g && x < Gd.X - P.g, yin = y >= P.g && y < Gd.Y - P.g;
          if (xin || yin) out[(size_t)x * Gd.Y + y] = in[(size_t)x * Gd.Y + y];  // a corner never changes
        }
      }
    } else {
      const float* in0 = odd ? Gd.b0 : Gd.a0;
      const float* in1 = odd ? Gd.b1 : Gd.a1;
      float* out0 = odd ? Gd.a0 : Gd.b0;
      float* out1 = odd ? Gd.a1 : Gd.b1;
      float2 u[HP][C], um[HP][C];  // the two levels, in turn
      if (strip) {
        brt_load(u, in0 + first, Gd.Y, V, W.H);
        brt_load(um, in1 + first, Gd.Y, V, W.H);
      }
      RTGhosts<C, RPT> gh;  // not read: 0 beyond the ring
      const float2 two = rt_pair(2.0f);
      by_edge([&](auto Y) {
        auto step = [&](float2 (&now)[HP][C], float2 (&old)[HP][C], int reach) {  // the new level over the old one
          brt_step<decltype(Y)::value, true>(now, V, own + par, w0, nz, reach, gh, []() {},
                                       [&](int i, int j, float2 a, float2 b, float2 l, float2 r) {
                                         const float2 mid = M(w1, now[i][j]);
                                         float2 acc = __fadd2_rn(a, mid);
                                         acc = __fadd2_rn(acc, b);
                                         acc = __fadd2_rn(acc, l);
                                         acc = __fadd2_rn(acc, mid);
                                         acc = __fadd2_rn(acc, r);
                                         // 2 u is exact: one rounding, as 2 u - u_prev has
                                         const float2 v =
                                             __ffma2_rn(two, now[i][j], make_float2(-old[i][j].x, -old[i][j].y));
                                         old[i][j] = __fadd2_rn(v, M(coef, acc));
                                       });
          par = flip - par;
        };
        if (!strip) {
          for (int s = 0; s < ks; ++s) __syncthreads();
          return;
        }
        int reach = ks - 1;
        for (; reach >= 1; reach -= 2) {
          step(u, um, reach);
          step(um, u, reach - 1);
        }
        if (reach == 0) step(u, um, 0);
      });
      if (strip) {
        const bool swapped = (ks & 1) != 0;
        rt_store<C, RPT>(u, (swapped ? out1 : out0) + first, Gd.Y, V);
        rt_store<C, RPT>(um, (swapped ? out0 : out1) + first, Gd.Y, V);
      }
      // The caller's fields come back 0 on the ring and the ghosts.  No window holds
      // those cells, so the tiles at the box's edges may write them at any time: in
      // the first block, away from the launch's tail (24 grids x 200 steps: 1.302 ms
      // by a walk over the grown tile in the last block, 1.280 ms so).
      if (tb == 0) {
        const int x0 = V.bx0 + pad, x1 = V.bx1 + pad, y0 = V.by0 + pad, y1 = V.by1 + pad;  // the tile in the array
        const int top = V.bx0 == 0 ? x0 : 0, bottom = V.bx1 == W.BX ? Gd.X - x1 : 0;
        const int left = V.by0 == 0 ? y0 : 0, right = V.by1 == W.BY ? Gd.Y - y1 : 0;
        const int wide = left + (y1 - y0) + right, rows_out = top + bottom, cols_out = left + right;
        for (int i = tid; i < rows_out * wide; i += (int)blockDim.x) {  // the rows above and below, corners included
          const int r = i / wide, x = r < top ? r : x1 + r - top;
          const size_t c = (size_t)x * Gd.Y + y0 - left + (i - r * wide);
          Gd.a0[c] = Gd.a1[c] = 0.0f;
        }
        for (int i = tid; i < (x1 - x0) * cols_out; i += (int)blockDim.x) {
          const int r = i / cols_out, q = i - r * cols_out, y = q < left ? q : y1 + q - left;
          const size_t c = (size_t)(x0 + r) * Gd.Y + y;
          Gd.a0[c] = Gd.a1[c] = 0.0f;
        }
      }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) st_release_gpu(P.progress + gt, (unsigned)(tb + 1));
  }
}

}  // namespace pde
