// Register tiles: the core of the temporally blocked 2D kernels.
//
// A block owns a tile of the stencil box [g, n-g) (boundary nodes included,
// ghosts not) and works on a window of it, the tile grown by a halo, held
// entirely in registers: warp w has RPT consecutive rows (x), lane l has C
// consecutive columns (y), so a thread holds RPT x C cells.  A step reads x
// neighbours from the thread's own registers (from shared memory at the strip's
// first and last R rows, which the warps publish once per step), y neighbours
// from the thread's own registers and by one shuffle per row, side and tap.
// Against the region in shared memory (one word read per tap, one written per
// cell) a cell costs 2 R / C shuffles and 4 R / RPT shared-memory words, so the
// arithmetic becomes the larger part.
//
// Arithmetic is packed f32x2 with the pair taken along x at a distance of half
// the strip: pair i of a column holds rows i and i + RPT/2, so the x neighbours
// of a pair are the pairs i - 1 and i + 1 (recombined only at the strip's two
// seams) and the y neighbours are the pair of the next column: no operand is
// ever packed.  Packed operations have the scalar rate per cell on this part
// (measured: 1 FADD or half an FADD2 per clock and scheduler) but take half the
// issue slots, which the shuffles and shared-memory words use.
//
// The window lies inside the box.  It starts H = k R cells before the tile, moved
// inward where that would leave the box; a window that reaches the box's low
// (high) end along an axis has its first (last) strip, or first (last) lane,
// aligned to it.  Ghosts are not stored: the boundary fill supplies them as the
// missing neighbours of the node rows and columns, from the partner cell next to
// the node, which the same thread holds.
#pragma once
#include "common.cuh"
#include "regtile_host.h"

namespace pde {

// One thread's view of its block's window.  Coordinates are box coordinates.
template <int C, int RPT>
struct RTView {
  int lane, warp, nw;
  int bx0, by0, bx1, by1;      // tile [bx0, bx1) x [by0, by1)
  int r0, c0;                  // the thread's first row and column
  int dist;                    // rows between this strip and the tile
  bool on;                     // this lane holds columns
  bool ylo, yhi;               // the window reaches the box's ends along y
  bool wlo, whi, xe;           // this strip is the box's first, last, either
  bool llo, lhi;               // this lane holds the box's first, last columns
  __device__ RTView(const RTGeom& G, int tile) {
    lane = (int)threadIdx.x & 31;
    warp = (int)threadIdx.x >> 5;
    nw = G.NR / RPT;
    const int tx = tile / G.tiles_y, ty = tile - tx * G.tiles_y;
    bx0 = G.X0 + tx * G.TBX;
    by0 = ty * G.TBY;
    bx1 = min(bx0 + G.TBX, G.X1);
    by1 = min(by0 + G.TBY, G.BY);
    const int rx0 = max(min(bx0 - G.H, G.BX - G.NR), 0), ry0 = max(min(by0 - G.H, G.BY - G.NC), 0);
    r0 = rx0 + warp * RPT;
    c0 = ry0 + lane * C;
    dist = max(max(bx0 - (r0 + RPT - 1), r0 - (bx1 - 1)), 0);
    const int lh = G.NC / C - 1;
    on = lane <= lh;
    ylo = ry0 == 0;
    yhi = ry0 + G.NC == G.BY;
    wlo = G.xlo && rx0 == 0 && warp == 0;
    whi = G.xhi && rx0 + G.NR == G.BX && warp == nw - 1;
    xe = wlo || whi;
    llo = ylo && lane == 0;
    lhi = yhi && lane == lh;
  }
  __device__ bool row_in(int r) const { return r0 + r >= bx0 && r0 + r < bx1; }           // the same for the whole warp
  __device__ bool col_in(int j) const { return on && c0 + j >= by0 && c0 + j < by1; }
};

// Element (row r, column j) of a strip held as pairs.
template <int C, int RPT>
__device__ __forceinline__ float& rt_at(float2 (&u)[RPT / 2][C], int r, int j) {
  return r < RPT / 2 ? u[r][j].x : u[r - RPT / 2][j].y;
}

__device__ __forceinline__ float2 rt_shfl_up(float2 v) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 rt_shfl_down(float2 v) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 rt_pair(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 rt_sel(bool c, float2 a, float2 b) {
  return make_float2(c ? a.x : b.x, c ? a.y : b.y);
}

// C consecutive floats of one lane to or from shared memory.
template <int C>
__device__ __forceinline__ void rt_put(float* p, const float* v) {
  if constexpr (C == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
}
template <int C>
__device__ __forceinline__ void rt_get(const float* p, float* v) {
  if constexpr (C == 4) {
    const float4 q = *reinterpret_cast<const float4*>(p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    const float2 q = *reinterpret_cast<const float2*>(p);
    v[0] = q.x; v[1] = q.y;
  }
}

// Shared-memory rows published by the warps of a block: R first and R last rows
// of each warp's strip, two buffers used in turn (one barrier per step).  The
// buffers start with R rows and end with R rows of padding, so the first and last
// strips read (unused) words of the block's own memory.
template <int R, int C>
constexpr size_t rt_buf_floats(int nw) {
  return (size_t)(nw * 2 * R + 2 * R) * 32 * C;
}
template <int R, int C>
constexpr size_t rt_rows_floats(int nw) {
  return 2 * rt_buf_floats<R, C>(nw);
}
// This thread's words of its strip's first row in buffer 0; row t (0..2R-1: first
// R rows, last R rows) is t * 32 * C further, the strip above's last R rows are at
// t = -R .. -1, the strip below's first R rows at t = 2R .. 3R-1.
template <int R, int C>
__device__ __forceinline__ float* rt_own_row(float* rows, int warp, int lane) {
  return rows + ((size_t)(R + warp * 2 * R) * 32 + lane) * C;
}

template <int R, int C, int RPT>
__device__ __forceinline__ void rt_publish(float* own, float2 (&e)[RPT / 2][C]) {
#pragma unroll
  for (int t = 0; t < 2 * R; ++t) {
    float v[C];
#pragma unroll
    for (int j = 0; j < C; ++j) v[j] = rt_at<C, RPT>(e, t < R ? t : RPT - 2 * R + t, j);
    rt_put<C>(own + t * 32 * C, v);
  }
}
// Rows -R .. -1 (up) and RPT .. RPT+R-1 (dn) of the strip, from the neighbouring warps.
template <int R, int C>
__device__ __forceinline__ void rt_neighbours(const float* own, float (&up)[R][C], float (&dn)[R][C]) {
#pragma unroll
  for (int t = 0; t < R; ++t) {
    rt_get<C>(own + (t - R) * 32 * C, up[t]);
    rt_get<C>(own + (2 * R + t) * 32 * C, dn[t]);
  }
}
// The strip extended by R pairs at either end: ext[R + i] = pair i; the seams
// take one half from the neighbouring rows, the other from this strip.
template <int R, int C, int RPT>
__device__ __forceinline__ void rt_extend(float2 (&e)[RPT / 2][C], const float (&up)[R][C], const float (&dn)[R][C],
                                          float2 (&ext)[RPT / 2 + 2 * R][C]) {
  constexpr int HP = RPT / 2;
#pragma unroll
  for (int j = 0; j < C; ++j) {
#pragma unroll
    for (int i = 0; i < HP; ++i) ext[R + i][j] = e[i][j];
#pragma unroll
    for (int t = 0; t < R; ++t) {
      ext[t][j] = make_float2(up[t][j], rt_at<C, RPT>(e, HP - R + t, j));
      ext[R + HP + t][j] = make_float2(rt_at<C, RPT>(e, HP + t, j), dn[t][j]);
    }
  }
}

// ---- boundary fill ------------------------------------------------------------
// The rules of a 2D one-component field as a table: a ghost's value is
// s * adj + c (Dirichlet: s = -1, c = 2 v; Neumann: s = 1, c = (-+2 dx) v), one
// fused multiply-add, which rounds exactly as the reference's formula since 2 v
// and the products with +-1 are exact.  Ghosts by edge (x low, x high, y low, y
// high) and class of the node along the other axis; nodes by both classes.
struct RTBc {
  float2 ghost[4][3];  // s, c
  float2 node[9];      // value, set (1 or 0)
};

__device__ __forceinline__ void rt_bc_entry(RTBc& T, const PdeBCRules& Rl, float dx32, int i) {
  if (i < 12) {
    const int edge = i / 3, cls = i - 3 * edge, axis = edge >> 1, side = edge & 1;
    const int along = side ? 2 : 0;
    const int K = axis == 0 ? along * 9 + cls * 3 + 1 : cls * 9 + along * 3 + 1;
    const int gi = Rl.ghost_group[K][axis][0];
    float2 t = make_float2(0.0f, 0.0f);
    if (gi >= 0) {
      const float v = Rl.group[gi].value;
      const int inc = side ? -1 : 1;
      t = Rl.group[gi].type == PDE_BC_DIRICHLET ? make_float2(-1.0f, mul(2.0f, v))
                                                : make_float2(1.0f, mul(mul((float)(-2 * inc), dx32), v));
    }
    T.ghost[edge][cls] = t;
  } else if (i < 21) {
    const int q = i - 12, K = (q / 3) * 9 + (q % 3) * 3 + 1;
    const int gi = Rl.node_group[K];
    T.node[q] = (gi >= 0 && (Rl.group[gi].comp_mask & 1u)) ? make_float2(Rl.group[gi].value, 1.0f)
                                                            : make_float2(0.0f, 0.0f);
  }
}

// The ghosts of this step, from the pre-boundary field: column ghosts of a lane
// at a y edge (one per row), row ghosts of a strip at an x edge (one per column).
template <int C, int RPT>
struct RTGhosts {
  float2 col[RPT / 2];
  float row[C];
};

// A thread's boundary coefficients in registers: a lane at a y edge meets one
// class of node on its first row (a corner when the strip is the box's first),
// one on its last row and the middle class between; a strip at an x edge the
// same along its columns.  A thread is at one y edge and one x edge at most.
struct RTEdge {
  float2 rf, rm, rl, cf, cm, cl;       // ghost (s, c): rows first, middle, last; columns first, middle, last
  float vrf, vrm, vrl, vcf, vcm, vcl;  // node values
  bool nrf, nrm, nrl, ncf, ncm, ncl;   // the node is set (rows: and this lane is at a y edge)
  template <int C, int RPT>
  __device__ __forceinline__ void load(const RTBc& T, const RTView<C, RPT>& V) {
    const bool ye = V.llo || V.lhi, xe = V.wlo || V.whi;
    {
      const int e = V.lhi ? 3 : 2, n = V.lhi ? 2 : 0, f = V.wlo ? 0 : 1, l = V.whi ? 2 : 1;
      rf = T.ghost[e][f];
      rm = T.ghost[e][1];
      rl = T.ghost[e][l];
      const float2 a = T.node[f * 3 + n], b = T.node[3 + n], c = T.node[l * 3 + n];
      vrf = a.x; vrm = b.x; vrl = c.x;
      nrf = ye && a.y != 0.0f; nrm = ye && b.y != 0.0f; nrl = ye && c.y != 0.0f;
    }
    {
      const int e = V.whi ? 1 : 0, n = V.whi ? 2 : 0, f = V.llo ? 0 : 1, l = V.lhi ? 2 : 1;
      cf = T.ghost[e][f];
      cm = T.ghost[e][1];
      cl = T.ghost[e][l];
      const float2 a = T.node[n * 3 + f], b = T.node[n * 3 + 1], c = T.node[n * 3 + l];
      vcf = a.x; vcm = b.x; vcl = c.x;
      ncf = xe && a.y != 0.0f; ncm = xe && b.y != 0.0f; ncl = xe && c.y != 0.0f;
    }
  }
};

// Ghosts of the step and, after them, the Dirichlet nodes.  YE: the window's y
// edges (1 low, 2 high), a template parameter so that a step has no branch for them.
template <int YE, int C, int RPT>
__device__ __forceinline__ void rt_bc_fill(float2 (&u)[RPT / 2][C], const RTView<C, RPT>& V, const RTEdge& E,
                                           RTGhosts<C, RPT>& gh) {
  constexpr int HP = RPT / 2;
  if constexpr (YE != 0) {
#pragma unroll
    for (int i = 0; i < HP; ++i) {
      const float2 a = i == 0 ? E.rf : E.rm, b = i == HP - 1 ? E.rl : E.rm;
      const float2 q = YE == 1 ? u[i][1] : YE == 2 ? u[i][C - 2] : rt_sel(V.lhi, u[i][C - 2], u[i][1]);  // the partner
      gh.col[i] = __ffma2_rn(make_float2(a.x, b.x), q, make_float2(a.y, b.y));
    }
  }
  if (V.xe) {
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const float2 t = j == 0 ? E.cf : (j == C - 1 ? E.cl : E.cm);
      const bool n = j == 0 ? E.ncf : j == C - 1 ? E.ncl : E.ncm;
      const float v = j == 0 ? E.vcf : j == C - 1 ? E.vcl : E.vcm;
      gh.row[j] = fmaf(t.x, V.wlo ? rt_at<C, RPT>(u, 1, j) : rt_at<C, RPT>(u, RPT - 2, j), t.y);
      rt_at<C, RPT>(u, 0, j) = V.wlo && n ? v : rt_at<C, RPT>(u, 0, j);
      rt_at<C, RPT>(u, RPT - 1, j) = V.whi && n ? v : rt_at<C, RPT>(u, RPT - 1, j);
    }
  }
  if constexpr (YE != 0) {
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const bool n = r == 0 ? E.nrf : r == RPT - 1 ? E.nrl : E.nrm;
      const float v = r == 0 ? E.vrf : r == RPT - 1 ? E.vrl : E.vrm;
      if constexpr ((YE & 1) != 0) rt_at<C, RPT>(u, r, 0) = V.llo && n ? v : rt_at<C, RPT>(u, r, 0);
      if constexpr ((YE & 2) != 0) rt_at<C, RPT>(u, r, C - 1) = V.lhi && n ? v : rt_at<C, RPT>(u, r, C - 1);
    }
  }
}

// The strip from and to a dense array (p: the thread's first cell, rows `pitch`
// floats apart); lanes beyond the window hold 0.
template <int C, int RPT>
__device__ __forceinline__ void rt_load(float2 (&u)[RPT / 2][C], const float* p, int pitch, bool on) {
  if constexpr (C * RPT >= 32) {  // one branch; small strips: a predicate per load (each 2% faster where it is used)
#pragma unroll
    for (int i = 0; i < RPT / 2; ++i)
#pragma unroll
      for (int j = 0; j < C; ++j) u[i][j] = rt_pair(0.0f);
    if (on) {
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int j = 0; j < C; ++j) rt_at<C, RPT>(u, r, j) = p[(size_t)r * pitch + j];
    }
  } else {
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int j = 0; j < C; ++j) rt_at<C, RPT>(u, r, j) = on ? p[(size_t)r * pitch + j] : 0.0f;
  }
}
// The tile's cells; rows are in or out for a whole warp, so a row costs one branch
// and its columns a predicate each.
template <int C, int RPT>
__device__ __forceinline__ void rt_store(float2 (&u)[RPT / 2][C], float* p, int pitch, const RTView<C, RPT>& V) {
  bool in[C];
#pragma unroll
  for (int j = 0; j < C; ++j) in[j] = V.col_in(j);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
    if (V.row_in(r)) {
#pragma unroll
      for (int j = 0; j < C; ++j)
        if (in[j]) p[(size_t)r * pitch + j] = rt_at<C, RPT>(u, r, j);
    }
}

// The tile, and the ghosts next to it as the last step's fill left them.
template <int C, int RPT>
__device__ __forceinline__ void rt_store_all(float2 (&u)[RPT / 2][C], const RTGhosts<C, RPT>& gh,
                                             const RTView<C, RPT>& V, float* o, int pitch) {
  constexpr int HP = RPT / 2;
  rt_store<C, RPT>(u, o, pitch, V);
  if ((V.llo || V.lhi) && V.col_in(V.llo ? 0 : C - 1)) {
#pragma unroll
    for (int r = 0; r < RPT; ++r)
      if (V.row_in(r))
        o[(size_t)r * pitch + (V.llo ? -1 : C)] = r < HP ? gh.col[r < HP ? r : 0].x : gh.col[r < HP ? 0 : r - HP].y;
  }
  if (V.xe && V.row_in(V.wlo ? 0 : RPT - 1)) {
    float* q = V.wlo ? o - pitch : o + (size_t)RPT * pitch;
#pragma unroll
    for (int j = 0; j < C; ++j)
      if (V.col_in(j)) q[j] = gh.row[j];
  }
}

// ---- order-2 sums of a strip, a row pair at a time -------------------------------
// The products of the outer weight are formed once per cell: those of the strip's
// first and last rows before the barrier, as the warps exchange them (rt_rows_put),
// the others as the rows go by (rt_rows_sum).
template <int C>
struct RTRows {
  float2 first[C], last[C];
};

template <int C, int RPT>
__device__ __forceinline__ void rt_rows_put(float2 (&u)[RPT / 2][C], float* buf, float2 w0, float2 nz, bool live,
                                            RTRows<C>& e) {
#pragma unroll
  for (int j = 0; j < C; ++j) {
    e.first[j] = __ffma2_rn(w0, u[0][j], nz);
    e.last[j] = __ffma2_rn(w0, u[RPT / 2 - 1][j], nz);
  }
  if (live) {
    float top[C], bot[C];
#pragma unroll
    for (int j = 0; j < C; ++j) {
      top[j] = e.first[j].x;
      bot[j] = e.last[j].y;
    }
    rt_put<C>(buf, top);
    rt_put<C>(buf + 32 * C, bot);
  }
}

// put(i, j, a, b, l, r): the products of pair (i, j)'s neighbours above, below, left
// and right.  ZERO: the field is 0 beyond the box; else its ghosts are in gh.
template <int YE, bool ZERO, int C, int RPT, class Put>
__device__ __forceinline__ void rt_rows_sum(float2 (&u)[RPT / 2][C], const RTView<C, RPT>& V, const float* buf,
                                            float2 w0, float2 nz, const RTRows<C>& e, const RTGhosts<C, RPT>& gh,
                                            Put put) {
  constexpr int HP = RPT / 2;
  auto M = [&](float2 a, float2 b) { return __ffma2_rn(a, b, nz); };
  const float2 zero = rt_pair(0.0f);
  float up[C], dn[C];
  rt_get<C>(buf - 32 * C, up);
  rt_get<C>(buf + 2 * 32 * C, dn);
  if (V.xe) {
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const float q = ZERO ? 0.0f : mul(w0.x, gh.row[j]);
      up[j] = V.wlo ? q : up[j];
      dn[j] = V.whi ? q : dn[j];
    }
  }
  float2 cur[C], above[C], below[C];
#pragma unroll
  for (int j = 0; j < C; ++j) {
    cur[j] = e.first[j];
    above[j] = make_float2(up[j], e.last[j].x);
    below[j] = make_float2(e.first[j].y, dn[j]);
  }
#pragma unroll
  for (int i = 0; i < HP; ++i) {
    float2 next[C];
#pragma unroll
    for (int j = 0; j < C; ++j)
      next[j] = i == HP - 1 ? below[j] : (i == HP - 2 ? e.last[j] : M(w0, u[i + 1 < HP ? i + 1 : i][j]));
    float2 le = rt_shfl_up(cur[C - 1]), ri = rt_shfl_down(cur[0]);
    if constexpr ((YE & 1) != 0) le = rt_sel(V.llo, ZERO ? zero : M(w0, gh.col[i]), le);
    if constexpr ((YE & 2) != 0) ri = rt_sel(V.lhi, ZERO ? zero : M(w0, gh.col[i]), ri);
#pragma unroll
    for (int j = 0; j < C; ++j)
      put(i, j, above[j], next[j], j > 0 ? cur[j > 0 ? j - 1 : 0] : le, j < C - 1 ? cur[j < C - 1 ? j + 1 : 0] : ri);
#pragma unroll
    for (int j = 0; j < C; ++j) {
      above[j] = cur[j];
      cur[j] = next[j];
    }
  }
}

// ---- heat -----------------------------------------------------------------------
struct RHParams {
  RTGeom W;
  int X, Y, g;        // array extents, ghost width
  int k;              // steps of this pass
  float w[3];         // Laplacian weights from the outermost tap to the centre (symmetric)
  float alpha, dt;
  float negzero;      // -0 at run time: a product a * b + (-0) is exactly rounded and never contracted
  double t0, tstep;   // ramps: step n of the rollout fills the boundary at fp32(t0 + n * tstep)
  int n0;
  const float* in;
  float* out;
};

// The array's cells outside the box that the fill never writes (corners, and all
// but the innermost ghost layer) keep the input's values; rows [lo, hi).
__device__ __forceinline__ void rt_copy_outer(const float* in, float* out, int X, int Y, int g, int lo, int hi) {
  const int band = g * Y, side = (X - 2 * g) * g, total = 2 * band + 2 * side;
  for (int i = blockIdx.x * (int)blockDim.x + (int)threadIdx.x; i < total; i += (int)(gridDim.x * blockDim.x)) {
    int x, y;
    if (i < 2 * band) {
      const int b = i % band;
      x = b / Y + (i < band ? 0 : X - g);
      y = b % Y;
      if ((x == g - 1 || x == X - g) && y >= g && y < Y - g) continue;
    } else {
      const int b = (i - 2 * band) % side;
      x = g + b / g;
      y = b % g + (i - 2 * band < side ? 0 : Y - g);
      if (y == g - 1 || y == Y - g) continue;
    }
    if (x >= lo && x < hi) out[(size_t)x * Y + y] = in[(size_t)x * Y + y];
  }
}

// Constant layer beyond the filled ghosts (order 4 reads it): cells of the input.
template <int R, int C, int RPT>
struct RTDeep {
  float2 col[R == 2 ? RPT / 2 : 1];
  float row[R == 2 ? C : 1];
  __device__ void load(const float* first, int Y, const RTView<C, RPT>& V) {
    if constexpr (R == 2) {
      constexpr int HP = RPT / 2;
#pragma unroll
      for (int i = 0; i < HP; ++i) {
        const float* p = first + (V.llo ? -2 : C + 1);
        col[i] = (V.llo || V.lhi) ? make_float2(p[(size_t)i * Y], p[(size_t)(i + HP) * Y]) : rt_pair(0.0f);
      }
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const float* p = V.wlo ? first - 2 * (size_t)Y : first + (size_t)(RPT + 1) * Y;
        row[j] = (V.wlo || V.whi) && V.on ? p[j] : 0.0f;
      }
    }
  }
};

// One step of the strip, u + dt * (alpha * L(u)), with the reference's sum (x taps
// low to high, then y taps).  YE: the window's y edges.
// R = 1: each cell's two products are formed once and the outer one is what the
// warps and lanes exchange; R = 2: they exchange the field (three products of a
// neighbour would be needed) and form the products of the cells they receive.
template <int R, int C, int RPT>
struct RTHeat {
  static constexpr int HP = RPT / 2;
  float2 w[R + 1], al, dt, nz;
  __device__ RTHeat(const RHParams& P) {
#pragma unroll
    for (int t = 0; t <= R; ++t) w[t] = rt_pair(P.w[t]);
    al = rt_pair(P.alpha);
    dt = rt_pair(P.dt);
    nz = rt_pair(P.negzero);
  }
  __device__ float2 M(float2 a, float2 b) const { return __ffma2_rn(a, b, nz); }

  template <int YE>
  __device__ __forceinline__ void step(float2 (&u)[HP][C], const RTView<C, RPT>& V, float* buf, const RTEdge& E,
                                       const RTDeep<R, C, RPT>& deep, int reach, RTGhosts<C, RPT>& gh) const {
    const bool live = V.dist <= reach + R;
    if (live) rt_bc_fill<YE, C, RPT>(u, V, E, gh);
    if constexpr (R == 1) {
      float2 p[HP + 2][C], le[HP], ri[HP];
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) p[i + 1][j] = M(w[0], u[i][j]);
      if (live) {
        float top[C], bot[C];
#pragma unroll
        for (int j = 0; j < C; ++j) {
          top[j] = p[1][j].x;
          bot[j] = p[HP][j].y;
        }
        rt_put<C>(buf, top);
        rt_put<C>(buf + 32 * C, bot);
      }
#pragma unroll
      for (int i = 0; i < HP; ++i) {
        le[i] = rt_shfl_up(p[i + 1][C - 1]);
        ri[i] = rt_shfl_down(p[i + 1][0]);
      }
      if constexpr ((YE & 1) != 0) {
#pragma unroll
        for (int i = 0; i < HP; ++i) le[i] = rt_sel(V.llo, M(w[0], gh.col[i]), le[i]);
      }
      if constexpr ((YE & 2) != 0) {
#pragma unroll
        for (int i = 0; i < HP; ++i) ri[i] = rt_sel(V.lhi, M(w[0], gh.col[i]), ri[i]);
      }
      __syncthreads();
      if (V.dist > reach) return;
      float up[C], dn[C];
      rt_get<C>(buf - 32 * C, up);
      rt_get<C>(buf + 2 * 32 * C, dn);
      if (V.xe) {
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const float q = mul(w[0].x, gh.row[j]);
          up[j] = V.wlo ? q : up[j];
          dn[j] = V.whi ? q : dn[j];
        }
      }
#pragma unroll
      for (int j = 0; j < C; ++j) {
        p[0][j] = make_float2(up[j], p[HP][j].x);
        p[HP + 1][j] = make_float2(p[1][j].y, dn[j]);
      }
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const float2 mid = M(w[1], u[i][j]);
          float2 acc = __fadd2_rn(p[i][j], mid);
          acc = __fadd2_rn(acc, p[i + 2][j]);
          acc = __fadd2_rn(acc, j > 0 ? p[i + 1][j > 0 ? j - 1 : 0] : le[i]);
          acc = __fadd2_rn(acc, mid);
          acc = __fadd2_rn(acc, j < C - 1 ? p[i + 1][j < C - 1 ? j + 1 : 0] : ri[i]);
          u[i][j] = __fadd2_rn(u[i][j], M(dt, M(al, acc)));
        }
    } else {
      if (live) rt_publish<R, C, RPT>(buf, u);
      // columns of the neighbouring lanes: le[t] is t + 1 columns to the left, ri[t] to the right
      float2 le[R][HP], ri[R][HP];
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int t = 0; t < R; ++t) {
          le[t][i] = rt_shfl_up(u[i][C - 1 - t]);
          ri[t][i] = rt_shfl_down(u[i][t]);
        }
      if constexpr ((YE & 1) != 0) {
#pragma unroll
        for (int i = 0; i < HP; ++i) {
          le[0][i] = rt_sel(V.llo, gh.col[i], le[0][i]);
          le[R - 1][i] = rt_sel(V.llo, deep.col[i], le[R - 1][i]);
        }
      }
      if constexpr ((YE & 2) != 0) {
#pragma unroll
        for (int i = 0; i < HP; ++i) {
          ri[0][i] = rt_sel(V.lhi, gh.col[i], ri[0][i]);
          ri[R - 1][i] = rt_sel(V.lhi, deep.col[i], ri[R - 1][i]);
        }
      }
      __syncthreads();
      if (V.dist > reach) return;
      float up[R][C], dn[R][C];
      rt_neighbours<R, C>(buf, up, dn);
      if (V.xe) {
#pragma unroll
        for (int j = 0; j < C; ++j) {
          up[R - 1][j] = V.wlo ? gh.row[j] : up[R - 1][j];
          up[0][j] = V.wlo ? deep.row[j] : up[0][j];
          dn[0][j] = V.whi ? gh.row[j] : dn[0][j];
          dn[R - 1][j] = V.whi ? deep.row[j] : dn[R - 1][j];
        }
      }
      float2 ext[HP + 2 * R][C], nu[HP][C];
      rt_extend<R, C, RPT>(u, up, dn, ext);
#pragma unroll
      for (int i = 0; i < HP; ++i) {
        float2 row[C + 2 * R];
#pragma unroll
        for (int j = 0; j < C; ++j) row[R + j] = u[i][j];
#pragma unroll
        for (int t = 0; t < R; ++t) {
          row[R - 1 - t] = le[t][i];
          row[R + C + t] = ri[t][i];
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const float2 mid = M(w[2], u[i][j]);
          float2 acc = __fadd2_rn(M(w[0], ext[i][j]), M(w[1], ext[i + 1][j]));
          acc = __fadd2_rn(acc, mid);
          acc = __fadd2_rn(acc, M(w[1], ext[i + 3][j]));
          acc = __fadd2_rn(acc, M(w[0], ext[i + 4][j]));
          acc = __fadd2_rn(acc, M(w[0], row[j]));
          acc = __fadd2_rn(acc, M(w[1], row[j + 1]));
          acc = __fadd2_rn(acc, mid);
          acc = __fadd2_rn(acc, M(w[1], row[j + 3]));
          acc = __fadd2_rn(acc, M(w[0], row[j + 4]));
          nu[i][j] = __fadd2_rn(u[i][j], M(dt, M(al, acc)));
        }
      }
#pragma unroll
      for (int i = 0; i < HP; ++i)
#pragma unroll
        for (int j = 0; j < C; ++j) u[i][j] = nu[i][j];
    }
  }
};

// k steps of a pass.  Bound by issue and latency, not memory (256^2 and 1024^2 lie
// in L2).  Against the shared-memory kernel (heat2d_cells_kernel), which reads 5-10
// words of shared memory per cell and step, microseconds per step on one B200:
// 256^2 order 2 1.02 -> 0.47, 1024^2 order 2 3.9 -> 1.3, 2048^2 order 2 11.7 -> 4.5,
// 515 x 331 order 4 2.31 -> 1.02, 1024^2 order 4 5.2 -> 3.3.  A persistent form that
// exchanged halos through L2 words instead of relaunching cost 2.0 us per exchange
// against 2.6 us per dependent launch, and nothing at the depths in use: not kept.
template <int R, int C, int RPT>
__global__ void __launch_bounds__(rt_heat_warps(C, RPT) * 32) heat2d_rt_kernel(const RHParams P, const PdeBCRules Rl) {
  constexpr int HP = RPT / 2;
  pdl_launch_dependents();  // the next pass may be scheduled; it waits for this one
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
  float* const own = rt_own_row<R, C>(rows, V.warp, V.lane);
  const int flip = (int)rt_buf_floats<R, C>(V.nw);
  const RTHeat<R, C, RPT> op(P);
  const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
  const size_t first = (size_t)(P.g + V.r0) * P.Y + P.g + V.c0;  // the thread's first cell in the array
  pdl_wait();  // the previous pass's output (this pass's input) is complete
  float2 u[HP][C];
  rt_load<C, RPT>(u, P.in + first, P.Y, V.on);
  RTDeep<R, C, RPT> deep;
  deep.load(P.in + first, P.Y, V);
  int par = 0;
  // Step s only has to update the cells within R (k - 1 - s) of the tile: the
  // strips beyond that rest.  The fill and the rows are needed one R further.
  auto run = [&](auto Y) {
    for (int reach = R * (P.k - 1); reach >= 0; reach -= R) {
      if (Rl.has_ramp) {
        // every read of the table in the previous step came before its barrier
        if (tid < Rl.ngroups && Rl.group[tid].func == PDE_BC_FUNC_RAMP) {
          const float t = step_time(P.t0, P.tstep, P.n0 + P.k - 1 - reach / R);
          SR.group[tid].value = bc_value(PDE_BC_FUNC_RAMP, Rl.group[tid].value, Rl.group[tid].t_max, &t);
        }
        __syncthreads();
        for (int i = tid; i < 21; i += nt) rt_bc_entry(T, SR, Rl.dx32, i);
        __syncthreads();
        E.load(T, V);
      }
      op.template step<decltype(Y)::value>(u, V, own + par, E, deep, reach, gh);
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

// ---- Jacobi sweeps ------------------------------------------------------------------
struct RJParams {
  RTGeom W;
  int X, Y, g;
  int x0;             // global row of box row 0
  int own_lo, own_hi; // rows this launch writes (global)
  int k;
  float h2, negzero;
  const float* in;    // arrays addressed by global row
  float* out;
  const float* rhs;
  float* resid;       // if set: the sum of squared updates of the last sweep's tile cells
};

// k sweeps  p <- 0.25 * ((((pW + pE) + pS) + pN) - h^2 rhs)  of a pass on BC_p(p);
// h^2 rhs stays in registers.  Bound by a sweep's latency (barrier, dependent sums) with
// 41% of the issue slots used.  50 sweeps on one B200, against cell lists over shared memory
// (five words of it read and one written per cell and sweep): 1024^2 139 -> 60 us
// (one 128 x 128 window per SM, 4 x 8 cells a thread), 400^2 31 us, 100^2 24 us.
template <int C, int RPT>
__global__ void __launch_bounds__(RT_WARPS * 32) jacobi2d_rt_kernel(const RJParams P, const PdeBCRules Rl) {
  constexpr int HP = RPT / 2;
  pdl_launch_dependents();  // the next pass may be scheduled; it waits for this one
  extern __shared__ __align__(16) float rows[];
  __shared__ RTBc T;
  const RTView<C, RPT> V(P.W, blockIdx.x);
  for (int i = (int)threadIdx.x; i < 21; i += (int)blockDim.x) rt_bc_entry(T, Rl, Rl.dx32, i);
  __syncthreads();
  RTGhosts<C, RPT> gh;
  RTEdge E;
  if (RPT * C < 32) E.load(T, V);
  float* const own = rt_own_row<1, C>(rows, V.warp, V.lane);
  const int flip = (int)rt_buf_floats<1, C>(V.nw);
  const int ye = (V.ylo ? 1 : 0) | (V.yhi ? 2 : 0);
  const float2 nz = rt_pair(P.negzero), q4 = rt_pair(0.25f), h2 = rt_pair(P.h2);
  const size_t first = (size_t)(P.x0 + V.r0) * P.Y + P.g + V.c0;
  pdl_wait();  // the previous pass's pressure (this pass's input) is complete
  float2 u[HP][C], hr[HP][C];
  rt_load<C, RPT>(u, P.in + first, P.Y, V.on);
  rt_load<C, RPT>(hr, P.rhs + first, P.Y, V.on);
#pragma unroll
  for (int i = 0; i < HP; ++i)
#pragma unroll
    for (int j = 0; j < C; ++j) {
      const float2 t = __ffma2_rn(h2, hr[i][j], nz);
      hr[i][j] = make_float2(-t.x, -t.y);  // a - b as a + (-b)
    }
  float sq = 0.0f;
  auto sweep = [&](auto Y, auto N, float* buf, int reach) {
    constexpr int YE = decltype(Y)::value;
    constexpr bool norm = decltype(N)::value;  // the step's last sweep: its squared update
    const bool live = V.dist <= reach + 1;
    if (live) {
      if (RPT * C >= 32 && (YE != 0 || V.xe)) E.load(T, V);  // large strips: not kept in registers
      rt_bc_fill<YE, C, RPT>(u, V, E, gh);
      rt_publish<1, C, RPT>(buf, u);
    }
    float2 le[HP], ri[HP];
#pragma unroll
    for (int i = 0; i < HP; ++i) {
      le[i] = rt_shfl_up(u[i][C - 1]);
      ri[i] = rt_shfl_down(u[i][0]);
      if constexpr ((YE & 1) != 0) le[i] = rt_sel(V.llo, gh.col[i], le[i]);
      if constexpr ((YE & 2) != 0) ri[i] = rt_sel(V.lhi, gh.col[i], ri[i]);
    }
    __syncthreads();
    if (V.dist > reach) return;
    float up[1][C], dn[1][C];
    rt_neighbours<1, C>(buf, up, dn);
    if (V.xe) {
#pragma unroll
      for (int j = 0; j < C; ++j) {
        up[0][j] = V.wlo ? gh.row[j] : up[0][j];
        dn[0][j] = V.whi ? gh.row[j] : dn[0][j];
      }
    }
    float2 above[C];  // the old pair of row i - 1
#pragma unroll
    for (int j = 0; j < C; ++j) above[j] = make_float2(up[0][j], u[HP - 1][j].x);
    float2 below_last[C];
#pragma unroll
    for (int j = 0; j < C; ++j) below_last[j] = make_float2(u[0][j].y, dn[0][j]);
#pragma unroll
    for (int i = 0; i < HP; ++i) {
      float2 nu[C];
#pragma unroll
      for (int j = 0; j < C; ++j) {
        const float2 dnv = i == HP - 1 ? below_last[j] : u[i + 1 < HP ? i + 1 : i][j];
        float2 a = __fadd2_rn(above[j], dnv);
        a = __fadd2_rn(a, j > 0 ? u[i][j > 0 ? j - 1 : 0] : le[i]);
        a = __fadd2_rn(a, j < C - 1 ? u[i][j < C - 1 ? j + 1 : 0] : ri[i]);
        nu[j] = __ffma2_rn(q4, __fadd2_rn(a, hr[i][j]), nz);
      }
      if constexpr (norm) {
#pragma unroll
        for (int j = 0; j < C; ++j) {
          const float dx = nu[j].x - u[i][j].x, dy = nu[j].y - u[i][j].y;
          if (V.row_in(i) && V.col_in(j)) sq = fmaf(dx, dx, sq);
          if (V.row_in(i + HP) && V.col_in(j)) sq = fmaf(dy, dy, sq);
        }
      }
#pragma unroll
      for (int j = 0; j < C; ++j) {
        above[j] = u[i][j];
        u[i][j] = nu[j];
      }
    }
  };
  int par = 0;
  auto run = [&](auto Y) {
    for (int reach = P.k - 1; reach >= 0; --reach) {
      if (reach == 0 && P.resid) sweep(Y, std::true_type{}, own + par, reach);
      else sweep(Y, std::false_type{}, own + par, reach);
      par = flip - par;
    }
  };
  if (ye == 0) run(std::integral_constant<int, 0>{});
  else if (ye == 1) run(std::integral_constant<int, 1>{});
  else if (ye == 2) run(std::integral_constant<int, 2>{});
  else run(std::integral_constant<int, 3>{});
  rt_store_all<C, RPT>(u, gh, V, P.out + first, P.Y);
  rt_copy_outer(P.in, P.out, P.X, P.Y, P.g, P.own_lo, P.own_hi);
  if (P.resid) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
    __shared__ float wsum[32];
    if (V.lane == 0) wsum[V.warp] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      float b = 0.0f;
      for (int w = 0; w < V.nw; ++w) b += wsum[w];
      atomicAdd(P.resid, b);
    }
  }
}

}  // namespace pde
