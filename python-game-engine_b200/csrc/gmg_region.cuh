// Level kernels of the convergent multigrid on register regions, for levels that do not fill
// the GPU with the large register tiles and for levels with obstacles (included inside
// namespace sg by gmg.cu; uses w1 and rcp_open of gmg_weights.cuh).
//
//   k_gmg_pre_region    sweeps + residual + full weighting
//   k_gmg_post_region   prolongation + sweeps; FINAL: p += e
//   k_gmg_tail_region   every level of at most 64 x 64 cells and the exact coarsest solve in
//                       one block, V or W
//
// A block of 16 warps holds 16 RPT rows x 64 columns: lane l of warp w has columns i0 + 2l,
// i0 + 2l + 1 of rows j0 + w RPT .. + RPT - 1 (all even, so a register cell's colour is known at
// compile time); neighbours come by shuffle, from the thread's own registers, or through
// shared memory at a warp's first and last row (one barrier per half sweep, and only the
// colour that is read). Cells off the grid or not fluid hold e = 0 and have relaxation weight
// 0, so a half sweep has no branch and no test: a closed face contributes the 0 of the cell
// behind it. That needs every face between two fluid cells to be open, which holds on all
// levels but a fine one whose caller closed such a face (Level::simple).
//
// What bounds them: these levels sit in L2 and a launch is a few microseconds of latency
// (load, one barrier chain per half sweep, store), so what counts is the number of dependent
// launches and the length of one warp's instruction stream. Edge tests are selects: as branches
// they parted the edge lanes from the rest of every warp (tail 18.8 and 22.8 us in float32 and
// float64, pre / post 3.6 / 3.4). Measured, us: a 421 x 300 mixed cycle around obstacles (5
// levels of half-sweep launches, 55 in all, before) 117 -> 38; a 512^2 float64 cycle (4 levels of
// 16 x 16 shared-memory tiles and a 16^2 tail before) 71 -> 59; pre and post of a level 3.1 and
// 3.1 in float32, 3.8 and 3.8 in float64 (5.1 and 3.8 on the tiles); the tail from 64^2 down 15.2
// in float32, 20.7 in float64, for 27.2 as two tiled levels and a 16^2 tail.
#pragma once

// Bits 5..7 of a cell's code, for its transfer to the next coarser level: that the coarse
// candidate across in x, in y, or diagonally (after clamping to the grid) is another cell
// than the home one and not fluid, so that its weight goes to the home cell.
enum : uint8_t { C_XHOME = 32, C_YHOME = 64, C_DHOME = 128 };

constexpr int kRgWarps = 16;
constexpr int kRgThreads = 32 * kRgWarps;
constexpr int kRgCols = 64;
constexpr int kRgRows = 2;       // rows per thread of the level kernels

__host__ __device__ inline int region_tiles(int n, int span, int halo) {
  const int own = span - 2 * halo;
  return n <= span ? 1 : (n - 2 * halo + own - 1) / own;
}

struct RegionLevel {
  const uint8_t* code;  // H x W, row stride W; null on an open box
  int H, W;
};

template <typename T, int NW>
struct RegionEdges {
  T top[2][NW][2][32];
  T bot[2][NW][2][32];
};

template <bool PART>
__device__ __forceinline__ void region_barrier(int threads) {
  if (PART)
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  else
    __syncthreads();
}

// The thread's cells. code: one byte a cell, two cells a 16-bit half, two rows a word.
template <typename T, int RPT>
struct Region {
  T e[RPT][2], b[RPT][2];
  T rc[RPT][2], om[RPT][2];  // 1 / open faces and the relaxation weight (0: never updated)
  uint32_t code[(RPT + 1) / 2];

  __device__ __forceinline__ uint32_t c(int r, int q) const { return (code[r >> 1] >> (16 * (r & 1) + 8 * q)) & 255; }
  // Codes and weights of the cells at rows j + r, columns i + q (j, i >= 0). An open box's come
  // from one row part and one column part each: formed cell by cell from the position they
  // were a third of the tail's instructions.
  __device__ __forceinline__ void set_codes(const RegionLevel& m, int j, int i, T omega) {
    uint32_t k[RPT][2];
    if (m.code) {
#pragma unroll
      for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int q = 0; q < 2; ++q)  // clamped, so that all loads are in flight at once
          k[r][q] = m.code[(int64_t)min(j + r, m.H - 1) * m.W + min(i + q, m.W - 1)];
    } else {
      uint32_t col[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) col[q] = C_FLUID | (i + q > 0 ? C_L : 0) | (i + q < m.W - 1 ? C_R : 0);
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const uint32_t row = (j + r > 0 ? C_D : 0) | (j + r < m.H - 1 ? C_U : 0);
        k[r][0] = col[0] | row;
        k[r][1] = col[1] | row;
      }
    }
#pragma unroll
    for (int r = 0; r < (RPT + 1) / 2; ++r) code[r] = 0;
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (j + r >= m.H || i + q >= m.W) k[r][q] = 0;
        code[r >> 1] |= k[r][q] << (16 * (r & 1) + 8 * q);
        const uint32_t n = __popc(k[r][q] & (C_L | C_R | C_D | C_U));  // 0 .. 4: bit 2 is set for 4 only
        const T few = pick_bits(n, 1, pick_bits(n, 2, (T)(1.0 / 3.0), (T)1), (T)0.5);
        rc[r][q] = pick_bits(n, 4, (T)0.25, few);
        om[r][q] = pick_bits(n, 7, pick_bits(k[r][q], C_FLUID, omega, (T)0), (T)0);
      }
  }
};

// The value of the column left of the lane's first one, or right of its second one: the
// neighbouring lane's, or 0 at the region's ends (off the grid, or a halo cell).
template <typename T>
__device__ __forceinline__ T from_left(T v, int lane) {
  return pick_bits(lane, ~0u, __shfl_up_sync(0xffffffffu, v, 1), (T)0);
}
template <typename T>
__device__ __forceinline__ T from_right(T v, int lane) {
  return pick_bits(31 - lane, ~0u, __shfl_down_sync(0xffffffffu, v, 1), (T)0);
}

// One half sweep of colour COL. nw: warps that hold rows of the level; the rows outside
// the region count as 0.
template <typename T, int COL, int RPT, bool PART, typename E>
__device__ __forceinline__ void region_half_sweep(E& sh, int buf, int w, int lane, Region<T, RPT>& g,
                                                  int nw) {
  sh.bot[buf][w][0][lane] = g.e[RPT - 1][COL];  // for the next warp's first row
  sh.top[buf][w][0][lane] = g.e[0][1 - COL];    // for the previous warp's last row
  T acc[RPT];
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int q = (COL + r) & 1;
    const T far = q == 0 ? from_left(g.e[r][1], lane) : from_right(g.e[r][0], lane);
    acc[r] = g.b[r][q] + (q == 0 ? far : g.e[r][0]) + (q == 0 ? g.e[r][1] : far);
  }
  region_barrier<PART>(32 * nw);
  const T below = pick_bits(w, ~0u, sh.bot[buf][max(w - 1, 0)][0][lane], (T)0);
  const T above = pick_bits(nw - 1 - w, ~0u, sh.top[buf][min(w + 1, nw - 1)][0][lane], (T)0);
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int q = (COL + r) & 1;
    const T d = r > 0 ? g.e[r > 0 ? r - 1 : 0][q] : below;
    const T u = r < RPT - 1 ? g.e[r < RPT - 1 ? r + 1 : r][q] : above;
    const T x = g.e[r][q];
    acc[r] = acc[r] + d + u;
    g.e[r][q] = x + g.om[r][q] * (acc[r] * g.rc[r][q] - x);
  }
}

template <typename T, int RPT, bool PART, typename E>
__device__ __forceinline__ void region_sweeps(E& sh, int& buf, int w, int lane, Region<T, RPT>& g,
                                              int sweeps, int nw) {
  for (int s = 0; s < sweeps; ++s) {
    region_half_sweep<T, 0, RPT, PART>(sh, buf, w, lane, g, nw);
    buf ^= 1;
    region_half_sweep<T, 1, RPT, PART>(sh, buf, w, lane, g, nw);
    buf ^= 1;
  }
}

// Rows -1 and RPT of the thread's columns.
template <typename T, int RPT, bool PART, typename E>
__device__ __forceinline__ void region_rows(E& sh, int& buf, int w, int lane, const Region<T, RPT>& g,
                                            int nw, T (&below)[2], T (&above)[2]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    sh.bot[buf][w][q][lane] = g.e[RPT - 1][q];
    sh.top[buf][w][q][lane] = g.e[0][q];
  }
  region_barrier<PART>(32 * nw);
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    below[q] = pick_bits(w, ~0u, sh.bot[buf][max(w - 1, 0)][q][lane], (T)0);
    above[q] = pick_bits(nw - 1 - w, ~0u, sh.top[buf][min(w + 1, nw - 1)][q][lane], (T)0);
  }
  buf ^= 1;
}

// -(A e) of the thread's cells: the sum over open faces of e_nb - e (0 off the fluid).
template <typename T, int RPT>
__device__ __forceinline__ void region_minus_ae(const Region<T, RPT>& g, int lane, const T (&below)[2],
                                                const T (&above)[2], T (&out)[RPT][2]) {
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const T fl = from_left(g.e[r][1], lane), fr = from_right(g.e[r][0], lane);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t k = g.c(r, q);
      const T x = g.e[r][q];
      const T l = q == 0 ? fl : g.e[r][0], rt = q == 0 ? g.e[r][1] : fr;
      const T d = r > 0 ? g.e[r > 0 ? r - 1 : 0][q] : below[q];
      const T u = r < RPT - 1 ? g.e[r < RPT - 1 ? r + 1 : r][q] : above[q];
      // differences, not a sum less n x: they stay exact near convergence, where the sum cancels
      T s = (T)0;
      s += pick_bits(k, C_L, l - x, (T)0);
      s += pick_bits(k, C_R, rt - x, (T)0);
      s += pick_bits(k, C_D, d - x, (T)0);
      s += pick_bits(k, C_U, u - x, (T)0);
      out[r][q] = pick_bits(k, C_FLUID, s, (T)0);
    }
  }
}

// Full weighting of the residual b - A e: store(m, v) gets the coarse value of the thread's
// fine rows 2m, 2m + 1. j, i: the thread's first cell; H, W, Hc, Wc: the two levels. The
// weights are those of the bilinear prolongation with candidates clamped to the grid
// (separable); where a candidate is not fluid, its share is added to the home cell.
template <typename T, int RPT, bool PART, typename E, typename F>
__device__ __forceinline__ void region_restrict(E& sh, int& buf, int w, int lane, const Region<T, RPT>& g,
                                                int nw, int j, int i, int H, int W, int Hc, int Wc, F store) {
  T below[2], above[2], res[RPT][2];
  region_rows<T, RPT, PART>(sh, buf, w, lane, g, nw, below, above);
  region_minus_ae<T, RPT>(g, lane, below, above, res);
  const int I = i >> 1;
  // w1 of fine columns 2I - 1 .. 2I + 2 (0 off the grid): a fine cell's outer candidate is
  // clamped to its home one at an edge
  const T wx0 = I > 0 ? (T)0.25 : (T)0, wx3 = 2 * I + 2 < W ? (T)0.25 : (T)0;
  const T wx1 = I > 0 ? (T)0.75 : (T)1, wx2 = I < Wc - 1 ? (T)0.75 : (T)1;
  T X[RPT], home[RPT / 2];
  uint32_t fluid[RPT / 2];
#pragma unroll
  for (int m = 0; m < RPT / 2; ++m) {
    home[m] = (T)0;
    fluid[m] = 0;
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const uint32_t k = g.c(r, q);
      res[r][q] += pick_bits(k, C_FLUID, g.b[r][q], (T)0);
      fluid[r >> 1] |= k;
      const T extra = pick_bits(k, C_XHOME, (T)(3.0 / 16), (T)0) + pick_bits(k, C_YHOME, (T)(3.0 / 16), (T)0) +
                      pick_bits(k, C_DHOME, (T)(1.0 / 16), (T)0);
      home[r >> 1] += extra * res[r][q];
    }
    const T rl = from_left(res[r][1], lane), rr = from_right(res[r][0], lane);
    T acc = wx0 * rl;
    acc += wx1 * res[r][0];
    acc += wx2 * res[r][1];
    acc += wx3 * rr;
    X[r] = acc;
  }
  sh.bot[buf][w][0][lane] = X[RPT - 1];
  sh.top[buf][w][0][lane] = X[0];
  region_barrier<PART>(32 * nw);
  const T xa = pick_bits(w, ~0u, sh.bot[buf][max(w - 1, 0)][0][lane], (T)0);
  const T xb = pick_bits(nw - 1 - w, ~0u, sh.top[buf][min(w + 1, nw - 1)][0][lane], (T)0);
  buf ^= 1;
#pragma unroll
  for (int m = 0; m < RPT / 2; ++m) {
    const int J = (j >> 1) + m;
    const T wy0 = J > 0 ? (T)0.25 : (T)0, wy3 = 2 * J + 2 < H ? (T)0.25 : (T)0;
    const T wy1 = J > 0 ? (T)0.75 : (T)1, wy2 = J < Hc - 1 ? (T)0.75 : (T)1;
    T acc = wy0 * (m > 0 ? X[m > 0 ? 2 * m - 1 : 0] : xa);
    acc += wy1 * X[2 * m];
    acc += wy2 * X[2 * m + 1];
    acc += wy3 * (2 * m + 2 < RPT ? X[2 * m + 2 < RPT ? 2 * m + 2 : 0] : xb);
    store(m, pick_bits(fluid[m], C_FLUID, acc + home[m], (T)0));
  }
}

// e += P ec on the thread's fluid cells. coarse(J, lane's left, own and right column): the
// three values of coarse row J (clamped) around the lane's coarse column, edge columns clamped.
template <typename T, int RPT, typename F>
__device__ __forceinline__ void region_prolong(Region<T, RPT>& g, int j, F coarse) {
  const T w9 = (T)(9.0 / 16.0), w3 = (T)(3.0 / 16.0), wd = (T)(1.0 / 16.0);
  T pl, pm, pr, cl, cm, cr;
  coarse((j >> 1) - 1, pl, pm, pr);
  coarse(j >> 1, cl, cm, cr);
#pragma unroll
  for (int m = 0; m < RPT / 2; ++m) {
    T nl, nm, nr;
    coarse((j >> 1) + m + 1, nl, nm, nr);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = 2 * m + h;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t k = g.c(r, q);
        const T x = q == 0 ? cl : cr, y = h == 0 ? pm : nm;
        const T d = h == 0 ? (q == 0 ? pl : pr) : (q == 0 ? nl : nr);
        T acc = w9 * cm;
        acc += w3 * pick_bits(k, C_XHOME, cm, x);
        acc += w3 * pick_bits(k, C_YHOME, cm, y);
        acc += wd * pick_bits(k, C_DHOME, cm, d);
        g.e[r][q] = g.e[r][q] + pick_bits(k, C_FLUID, acc, (T)0);
      }
    }
    pl = cl;
    pm = cm;
    pr = cr;
    cl = nl;
    cm = nm;
    cr = nr;
  }
}

// ------------------------------------------------------------------ level kernels
template <typename T>
struct RegionArgs {
  RegionLevel m;
  int Hc, Wc;
  int64_t ld, ldc;
  const T* e_in;   // null: from zero
  T* e_out;        // FINAL: not written
  const T* b;
  T* bc;           // pre: the coarse rhs
  const T* ec;     // post: the coarse correction
  T omega;
  int sweeps, halo;
  const GmgState* st;
};

// The block's place: its first row and column, and the range it owns.
struct RegionPlace {
  int w, lane, j, i, oy0, oy1;
  bool own_col;
  template <typename T>
  __device__ __forceinline__ void set(const RegionArgs<T>& a) {
    constexpr int RR = kRgWarps * kRgRows;
    lane = threadIdx.x & 31;
    w = threadIdx.x >> 5;
    const int r0 = blockIdx.y * (RR - 2 * a.halo), c0 = blockIdx.x * (kRgCols - 2 * a.halo);
    j = r0 + w * kRgRows;
    i = c0 + 2 * lane;
    oy0 = blockIdx.y == 0 ? 0 : r0 + a.halo;
    oy1 = blockIdx.y == gridDim.y - 1 ? a.m.H : r0 + RR - a.halo;
    own_col = i >= (blockIdx.x == 0 ? 0 : c0 + a.halo) &&
              i < (blockIdx.x == gridDim.x - 1 ? a.m.W : c0 + kRgCols - a.halo);
  }
};

template <typename T>
__device__ __forceinline__ void region_load(Region<T, kRgRows>& g, const RegionArgs<T>& a, const RegionPlace& at) {
#pragma unroll
  for (int r = 0; r < kRgRows; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int64_t o = (int64_t)min(at.j + r, a.m.H - 1) * a.ld + min(at.i + q, a.m.W - 1);
      g.b[r][q] = a.b[o];
      g.e[r][q] = a.e_in ? a.e_in[o] : (T)0;
    }
#pragma unroll
  for (int r = 0; r < kRgRows; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (at.j + r >= a.m.H || at.i + q >= a.m.W) g.b[r][q] = g.e[r][q] = (T)0;
  g.set_codes(a.m, at.j, at.i, a.omega);
}

template <typename T>
__device__ __forceinline__ void region_store(const Region<T, kRgRows>& g, const RegionArgs<T>& a,
                                             const RegionPlace& at) {
  if (!at.own_col) return;
#pragma unroll
  for (int r = 0; r < kRgRows; ++r) {
    const int jj = at.j + r;
    if (jj < at.oy0 || jj >= at.oy1 || !SG_IN_BOUNDS(jj < a.m.H && at.i < a.m.W)) continue;
    T* o = a.e_out + (int64_t)jj * a.ld + at.i;
    o[0] = g.e[r][0];
    if (at.i + 1 < a.m.W) o[1] = g.e[r][1];
  }
}

template <typename T>
__global__ void __launch_bounds__(kRgThreads) k_gmg_pre_region(const __grid_constant__ RegionArgs<T> a) {
  __shared__ RegionEdges<T, kRgWarps> sh;
  RegionPlace at;
  at.set(a);
  Region<T, kRgRows> g;
  region_load(g, a, at);
  int buf = 0;
  region_sweeps<T, kRgRows, false>(sh, buf, at.w, at.lane, g, a.sweeps, kRgWarps);
  region_store(g, a, at);
  region_restrict<T, kRgRows, false>(sh, buf, at.w, at.lane, g, kRgWarps, at.j, at.i, a.m.H, a.m.W, a.Hc, a.Wc,
                                     [&](int m, T v) {
                                       const int jj = at.j + 2 * m, J = jj >> 1, I = at.i >> 1;
                                       if (at.own_col && jj >= at.oy0 && jj < at.oy1 && J < a.Hc &&
                                           SG_IN_BOUNDS(I < a.Wc))
                                         a.bc[(int64_t)J * a.ldc + I] = v;
                                     });
}

// FINAL: the fine level of a solve, which adds e to p (in TP) instead of storing it. The residual
// is formed from p afresh after every cycle, so that what a solve reports is its pressure's own:
// carried on as r - A e it went on falling where p no longer gained, and p ended further off
// (200 x 256 float64, 1e-15 asked: 5e-16 reported and 5.5e-12 true after 19 cycles; 7.6e-13 both so).
template <typename T, typename TP, bool FINAL>
__global__ void __launch_bounds__(kRgThreads) k_gmg_post_region(const __grid_constant__ RegionArgs<T> a) {
  __shared__ RegionEdges<T, kRgWarps> sh;
  RegionPlace at;
  at.set(a);
  Region<T, kRgRows> g;
  region_load(g, a, at);
  const int I = at.i >> 1, Ic = min(I, a.Wc - 1);
  const int Iedge = at.lane == 0 ? max(I - 1, 0) : min(I + 1, a.Wc - 1);
  const bool edge = at.lane == 0 || at.lane == 31;
  region_prolong<T, kRgRows>(g, at.j, [&](int J, T& l, T& m, T& r) {
    const T* row = a.ec + (int64_t)min(max(J, 0), a.Hc - 1) * a.ldc;
    m = row[Ic];
    const T ve = edge ? row[min(Iedge, a.Wc - 1)] : (T)0;
    const T lv = __shfl_up_sync(0xffffffffu, m, 1), rv = __shfl_down_sync(0xffffffffu, m, 1);
    l = at.lane == 0 ? ve : lv;
    r = at.lane == 31 ? ve : rv;
  });
  int buf = 0;
  region_sweeps<T, kRgRows, false>(sh, buf, at.w, at.lane, g, a.sweeps, kRgWarps);
  if constexpr (!FINAL) {
    region_store(g, a, at);
  } else if (at.own_col) {
    TP* p = (TP*)a.st->f.p;
    const int64_t ldp = a.st->f.ldp;
#pragma unroll
    for (int r = 0; r < kRgRows; ++r) {
      const int jj = at.j + r;
      if (jj < at.oy0 || jj >= at.oy1 || !SG_IN_BOUNDS(jj < a.m.H && at.i < a.m.W)) continue;
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (at.i + q < a.m.W) p[(int64_t)jj * ldp + at.i + q] += (TP)g.e[r][q];
    }
  }
}

// ------------------------------------------------------------------ tail
constexpr int kRgTailSide = 64;
constexpr int kRgTailRows = 2;
constexpr int kRgTailWarps = kRgTailSide / kRgTailRows;
constexpr int kRgTailThreads = 32 * kRgTailWarps;
constexpr int kRgPinvShared = 64;  // coarsest cells up to which the pseudo-inverse is kept in shared memory

template <typename T>
struct RegionTailArgs {
  int n;  // levels; the last one is the coarsest (exact solve)
  RegionLevel m[kMaxLevels];
  int off[kMaxLevels];  // the level's first cell in the shared arrays
  int cells;
  T* ge;                // the first level in global memory (e in/out, b in)
  const T* gb;
  int64_t gld;
  const double* pinv;
  T omega;
  int pre, post, wcycle, zero_init;
};

template <typename T>
static size_t region_tail_smem(int cells, int coarsest_cells) {
  const int pinv = coarsest_cells <= kRgPinvShared ? coarsest_cells * coarsest_cells : 0;
  return sizeof(RegionEdges<T, kRgTailWarps>) + (size_t)pinv * 8 + (size_t)cells * 2 * sizeof(T);
}

template <typename T>
struct RegionTailShared {
  double* pinv;
  T* e;
  T* b;
  // the level table, copied here: parameters indexed by a run-time level are slow constant
  // loads (32^2 visit: 1400 of 4900 clocks for the codes alone)
  RegionLevel m[kMaxLevels];
  int off[kMaxLevels];
};

// Level l: its pre side (sweeps from e, or from zero; the next level's rhs) or its post side.
template <typename T>
__device__ __forceinline__ void region_tail_visit(const RegionTailArgs<T>& a, const RegionTailShared<T>& t,
                                                  RegionEdges<T, kRgTailWarps>& sh, int l, bool post, bool zero) {
  constexpr int RPT = kRgTailRows;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const RegionLevel m = t.m[l];
  const int H = m.H, W = m.W, Hc = t.m[l + 1].H, Wc = t.m[l + 1].W, o = t.off[l], oc = t.off[l + 1];
  const int nw = (H + RPT - 1) / RPT;
  if (w >= nw) return;
  const int j = w * RPT, i = 2 * lane;
  Region<T, RPT> g;
  // the first level's rhs (and its start value) stay in global memory, the others' lie in the
  // shared arrays; clamped addresses, so that all loads are in flight at once
  const int j1 = min(j + 1, H - 1), i0 = min(i, W - 1), i1 = min(i + 1, W - 1);
  static_assert(RPT == 2, "rows j and j1");
  if (l == 0) {
    const int64_t r0 = j * a.gld, r1 = j1 * a.gld;
    g.b[0][0] = a.gb[r0 + i0], g.b[0][1] = a.gb[r0 + i1], g.b[1][0] = a.gb[r1 + i0], g.b[1][1] = a.gb[r1 + i1];
    if (!post && !zero)
      g.e[0][0] = a.ge[r0 + i0], g.e[0][1] = a.ge[r0 + i1], g.e[1][0] = a.ge[r1 + i0], g.e[1][1] = a.ge[r1 + i1];
  } else {
    const T* bs = t.b + o;
    const int r0 = j * W, r1 = j1 * W;
    g.b[0][0] = bs[r0 + i0], g.b[0][1] = bs[r0 + i1], g.b[1][0] = bs[r1 + i0], g.b[1][1] = bs[r1 + i1];
  }
  if (zero) {
    g.e[0][0] = g.e[0][1] = g.e[1][0] = g.e[1][1] = (T)0;
  } else if (post || l > 0) {
    const T* es = t.e + o;
    const int r0 = j * W, r1 = j1 * W;
    g.e[0][0] = es[r0 + i0], g.e[0][1] = es[r0 + i1], g.e[1][0] = es[r1 + i0], g.e[1][1] = es[r1 + i1];
  }
  g.set_codes(m, j, i, a.omega);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (j + r >= H || i + q >= W) g.b[r][q] = g.e[r][q] = (T)0;
  if (post) {
    const int I = min(i >> 1, Wc - 1), Il = max((i >> 1) - 1, 0), Ir = min((i >> 1) + 1, Wc - 1);
    region_prolong<T, RPT>(g, j, [&](int J, T& cl, T& cm, T& cr) {
      const T* row = t.e + oc + min(max(J, 0), Hc - 1) * Wc;
      cl = row[min(Il, Wc - 1)];
      cm = row[I];
      cr = row[Ir];
    });
  }
  int buf = 0;
  region_sweeps<T, RPT, true>(sh, buf, w, lane, g, post ? a.post : a.pre, nw);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (j + r < H && i + q < W && SG_IN_BOUNDS(o + (j + r) * W + i + q < a.cells)) {
        if (post && l == 0)
          a.ge[(int64_t)(j + r) * a.gld + i + q] = g.e[r][q];
        else
          t.e[o + (j + r) * W + i + q] = g.e[r][q];
      }
  if (post) return;
  region_restrict<T, RPT, true>(sh, buf, w, lane, g, nw, j, i, H, W, Hc, Wc, [&](int m, T v) {
    const int J = (j >> 1) + m, I = i >> 1;
    if (J < Hc && I < Wc && SG_IN_BOUNDS(oc + J * Wc + I < a.cells)) t.b[oc + J * Wc + I] = v;
  });
}

// The warps whose rows lie beyond a level wait for the others at the visit's end. Two rows a
// thread: what a small level costs is the length of one warp's instruction stream. That stream
// has no branch that lanes could part at: as ternaries, the edge tests of codes, weights,
// residual and prolongation were branches that the grid's edge lanes took apart from the others
// (64^2 down, float32: 17.8 us with them, 15.2 us with selects).
template <typename T>
__global__ void __launch_bounds__(kRgTailThreads) k_gmg_tail_region(const __grid_constant__ RegionTailArgs<T> a) {
  extern __shared__ __align__(16) unsigned char region_smem[];
  RegionEdges<T, kRgTailWarps>& sh = *reinterpret_cast<RegionEdges<T, kRgTailWarps>*>(region_smem);
  const int last = a.n - 1, nc = a.m[last].H * a.m[last].W;
  const bool keep = nc <= kRgPinvShared;
  __shared__ RegionTailShared<T> t;
  double* const pinv_s = reinterpret_cast<double*>(region_smem + sizeof(sh));
  const int tid = threadIdx.x;
  if (tid == 0) {
    t.pinv = pinv_s;
    t.e = reinterpret_cast<T*>(pinv_s + (keep ? nc * nc : 0));
    t.b = t.e + a.cells;
  }
  if (tid < a.n) {
    t.m[tid] = a.m[tid];
    t.off[tid] = a.off[tid];
  }
  if (keep)  // lands while the levels above run
    for (int q = tid; q < nc * nc; q += kRgTailThreads)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(pinv_s + q)), "l"(a.pinv + q) : "memory");
  __syncthreads();
  int l = 0;
  bool down = true;
  unsigned second = 0;  // bit l: level l already sent its first visit to level l + 1
  unsigned fresh = a.zero_init ? ~0u : ~1u;  // bit l: level l starts from zero
  while (true) {
    if (l == last) {  // e = pinv b, eight threads a row
      asm volatile("cp.async.wait_all;" ::: "memory");
      __syncthreads();
      const T* bc = last == 0 ? a.gb : t.b + t.off[l];
      const int Wl = t.m[l].W;
      const double* pinv = keep ? t.pinv : a.pinv;
      for (int row = tid >> 3; row < ((nc + 127) & ~127); row += kRgTailThreads / 8) {
        double acc = 0.0;
        if (row < nc)
          for (int q = tid & 7; q < nc; q += 8)
            acc += pinv[(int64_t)row * nc + q] * (double)(last == 0 ? bc[(int64_t)(q / Wl) * a.gld + q % Wl] : bc[q]);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (row < nc && (tid & 7) == 0) {
          if (last == 0)
            a.ge[(int64_t)(row / a.m[0].W) * a.gld + row % a.m[0].W] = (T)acc;
          else
            t.e[t.off[l] + row] = (T)acc;
        }
      }
      __syncthreads();
      if (l == 0) break;
      --l;
      down = false;
      continue;
    }
    if (!down && a.wcycle && l + 1 < last && !((second >> l) & 1u)) {  // the second visit below
      second |= 1u << l;
      ++l;
      fresh &= ~(1u << l);
      down = true;
      continue;
    }
    const bool zero = down && ((fresh >> l) & 1u);
    region_tail_visit<T>(a, t, sh, l, !down, zero);
    __syncthreads();
    if (down) {
      second &= ~(1u << l);
      ++l;
      fresh |= 1u << l;
    } else {
      if (l == 0) break;
      --l;
    }
  }
}
