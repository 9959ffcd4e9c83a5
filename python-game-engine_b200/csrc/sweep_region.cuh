// Red-black SOR half sweeps and Jacobi sweeps on a region of cells that a block holds in
// registers: 16 warps of RPT rows x 64 columns; lane l of warp w has columns i0 + 2l,
// i0 + 2l + 1 of rows j0 + w RPT .. + RPT - 1 (j0, i0 and RPT even, so the colour of a
// register cell is known at compile time). For units compiled with -fmad=false: the updates
// are the reference's expressions in the reference's order.
#pragma once

#include "sweeps.cuh"

namespace sg {

constexpr int kResWarps = 16;
constexpr int kResThreads = 32 * kResWarps;
constexpr int kResCols = 64;

// Tile t of an axis of n cells covers [t own, t own + span), own = span - 2 halo, and owns what
// lies halo or more inside, plus everything up to a grid edge.
__host__ __device__ inline int res_tiles(int n, int span, int halo) {
  const int own = span - 2 * halo;
  return n <= span ? 1 : (n - 2 * halo + own - 1) / own;
}

template <typename T>
struct ResEdges {  // first and last row of each warp, double-buffered; SOR uses one column of two
  T top[2][kResWarps][2][32];
  T bot[2][kResWarps][2][32];
};

// v where the bit is set, else c, without a branch around what v took to compute
__device__ __forceinline__ float pick(uint32_t bit, float v, float c) {
  float o;
  asm("{.reg .pred p; setp.ne.u32 p, %1, 0; selp.f32 %0, %2, %3, p;}" : "=f"(o) : "r"(bit), "f"(v), "f"(c));
  return o;
}
__device__ __forceinline__ double pick(uint32_t bit, double v, double c) {
  double o;
  asm("{.reg .pred p; setp.ne.u32 p, %1, 0; selp.f64 %0, %2, %3, p;}" : "=d"(o) : "r"(bit), "d"(v), "d"(c));
  return o;
}

// One half sweep of colour COL (SOR), or one whole sweep (Jacobi), over the thread's cells,
// with the trade of the warps' edge rows. CODED: faces by the cells' codes (five bits a cell,
// four cells a word); otherwise every cell is updated and all its faces are open but those of
// column 0 (edge0) and of the last column (edge1: the lane's second one).
// Written stage by stage over the rows, so that the rows' chains overlap, with all that does
// not need another warp's row ahead of the barrier: the shuffles, the sum's first term and the
// old value's share. A half sweep reads one colour of its neighbours' rows, so that is all the
// warps store. (float32 SOR at 128^2: 0.65 us a sweep, 0.73 row by row with whole rows stored.)
//   res_ahead  stores the edge rows and does what comes ahead of the barrier
//   res_after  the rest
template <typename T, bool SOR, int COL, int RPT, bool CODED>
__device__ __forceinline__ void res_ahead(ResEdges<T>& sh, int buf, int w, int lane, const T (&e)[RPT][2],
                                          const uint32_t* code, bool edge0, bool edge1, double keep,
                                          T (&s)[RPT][SOR ? 1 : 2], double (&x)[RPT][SOR ? 1 : 2]) {
  constexpr int Q = SOR ? 1 : 2;  // updated cells per row
  if (SOR) {
    sh.bot[buf][w][0][lane] = e[RPT - 1][COL];  // for the next warp's first row
    sh.top[buf][w][0][lane] = e[0][1 - COL];    // for the previous warp's last row
  } else {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      sh.bot[buf][w][q][lane] = e[RPT - 1][q];
      sh.top[buf][w][q][lane] = e[0][q];
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const int q = SOR ? (COL + r) & 1 : n;
      const T far = q == 0 ? __shfl_up_sync(0xffffffffu, e[r][1], 1) : __shfl_down_sync(0xffffffffu, e[r][0], 1);
      const T c = e[r][q];
      T l = q == 0 ? far : e[r][0];
      T rt = q == 0 ? e[r][1] : far;
      if (CODED) {
        const uint32_t k = code[r >> 1] >> (10 * (r & 1) + 5 * q);
        l = pick(k & K_L, l, c);
        rt = pick(k & K_R, rt, c);
      } else {
        if (q == 0) l = edge0 ? c : l;
        if (q == 1) rt = edge1 ? c : rt;
      }
      s[r][n] = l + rt;
      if (SOR) x[r][n] = keep * (double)c;
    }
  }
}

template <typename T, bool SOR, int COL, int RPT, bool CODED>
__device__ __forceinline__ void res_after(const ResEdges<T>& sh, int buf, int w, int lane, T (&e)[RPT][2],
                                          const double (&ab)[RPT][2], const uint32_t* code, double rb, double omega,
                                          T (&s)[RPT][SOR ? 1 : 2], double (&x)[RPT][SOR ? 1 : 2]) {
  constexpr int Q = SOR ? 1 : 2;
  const int wb = w > 0 ? w - 1 : w, wa = w < kResWarps - 1 ? w + 1 : w;
  T below[Q], above[Q];
#pragma unroll
  for (int n = 0; n < Q; ++n) {
    below[n] = sh.bot[buf][wb][n][lane];
    above[n] = sh.top[buf][wa][n][lane];
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const int q = SOR ? (COL + r) & 1 : n;
      T d = r > 0 ? e[r > 0 ? r - 1 : 0][q] : below[n];
      T u = r < RPT - 1 ? e[r < RPT - 1 ? r + 1 : r][q] : above[n];
      if (CODED) {
        const uint32_t k = code[r >> 1] >> (10 * (r & 1) + 5 * q);
        d = pick(k & K_D, d, e[r][q]);
        u = pick(k & K_U, u, e[r][q]);
      }
      s[r][n] = s[r][n] + d;
      s[r][n] = s[r][n] + u;
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const int q = SOR ? (COL + r) & 1 : n;
      const double np_ = ((double)s[r][n] + ab[r][q]) * rb;
      x[r][n] = SOR ? x[r][n] + omega * np_ : np_;
    }
  }
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const int q = SOR ? (COL + r) & 1 : n;
      const T v = (T)x[r][n];
      e[r][q] = CODED ? pick((code[r >> 1] >> (10 * (r & 1) + 5 * q)) & K_FLUID, v, e[r][q]) : v;
    }
  }
}

// Barrier of the block, or (PART) of its first `threads` threads, when the warps beyond them
// hold no cells of the grid and skip the sweeps.
template <bool PART>
__device__ __forceinline__ void res_barrier(int threads) {
  if (PART)
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  else
    __syncthreads();
}

// n half sweeps (SOR; even, red first) or n sweeps (Jacobi). plain: the warp takes the form
// without codes (uniform over the warp). buf: the edge buffer to use next.
template <typename T, bool SOR, int RPT, bool PART = false>
__device__ __forceinline__ void res_sweeps(ResEdges<T>& sh, int& buf, int w, int lane, T (&e)[RPT][2],
                                           const double (&ab)[RPT][2], const uint32_t* code, bool plain, bool edge0,
                                           bool edge1, double rb, double omega, double keep, int n, int threads = 0) {
  for (int h = 0; h < n; h += 2) {
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      if (!SOR && h + c >= n) break;
      T sum[RPT][SOR ? 1 : 2];
      double x[RPT][SOR ? 1 : 2];
      if (plain) {
        if (c == 0)
          res_ahead<T, SOR, 0, RPT, false>(sh, buf, w, lane, e, code, edge0, edge1, keep, sum, x);
        else
          res_ahead<T, SOR, 1, RPT, false>(sh, buf, w, lane, e, code, edge0, edge1, keep, sum, x);
      } else {
        if (c == 0)
          res_ahead<T, SOR, 0, RPT, true>(sh, buf, w, lane, e, code, edge0, edge1, keep, sum, x);
        else
          res_ahead<T, SOR, 1, RPT, true>(sh, buf, w, lane, e, code, edge0, edge1, keep, sum, x);
      }
      res_barrier<PART>(threads);
      if (plain) {
        if (c == 0)
          res_after<T, SOR, 0, RPT, false>(sh, buf, w, lane, e, ab, code, rb, omega, sum, x);
        else
          res_after<T, SOR, 1, RPT, false>(sh, buf, w, lane, e, ab, code, rb, omega, sum, x);
      } else {
        if (c == 0)
          res_after<T, SOR, 0, RPT, true>(sh, buf, w, lane, e, ab, code, rb, omega, sum, x);
        else
          res_after<T, SOR, 1, RPT, true>(sh, buf, w, lane, e, ab, code, rb, omega, sum, x);
      }
      buf ^= 1;
    }
  }
}

// The code of column i + q of row r in the thread's words.
__device__ __forceinline__ uint32_t res_code(const uint32_t* code, int r, int q) {
  return (code[r >> 1] >> (10 * (r & 1) + 5 * q)) & K_ALL;
}

// Whether the warp's cells are all inside the grid and fluid with every face open but the
// grid's left and right edges: then res_sweeps needs no codes. k: the cell's code. Column i is
// never the last one of such a warp (odd W: the last pair stays coded).
__device__ __forceinline__ bool res_is_plain(uint32_t k, int ii, int W) {
  return k == (K_ALL & ~(ii == 0 ? (uint32_t)K_L : 0u) & ~(ii == W - 1 ? (uint32_t)K_R : 0u));
}

// Residual of every cell of the thread (residual.py:39-40; 0 off the fluid). cells: bit
// 2 r + q, whether the cell is fluid there.
template <typename T, int RPT, bool PART = false>
__device__ __forceinline__ void res_residual(ResEdges<T>& sh, int& buf, int w, int lane, const T (&e)[RPT][2],
                                             const double (&ab)[RPT][2], const uint32_t* code, uint32_t cells,
                                             double beta, T (&res)[RPT][2], int threads = 0) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    sh.bot[buf][w][q][lane] = e[RPT - 1][q];
    sh.top[buf][w][q][lane] = e[0][q];
  }
  res_barrier<PART>(threads);
  const int wb = w > 0 ? w - 1 : w, wa = w < kResWarps - 1 ? w + 1 : w;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const T fl = __shfl_up_sync(0xffffffffu, e[r][1], 1), fr = __shfl_down_sync(0xffffffffu, e[r][0], 1);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const T c = e[r][q];
      const uint32_t k = res_code(code, r, q);
      const T l = pick(k & K_L, q == 0 ? fl : e[r][0], c);
      const T rt = pick(k & K_R, q == 0 ? e[r][1] : fr, c);
      const T d = pick(k & K_D, r > 0 ? e[r > 0 ? r - 1 : 0][q] : sh.bot[buf][wb][q][lane], c);
      const T u = pick(k & K_U, r < RPT - 1 ? e[r < RPT - 1 ? r + 1 : r][q] : sh.top[buf][wa][q][lane], c);
      T s = l + rt;
      s = s + d;
      s = s + u;
      res[r][q] = pick(cells >> (2 * r + q) & 1, (T)(((double)s + ab[r][q]) - beta * (double)c), (T)0);
    }
  }
  buf ^= 1;
}

// The thread's share of the residual's sum of squares: rows [r_lo, r_hi) of its columns, each
// residual rounded as above. The edge rows must have come with res_edges and a barrier.
template <typename T, int RPT>
__device__ __forceinline__ void res_edges(ResEdges<T>& sh, int buf, int w, int lane, const T (&e)[RPT][2]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    sh.bot[buf][w][q][lane] = e[RPT - 1][q];
    sh.top[buf][w][q][lane] = e[0][q];
  }
}
template <typename T, int RPT>
__device__ __forceinline__ double res_sumsq(const ResEdges<T>& sh, int buf, int w, int lane, const T (&e)[RPT][2],
                                            const double (&ab)[RPT][2], const uint32_t* code, double beta, int r_lo,
                                            int r_hi) {
  const int wb = w > 0 ? w - 1 : w, wa = w < kResWarps - 1 ? w + 1 : w;
  double sq = 0.0;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const T fl = __shfl_up_sync(0xffffffffu, e[r][1], 1), fr = __shfl_down_sync(0xffffffffu, e[r][0], 1);
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const T c = e[r][q];
      const uint32_t k = res_code(code, r, q);
      const T l = pick(k & K_L, q == 0 ? fl : e[r][0], c);
      const T rt = pick(k & K_R, q == 0 ? e[r][1] : fr, c);
      const T d = pick(k & K_D, r > 0 ? e[r > 0 ? r - 1 : 0][q] : sh.bot[buf][wb][q][lane], c);
      const T u = pick(k & K_U, r < RPT - 1 ? e[r < RPT - 1 ? r + 1 : r][q] : sh.top[buf][wa][q][lane], c);
      T s = l + rt;
      s = s + d;
      s = s + u;
      const T x = (T)(((double)s + ab[r][q]) - beta * (double)c);
      if (r >= r_lo && r < r_hi) sq += pick(k & K_FLUID, (double)x * (double)x, 0.0);
    }
  }
  return sq;
}

}  // namespace sg
