// Sweeps with the iterate held on the chip (sweeps.cu), for the solver entry points.
#pragma once

#include "common.cuh"

namespace sg {

// Per-cell code: the open faces towards a neighbour inside the grid, and whether the cell is
// fluid. A closed face, and an open one at the grid's edge (whose clamped neighbour is the
// cell itself), both contribute the cell's own value.
enum : uint32_t { K_L = 1, K_R = 2, K_D = 4, K_U = 8, K_FLUID = 16, K_ALL = 31 };

__device__ __forceinline__ uint32_t faces_code(bool l, bool r, bool d, bool u, int H, int W, int j, int i) {
  uint32_t c = 0;
  if (l && i > 0) c |= K_L;
  if (r && i < W - 1) c |= K_R;
  if (d && j > 0) c |= K_D;
  if (u && j < H - 1) c |= K_U;
  if (l || r || d || u) c |= K_FLUID;
  return c;
}
__device__ __forceinline__ uint32_t cell_code(const Masks& m, int H, int W, int j, int i) {
  return faces_code(m.u(j, i), m.u(j, i + 1), m.v(j, i), m.v(j + 1, i), H, W, j, i);
}

// Rows per thread of the resident sweeps on an H x W grid, 0 when it does not fit the chip,
// and the bytes of the buffer through which their blocks trade.
int resident_rows(int64_t H, int64_t W);
int64_t resident_workspace_bytes(int64_t elem, int64_t H, int64_t W);

constexpr int kResidentSweeps = 1 << 14;  // sweeps of one resident launch (some tens of ms)
// Trades that a launch of so many sweeps makes (each takes one tag).
int resident_trades(int sor, int sweeps);

// `sweeps` Jacobi (sor = 0) or red-black SOR sweeps of p in place. split: p, p1 and b, b1 are
// colour planes. Launches of kResidentSweeps. xchg: resident_workspace_bytes bytes, zeroed before
// the first call that uses it; *tag: 1 + the trades of the calls before on the same buffer, moved
// on. from_zero: p is 0 and not read.
template <typename T>
int resident_sweeps(int sor, int split, int H, int W, T* p, T* p1, int64_t ldp, const T* b, const T* b1, int64_t ldb,
                    const Masks& m, double alpha, double rb, double omega, int64_t sweeps, bool from_zero, void* xchg,
                    uint32_t* tag, cudaStream_t s);

// Red-black SOR sweeps of the colour planes p0, p1 until the residual's norm over r0 is at most
// tol: checked after every check_every sweeps, at most max_sweeps of them (a multiple of
// check_every, or fewer). best, stalls, stall_limit: also stops when stall_limit checks in a row
// gained less than 1 % on the best one (0: never).
struct SweepsUntil {
  double r0, tol, best;
  int check_every, max_sweeps, stalls, stall_limit;
};
struct SweepsReached {
  double sq, best;  // the last check's sum of squares
  int64_t sweeps, stalls;
};
bool resident_until_fits(int64_t H, int64_t W);
template <typename T>
int resident_sweeps_until(int H, int W, T* p0, T* p1, int64_t ldp, const T* b0, const T* b1, int64_t ldb,
                          const Masks& m, double alpha, double rb, double beta, double omega, const SweepsUntil& u,
                          void* xchg, uint32_t tag, SweepsReached* reached, cudaStream_t s);

// SMs of the current device (0: unknown).
int sm_count();

// Lexicographic Gauss-Seidel sweeps; *ran is false when the grid is too wide for it.
// workspace: gauss_seidel_workspace bytes (M: the shorter side; 0: none needed), cleared by the
// call, or null for one block.
template <typename T>
int64_t gauss_seidel_workspace(int M, int iterations);
template <typename T>
int gauss_seidel_wave(int H, int W, T* p, int64_t ldp, const T* div, int64_t ldd, const Masks& m, double alpha,
                      double rb, int iterations, void* workspace, bool* ran, cudaStream_t s);

}  // namespace sg
