// Fixed-count sweeps with the iterate held on the chip: Jacobi (jacobi.py:8-24) and red-black
// SOR (red_black_sor_gauss_seidel.py:8-27), all sweeps of a call in one cooperative launch,
// the cells in registers.
//
// Every update evaluates the reference's expression in the reference's order (masked
// neighbour sum in T, l + r + d + up; the rest in double; one rounding to T), so the iterates
// are those of the one-launch-per-sweep kernels bit for bit. Compiled with -fmad=false like
// the other operator units.
#include <algorithm>
#include <type_traits>

#include "sweeps.cuh"
#include "sweep_region.cuh"
#include "waits.cuh"

namespace sg {

// ------------------------------------------------------------------ resident sweeps
// A block of 16 warps holds a region of 16 RPT rows x 64 columns in registers: lane l of warp
// w has columns i0 + 2l, i0 + 2l + 1 of rows j0 + w RPT .. + RPT - 1 (j0, i0 and RPT even, so
// the colour of a register cell is known at compile time). Horizontal neighbours come by
// shuffle, vertical ones from the thread's own registers or, at a warp's first and last row,
// through shared memory with one barrier per half sweep (Jacobi: per sweep). The region
// overlaps its neighbours' by kHalo cells on each side inside the grid: values grown wrong
// from its edge move in one cell per half sweep, so after kHalo of them the block's own cells
// still hold exactly the grid-wide iterates. Then the blocks trade the kHalo-wide frames of
// their own cells and go on.
//
// What bounds it: a call is a chain of `sweeps` dependent sweeps of grids that sit on the
// chip, so its time is the chain's latency: barrier, shuffle and the float64 part of the
// update (for float32 fields the conversions, 16 lanes per clock) per half sweep, plus one
// trade every kHalo of them (about 1.5 us). One launch per kHalo half sweeps pays the load,
// store and launch of a whole tile at each trade instead. Measured, us a sweep (shared-memory
// tiles of 8 Jacobi sweeps or 4 split-layout SOR sweeps a launch, one-colour launches before):
//   Jacobi  128^2 float64 1.21 -> 0.54, 600 x 800 float32 3.9 -> 1.8
//   SOR     389 x 514 float32 with obstacles 7.2 -> 1.1, 512^2 float64 to 1e-6 3.7 -> 1.3
// 16 warps of few rows beat 8 warps of twice as many (512^2 float32 SOR 1.00 against 1.33).
constexpr int kHalo = 8;
constexpr int kResOwnCols = kResCols - 2 * kHalo;

template <typename T>
struct ResArgs {
  int H, W;
  T* p;          // natural layout, or colour plane 0
  T* p1;         // colour plane 1 (split layout)
  int64_t ldp;   // row stride of p, or of the planes
  const T* b;    // divergence (rhs), laid out likewise
  const T* b1;
  int64_t ldb;
  Masks m;
  double alpha, rb, omega;
  int sweeps;
  int from_zero;   // start from p = 0 without reading p
  uint64_t* xchg;  // two parities of H x Wx cells, one or two tagged words each; null: one tile
  int64_t ldx;     // cells per row of xchg (even)
  uint32_t tag;    // tag of the launch's first trade; the words hold smaller tags or 0 before it
  // sweeps to a tolerance: the checks' sums, two parities of a block's two words, and the outcome
  double beta;
  SweepsUntil u;
  uint64_t* sums;
  SweepsReached* reached;
};

// A trade moves tagged words: 32 bits of a value beside the 32-bit number of the trade, so the
// data say themselves when they are there and no flag, fence or second round trip is needed
// (64-bit accesses are single). A reader of trade n has every neighbour's trade n - 1 behind
// it, and each neighbour sent that after reading trade n - 2, so two parities suffice.
constexpr int kTradeSpins = 1 << 21;  // polls of about a microsecond each

__device__ __forceinline__ void st_words(uint64_t* p, uint64_t a, uint64_t b) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ void ld_words(const uint64_t* p, uint64_t& a, uint64_t& b) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ uint64_t tagged(uint32_t v, uint32_t tag) { return ((uint64_t)tag << 32) | v; }

// the two cells (columns i, i + 1; i even) of one row, at cell offset o (even) of the buffer
__device__ __forceinline__ void trade_put(uint64_t* x, int64_t o, const float (&v)[2], uint32_t tag) {
  st_words(x + o, tagged(__float_as_uint(v[0]), tag), tagged(__float_as_uint(v[1]), tag));
}
__device__ __forceinline__ void trade_put(uint64_t* x, int64_t o, const double (&v)[2], uint32_t tag) {
#pragma unroll
  for (int q = 0; q < 2; ++q)
    st_words(x + 2 * (o + q), tagged((uint32_t)__double2loint(v[q]), tag),
             tagged((uint32_t)__double2hiint(v[q]), tag));
}
__device__ __forceinline__ bool trade_get(const uint64_t* x, int64_t o, float (&v)[2], uint32_t tag) {
  uint64_t a, b;
  ld_words(x + o, a, b);
  v[0] = __uint_as_float((uint32_t)a);
  v[1] = __uint_as_float((uint32_t)b);
  return (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag;
}
__device__ __forceinline__ bool trade_get(const uint64_t* x, int64_t o, double (&v)[2], uint32_t tag) {
  bool ok = true;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint64_t a, b;
    ld_words(x + 2 * (o + q), a, b);
    v[q] = __hiloint2double((int)(uint32_t)b, (int)(uint32_t)a);
    ok = ok && (uint32_t)(a >> 32) == tag && (uint32_t)(b >> 32) == tag;
  }
  return ok;
}

// UNTIL: to a tolerance (SweepsUntil) instead of a.sweeps. A check comes right after a trade, when
// the cells beside the block's own are current: each block sums its own residuals, publishes the
// sum as a trade does its cells, and adds up all blocks' sums in the same order, so all take the
// same decision. 512^2 float64, 100 sweeps a check: 168 us a check with a launch for the sweeps,
// two for the sum and a host read, 135 in one launch.
template <typename T, bool SOR, bool SPLIT, int RPT, bool UNTIL>
__global__ void __launch_bounds__(kResThreads, 1) k_sweeps_resident(const __grid_constant__ ResArgs<T> a) {
  constexpr int RR = kResWarps * RPT;
  __shared__ ResEdges<T> sh;
  __shared__ int s_lost;
  __shared__ double s_sq;
  const int H = a.H, W = a.W;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int r0 = blockIdx.y * (RR - 2 * kHalo), c0 = blockIdx.x * kResOwnCols;
  const int j = r0 + w * RPT, i = c0 + 2 * lane;
  // the block's own cells
  const bool first_y = blockIdx.y == 0, last_y = blockIdx.y == gridDim.y - 1;
  const bool first_x = blockIdx.x == 0, last_x = blockIdx.x == gridDim.x - 1;
  const int oy0 = first_y ? 0 : r0 + kHalo, oy1 = last_y ? H : r0 + RR - kHalo;
  const int ox0 = first_x ? 0 : c0 + kHalo, ox1 = last_x ? W : c0 + kResCols - kHalo;
  const bool own_col = i >= ox0 && i < ox1;  // both of the lane's columns: the bounds are even or W
  if (threadIdx.x == 0) s_lost = 0;
  T e[RPT][2];
  double ab[RPT][2];
  uint32_t code[(RPT + 1) / 2];
#pragma unroll
  for (int r = 0; r < (RPT + 1) / 2; ++r) code[r] = 0;
  bool plain = true;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int jj = j + r, ii = i + q;
      e[r][q] = (T)0;
      ab[r][q] = 0.0;
      uint32_t k = 0;
      if (jj < H && ii < W) {
        const int col = (jj + ii) & 1;
        const int64_t o = SPLIT ? (int64_t)jj * a.ldp + (ii >> 1) : (int64_t)jj * a.ldp + ii;
        const int64_t ob = SPLIT ? (int64_t)jj * a.ldb + (ii >> 1) : (int64_t)jj * a.ldb + ii;
        if (!a.from_zero) e[r][q] = (SPLIT && col ? a.p1 : a.p)[o];
        ab[r][q] = a.alpha * (double)(SPLIT && col ? a.b1 : a.b)[ob];
        k = cell_code(a.m, H, W, jj, ii);
      }
      plain = plain && res_is_plain(k, ii, W);
      code[r >> 1] |= k << (10 * (r & 1) + 5 * q);
    }
  }
  plain = __all_sync(0xffffffffu, plain && i + 1 < W);
  const bool edge0 = i == 0, edge1 = i + 1 == W - 1;
  const double rb = a.rb, omega = a.omega, keep = 1.0 - a.omega;
  const int64_t parity = (int64_t)H * a.ldx * (sizeof(T) / 4);  // words of one parity

  const int bid = blockIdx.y * gridDim.x + blockIdx.x;
  const bool many = gridDim.x * gridDim.y > 1;
  int left = SOR ? 2 * a.sweeps : a.sweeps;
  int done = 0, stalls = a.u.stalls, par = 0;
  double best = a.u.best;
  if (UNTIL) left = 2 * min(a.u.check_every, a.u.max_sweeps);
  int buf = 0;
  uint32_t tag = a.tag;
  bool traded = !many, lost = false;
  while (true) {
    const int n = left < kHalo ? left : kHalo;  // even for SOR
    res_sweeps<T, SOR, RPT>(sh, buf, w, lane, e, ab, code, plain, edge0, edge1, rb, omega, keep, n);
    left -= n;
    // one trade at least: no block may write p before its neighbours have read it
    if (!UNTIL && left <= 0 && traded) break;
    if (many) {
      if (!traded) __syncthreads();  // the whole block has read its region of p
      uint64_t* x = a.xchg + (tag & 1) * parity;
      if (*(volatile int*)&s_lost != 0) {  // a wait that ran out, in a trade before this one's sweeps and barriers
#pragma unroll
        for (int r = 0; r < RPT; ++r) e[r][0] = e[r][1] = (T)__int_as_float(0x7fc00000);
      }
#pragma unroll
      for (int r = 0; r < RPT; ++r) {
        const int jj = j + r;
        if (!own_col || jj < oy0 || jj >= oy1) continue;
        const bool frame = (!first_y && jj < oy0 + kHalo) || (!last_y && jj >= oy1 - kHalo) ||
                           (!first_x && i < ox0 + kHalo) || (!last_x && i >= ox1 - kHalo);
        if (frame && SG_IN_BOUNDS(jj < H && i + 1 < a.ldx)) trade_put(x, (int64_t)jj * a.ldx + i, e[r], tag);
      }
      // the halo: cells of the region inside the grid that other blocks own
      const bool halo_col = !own_col && i < W;
      bool wait = false;
#pragma unroll
      for (int r = 0; r < RPT; ++r) wait |= j + r < H && i < W && (halo_col || j + r < oy0 || j + r >= oy1);
      if (wait && !lost) {
        int spins = 0;
        bool all;
        do {
          all = true;
#pragma unroll
          for (int r = 0; r < RPT; ++r) {
            const int jj = j + r;
            if (jj < H && (halo_col || jj < oy0 || jj >= oy1) && SG_IN_BOUNDS(i + 1 < a.ldx)) {
              if (!trade_get(x, (int64_t)jj * a.ldx + i, e[r], tag)) all = false;
            }
          }
        } while (!all && ++spins < kTradeSpins);
        if (!all || lose_waits(bid)) {
          s_lost = 1;
          lost = true;
        }
      }
      // the lanes leave the polls at different times; the next barrier counts whole warps
      __syncwarp();
      traded = true;
      ++tag;
    }
    if (left > 0) continue;
    if (!UNTIL) break;
    const int nblk = gridDim.x * gridDim.y, tid = threadIdx.x;
    res_edges<T, RPT>(sh, buf, w, lane, e);
    __syncthreads();
    double sq = res_sumsq<T, RPT>(sh, buf, w, lane, e, ab, code, a.beta, own_col ? oy0 - j : RPT,
                                  own_col ? oy1 - j : 0);
    buf ^= 1;
    sq = block_sum(sq);
    if (s_lost) sq = (double)__int_as_float(0x7fc00000);  // and so every block's sum of them all
    if (many) {
      uint64_t* sums = a.sums + (int64_t)par * nblk * 2;
      par ^= 1;
      if (tid == 0)
        st_words(sums + 2 * bid, tagged((uint32_t)__double2loint(sq), tag), tagged((uint32_t)__double2hiint(sq), tag));
      sq = 0.0;
      if (tid < nblk && SG_IN_BOUNDS(nblk <= kResThreads)) {
        uint64_t lo, hi;
        int spins = 0;
        do {
          ld_words(sums + 2 * tid, lo, hi);
        } while (((uint32_t)(lo >> 32) != tag || (uint32_t)(hi >> 32) != tag) && *(volatile int*)&s_lost == 0 &&
                 ++spins < kTradeSpins);
        if ((uint32_t)(lo >> 32) != tag || (uint32_t)(hi >> 32) != tag) s_lost = 1;
        sq = __hiloint2double((int)(uint32_t)hi, (int)(uint32_t)lo);
      }
      __syncwarp();
      sq = block_sum(sq);
    }
    if (tid == 0) s_sq = s_lost ? (double)__int_as_float(0x7fc00000) : sq;
    __syncthreads();
    sq = s_sq;
    done += min(a.u.check_every, a.u.max_sweeps - done);
    const double rel = a.u.r0 > 0.0 ? sqrt(sq) / a.u.r0 : 0.0;
    bool stop = !(rel > a.u.tol) || !isfinite(rel) || done >= a.u.max_sweeps;
    if (rel < 0.99 * best) {
      best = rel;
      stalls = 0;
    } else {
      ++stalls;
      stop = stop || (a.u.stall_limit > 0 && stalls >= a.u.stall_limit);
    }
    if (stop) {
      if (bid == 0 && tid == 0) *a.reached = SweepsReached{sq, best, done, stalls};
      break;
    }
    left = 2 * min(a.u.check_every, a.u.max_sweeps - done);
  }
  __syncthreads();
  // a wait that ran out (waits.cuh) leaves no usable iterate: say so in p
  const bool bad = s_lost != 0;
  count_lost_wait(s_lost);
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int jj = j + r;
    if (!own_col || jj < oy0 || jj >= oy1) continue;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int ii = i + q;
      if (ii >= W || !SG_IN_BOUNDS(jj < H)) continue;
      const int64_t o = SPLIT ? (int64_t)jj * a.ldp + (ii >> 1) : (int64_t)jj * a.ldp + ii;
      (SPLIT && ((jj + ii) & 1) ? a.p1 : a.p)[o] = bad ? (T)__int_as_float(0x7fc00000) : e[r][q];
    }
  }
}

// ------------------------------------------------------------------ host side
int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return 0;
  return n;
}

// Rows per thread: the fewest whose tiles all fit on the chip at once, one block an SM (the
// blocks wait for one another). 0: the grid does not fit. One row and one column have no
// tile form worth the launch (and a single cell no fluid).
int resident_rows(int64_t H, int64_t W) {
  if (H < 2 || W < 2 || H > (1 << 15) || W > (1 << 15)) return 0;
  const int sms = sm_count();
  for (int rpt = 2; rpt <= 8; rpt *= 2)
    if ((int64_t)res_tiles((int)H, kResWarps * rpt, kHalo) * res_tiles((int)W, kResCols, kHalo) <= sms) return rpt;
  return 0;
}

// Up to four rows a thread: with eight the check's registers spill in the float64 sweeps. us a
// check, from the host against inside the launch: every 100 sweeps (the solver's default) float64
// 283 against 442 at 600 x 801 and 284 against 420 at 800 x 900, float32 307 / 304 and 297 / 300;
// every 10 sweeps the launch wins in both types (66 / 56 and 69 / 45 at 600 x 801).
bool resident_until_fits(int64_t H, int64_t W) {
  const int rpt = resident_rows(H, W);
  return rpt == 2 || rpt == 4;
}

static int64_t resident_trade_bytes(int64_t elem, int64_t H, int64_t W) {
  return 2 * H * ((W + 1) & ~(int64_t)1) * 2 * elem;
}
int64_t resident_workspace_bytes(int64_t elem, int64_t H, int64_t W) {
  const int rpt = resident_rows(H, W);
  if (rpt == 0) return 0;
  return resident_trade_bytes(elem, H, W) + (int64_t)sm_count() * 4 * 8 + (int64_t)sizeof(SweepsReached);
}

template <typename T, bool SOR, bool SPLIT, int RPT, bool UNTIL>
static int launch_resident_rpt(ResArgs<T>& a, cudaStream_t s) {
  dim3 grid((unsigned)res_tiles(a.W, kResCols, kHalo), (unsigned)res_tiles(a.H, kResWarps * RPT, kHalo));
  void* args[] = {&a};
  cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_sweeps_resident<T, SOR, SPLIT, RPT, UNTIL>, grid,
                                              dim3(kResThreads), args, 0, s);
  note_launch();
  return e == cudaSuccess ? SG_OK : fail(SG_ERR_CUDA, "resident sweeps: %s", cudaGetErrorString(e));
}

int resident_trades(int sor, int sweeps) {
  const int n = sor ? 2 * sweeps : sweeps;
  return std::max(1, (n + kHalo - 1) / kHalo);
}

template <typename T>
int resident_sweeps(int sor, int split, int H, int W, T* p, T* p1, int64_t ldp, const T* b, const T* b1, int64_t ldb,
                    const Masks& m, double alpha, double rb, double omega, int64_t sweeps, bool from_zero, void* xchg,
                    uint32_t* tag, cudaStream_t s) {
  const int rpt = resident_rows(H, W);
  if (rpt == 0) return fail(SG_ERR_CAPACITY, "%d x %d cells do not fit the resident sweeps", H, W);
  ResArgs<T> a{H, W, p, p1, ldp, b, b1, ldb, m, alpha, rb, omega, 0, from_zero, (uint64_t*)xchg, (W + 1) & ~1, 0,
               0.0, SweepsUntil{}, nullptr, nullptr};
  auto go = [&](auto SOR_, auto SPLIT_) {
    constexpr bool S = decltype(SOR_)::value, P = decltype(SPLIT_)::value;
    if (rpt == 2) return launch_resident_rpt<T, S, P, 2, false>(a, s);
    if (rpt == 4) return launch_resident_rpt<T, S, P, 4, false>(a, s);
    return launch_resident_rpt<T, S, P, 8, false>(a, s);
  };
  for (; sweeps > 0; sweeps -= a.sweeps) {
    a.sweeps = (int)std::min<int64_t>(sweeps, kResidentSweeps);
    a.tag = *tag;
    *tag += (uint32_t)resident_trades(sor, a.sweeps);
    SG_CHECK(!sor ? go(std::false_type{}, std::false_type{})
                  : split ? go(std::true_type{}, std::true_type{}) : go(std::true_type{}, std::false_type{}));
    a.from_zero = 0;
  }
  return SG_OK;
}
template int resident_sweeps<float>(int, int, int, int, float*, float*, int64_t, const float*, const float*, int64_t,
                                    const Masks&, double, double, double, int64_t, bool, void*, uint32_t*,
                                    cudaStream_t);
template int resident_sweeps<double>(int, int, int, int, double*, double*, int64_t, const double*, const double*,
                                     int64_t, const Masks&, double, double, double, int64_t, bool, void*, uint32_t*,
                                     cudaStream_t);

template <typename T>
int resident_sweeps_until(int H, int W, T* p0, T* p1, int64_t ldp, const T* b0, const T* b1, int64_t ldb,
                          const Masks& m, double alpha, double rb, double beta, double omega, const SweepsUntil& u,
                          void* xchg, uint32_t tag, SweepsReached* reached, cudaStream_t s) {
  const int rpt = resident_rows(H, W);
  if (!resident_until_fits(H, W) || u.max_sweeps <= 0 || u.check_every <= 0)
    return fail(SG_ERR_CAPACITY, "%d x %d cells do not fit the resident sweeps", H, W);
  uint64_t* sums = (uint64_t*)((char*)xchg + resident_trade_bytes(sizeof(T), H, W));
  ResArgs<T> a{H, W, p0, p1, ldp, b0, b1, ldb, m, alpha, rb, omega, 0, 0, (uint64_t*)xchg, (W + 1) & ~1, tag,
               beta, u, sums, (SweepsReached*)(sums + (int64_t)sm_count() * 4)};
  SG_CHECK(rpt == 2 ? (launch_resident_rpt<T, true, true, 2, true>(a, s))
                    : (launch_resident_rpt<T, true, true, 4, true>(a, s)));
  cudaError_t e = cudaMemcpyAsync(reached, a.reached, sizeof(*reached), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  return e == cudaSuccess ? SG_OK : fail(SG_ERR_CUDA, "resident sweeps: %s", cudaGetErrorString(e));
}
template int resident_sweeps_until<float>(int, int, float*, float*, int64_t, const float*, const float*, int64_t,
                                          const Masks&, double, double, double, double, const SweepsUntil&, void*,
                                          uint32_t, SweepsReached*, cudaStream_t);
template int resident_sweeps_until<double>(int, int, double*, double*, int64_t, const double*, const double*, int64_t,
                                           const Masks&, double, double, double, double, const SweepsUntil&, void*,
                                           uint32_t, SweepsReached*, cudaStream_t);

}  // namespace sg

using namespace sg;

extern "C" {

int64_t sg_sweeps_workspace_bytes(int dtype, int64_t H, int64_t W) {
  if ((dtype != SG_F32 && dtype != SG_F64) || H < 1 || W < 1) return -1;
  return resident_workspace_bytes(dtype == SG_F32 ? 4 : 8, H, W);
}

int sg_sweeps_solve(int dtype, int sor, int64_t H, int64_t W, void* p, int64_t ld_p, const void* div, int64_t ld_div,
                    int mask_mode, const uint8_t* fmu, int64_t ld_fmu, const uint8_t* fmv, int64_t ld_fmv,
                    double alpha, double reciprocal_beta, double omega, int iterations, int from_zero,
                    void* workspace, int64_t workspace_bytes, void* stream) {
  SG_REQUIRE(H >= 1 && W >= 1 && H <= (1 << 28) && W <= (1 << 28), "bad grid %lld x %lld", (long long)H, (long long)W);
  SG_REQUIRE(p && div && ld_p >= W && ld_div >= W, "bad fields");
  SG_REQUIRE(iterations >= (from_zero ? 1 : 0), "iterations must be >= 0, and >= 1 from zero");
  SG_REQUIRE(mask_mode == SG_MASK_OPEN || mask_mode == SG_MASK_RING || (mask_mode == SG_MASK_PLANES && fmu && fmv),
             "bad mask mode %d or missing mask planes", mask_mode);
  const int64_t need = sg_sweeps_workspace_bytes(dtype, H, W);
  if (need < 0) return fail(SG_ERR_DTYPE, "unsupported dtype code %d", dtype);
  if (need == 0)
    return fail(SG_ERR_CAPACITY, "%lld x %lld cells do not fit the resident sweeps", (long long)H, (long long)W);
  SG_REQUIRE(workspace && !((uintptr_t)workspace & 15) && workspace_bytes >= need,
             "workspace must be 16-byte aligned and hold %lld bytes", (long long)need);
  if (iterations == 0) return SG_OK;
  Masks m = make_masks(mask_mode, H, W, fmu, ld_fmu, fmv, ld_fmv, nullptr, 0);
  cudaStream_t s = as_stream(stream);
  cudaError_t e = cudaMemsetAsync(workspace, 0, (size_t)need, s);
  if (e != cudaSuccess) return fail(SG_ERR_CUDA, "sg_sweeps_solve: %s", cudaGetErrorString(e));
  uint32_t tag = 1;
  SG_DISPATCH(dtype, {
    return resident_sweeps<T>(sor != 0, 0, (int)H, (int)W, (T*)p, nullptr, ld_p, (const T*)div, nullptr, ld_div, m,
                              alpha, reciprocal_beta, omega, iterations, from_zero != 0, workspace, &tag, s);
  });
}

}  // extern "C"

SG_BOUNDS_ACCESSOR(sweeps)
SG_WAITS_ACCESSOR(sweeps)
