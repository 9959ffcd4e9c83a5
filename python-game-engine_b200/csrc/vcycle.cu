// The reference's V-cycles (multigrid/solver.py:94-176) in two launches per level and cycle.
//
//   k_mg_codes level 0's cell codes from the caller's planes, once a call
//   k_mg_down  smoothing sweeps, the residual, its mean over fluid children divided by
//              alpha(2h) as the next level's rhs
//   k_mg_up    bilinear prolongation added to the pressure, smoothing sweeps
//   k_mg_tail  every level of at most 64 x 64 cells, both ways, and the coarsest sweeps, in
//              one block
//
// Each value is formed by the expressions of the separate kernels (k_jacobi / k_rbsor_half,
// k_residual, k_restrict_avg, k_prolong of operators.cu) in the same order, so the results are
// theirs bit for bit; compiled with -fmad=false like them.
//
// What bounds them: the levels sit in L2 and a launch is a few microseconds of latency (load,
// one barrier chain per half sweep, store), so the number of dependent launches is the time:
// 512^2, 7 levels, V(2,2) with red-black smoothing took 260 launches of 2.7 us per pair of
// cycles as separate kernels (742 us of kernels, 1.5 ms with their issue from the host) and
// takes 15 launches and 135 us now; 2048^2 float32, 9 levels, 370 us. Cell codes made once per
// hierarchy (level 0's once a call, 4 us at 512^2) instead of four mask bytes a cell and launch: 512^2 down / up 7.0 / 8.3 -> 5.0 / 5.3 us
// (4.3 / 4.7 on average over the levels above 64^2, tail 25),
// 1024^2 19.2 / 20.1 -> 12.1 / 12.1.
#include <algorithm>
#include <type_traits>

#include "sweep_region.cuh"

namespace sg {

constexpr int kMgMaxLevels = 16;
// Rows per thread of the level launches: 2 (32 x 64 regions). 4 rows do less halo work in half
// the blocks and lost at every size, us down / up of a level: 512^2 float32 7.0 / 8.3 against
// 9.5 / 11.2, 1024^2 float64 23.6 / 22.3 against 27.5 / 30.5, 2048^2 float64 100 / 91 against
// 129 / 128.
constexpr int kMgRows = 2;
constexpr int kMgTailRows = 64, kMgTailCols = 64;  // 16 warps x 4 rows, 32 lanes x 2 columns

template <typename T>
struct MgLevelArgs {
  int H, W;
  const T* pin;   // null: the sweeps start from zero
  int64_t ldin;
  T* pout;
  int64_t ldout;
  const T* b;
  int64_t ldb;
  const uint8_t* code;  // cell codes (k_mg_codes)
  double alpha, omega, rb, beta;
  int n;          // half sweeps (SOR) or sweeps (Jacobi) a side
  int halo;       // even, at least n, or n + 1 where the residual is formed too
  T* bc;          // down: the next level's rhs, row stride W / 2; up: its correction
  const T* ec;
  T divisor;      // down: alpha(2h)
};

// A level's code bytes, row stride W rounded up to even: the K_ bits of the faces, and K_CELL,
// that the cell is fluid in the hierarchy. The sweeps go by the faces, the residual and the
// transfers by the hierarchy's cells, as the separate kernels do with is_fluid; the two differ on
// the fine level where the caller has edited its planes since the hierarchy was built.
enum : uint32_t { K_CELL = 32 };

// Codes of the cell pair (j, i), (j, i + 1), i even: ten bits (0 off the grid). cells: their
// K_CELL bits, from bit 2 r on.
__device__ __forceinline__ uint32_t mg_codes(const uint8_t* code, int H, int W, int j, int i, int r,
                                             uint32_t& cells) {
  if (j >= H || i >= W) return 0;
  const uchar2 c = *reinterpret_cast<const uchar2*>(code + (int64_t)j * ((W + 1) & ~1) + i);
  cells |= (((uint32_t)c.x >> 5) | (((uint32_t)c.y >> 5) << 1)) << (2 * r);
  return (c.x & K_ALL) | ((c.y & K_ALL) << 5);
}

// Loads the region's cells: values (pin, or 0), alpha * rhs and codes; the block's own range.
template <typename T, int RPT>
struct MgRegion {
  int j, i, lane, w, oy0, oy1;
  bool own_col, plain, edge0, edge1;
  T e[RPT][2];
  double ab[RPT][2];
  uint32_t code[(RPT + 1) / 2], cells;

  __device__ __forceinline__ void load(const MgLevelArgs<T>& a) {
    constexpr int RR = kResWarps * RPT;
    lane = threadIdx.x & 31;
    w = threadIdx.x >> 5;
    const int r0 = blockIdx.y * (RR - 2 * a.halo), c0 = blockIdx.x * (kResCols - 2 * a.halo);
    j = r0 + w * RPT;
    i = c0 + 2 * lane;
    oy0 = blockIdx.y == 0 ? 0 : r0 + a.halo;
    oy1 = blockIdx.y == gridDim.y - 1 ? a.H : r0 + RR - a.halo;
    own_col = i >= (blockIdx.x == 0 ? 0 : c0 + a.halo) &&
              i < (blockIdx.x == gridDim.x - 1 ? a.W : c0 + kResCols - a.halo);
#pragma unroll
    for (int r = 0; r < (RPT + 1) / 2; ++r) code[r] = 0;
    cells = 0;
    bool all = i + 1 < a.W;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int jj = j + r;
      const uint32_t kk = mg_codes(a.code, a.H, a.W, jj, i, r, cells);
      all = all && res_is_plain(kk & K_ALL, i, a.W) && res_is_plain(kk >> 5, i + 1, a.W);
      code[r >> 1] |= kk << (10 * (r & 1));
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        e[r][q] = (T)0;
        ab[r][q] = 0.0;
        if (jj < a.H && i + q < a.W && SG_IN_BOUNDS(jj >= 0 && i >= 0)) {
          if (a.pin) e[r][q] = a.pin[(int64_t)jj * a.ldin + i + q];
          ab[r][q] = a.alpha * (double)a.b[(int64_t)jj * a.ldb + i + q];
        }
      }
    }
    plain = __all_sync(0xffffffffu, all);
    edge0 = i == 0;
    edge1 = i + 1 == a.W - 1;
  }
  __device__ __forceinline__ void store(const MgLevelArgs<T>& a) const {
    if (!own_col) return;
#pragma unroll
    for (int r = 0; r < RPT; ++r) {
      const int jj = j + r;
      if (jj < oy0 || jj >= oy1 || !SG_IN_BOUNDS(jj < a.H)) continue;
      a.pout[(int64_t)jj * a.ldout + i] = e[r][0];
      if (i + 1 < a.W) a.pout[(int64_t)jj * a.ldout + i + 1] = e[r][1];
    }
  }
};

// multigrid/transfer.py:5-36 for the 2 x 2 cells at rows r, r + 1 of the thread
template <typename T, int RPT>
__device__ __forceinline__ T mg_restrict(const T (&res)[RPT][2], uint32_t cells, int r, T divisor) {
  double total = 0.0;  // res is 0 off the fluid
#pragma unroll
  for (int d = 0; d < 2; ++d)
#pragma unroll
    for (int q = 0; q < 2; ++q) total += (double)res[r + d][q];
  const int count = __popc((cells >> (2 * r)) & 15);
  // a division by 4, 2 or 1 is the multiplication by its exact reciprocal
  const double by = count == 4 ? 0.25 : (count == 2 ? 0.5 : 1.0);
  const double mean = count == 3 ? total / 3.0 : total * by;
  return (T)mean / divisor;
}

// multigrid/transfer.py:38-72: the correction of fluid cell (j, i), sample_ref at
// (i / 2 - 1/4, j / 2 - 1/4): cells (i - 1) >> 1 and (i + 1) >> 1 with weight 3/4 or 1/4 on the
// latter, exact in both forms; at an edge both are the same cell and the weight is void.
template <typename T>
__device__ __forceinline__ T mg_prolong(const T* c, int64_t ldc, int Hc, int Wc, int j, int i) {
  const int x1 = min((i + 1) >> 1, Wc - 1), x0 = min(max((i - 1) >> 1, 0), x1);  // i, j may lie off the grid
  const int y1 = min((j + 1) >> 1, Hc - 1), y0 = min(max((j - 1) >> 1, 0), y1);
  const double tx = (i & 1) ? 0.25 : 0.75, ty = (j & 1) ? 0.25 : 0.75;
  if (!SG_IN_BOUNDS(x0 >= 0 && x1 < Wc && y0 >= 0 && y1 < Hc)) return (T)0;
  const T* r0 = c + (int64_t)y0 * ldc;
  const T* r1 = c + (int64_t)y1 * ldc;
  const double c0 = lerp_ref(r0[x0], r0[x1], tx);
  const double c1 = lerp_ref(r1[x0], r1[x1], tx);
  return (T)(c0 + (c1 - c0) * ty);
}

// Codes of a level from its face masks; K_CELL from the codes `built` at the hierarchy's making
// (null: from the masks).
__global__ void k_mg_codes(int H, int W, Masks m, const uint8_t* __restrict__ built, uint8_t* __restrict__ code,
                           int ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= ld || j >= H) return;
  const int64_t o = (int64_t)j * ld + i;
  const uint32_t c = i < W ? cell_code(m, H, W, j, i) : 0;
  const uint32_t cell = built ? built[o] & K_CELL : (c & K_FLUID) << 1;
  code[o] = (uint8_t)(c | cell);
}
static_assert(K_CELL == K_FLUID << 1, "the next bit");

template <typename T, bool SOR>
__global__ void __launch_bounds__(kResThreads) k_mg_down(const __grid_constant__ MgLevelArgs<T> a) {
  constexpr int RPT = kMgRows;
  __shared__ ResEdges<T> sh;
  MgRegion<T, RPT> g;
  g.load(a);
  int buf = 0;
  res_sweeps<T, SOR, RPT>(sh, buf, g.w, g.lane, g.e, g.ab, g.code, g.plain, g.edge0, g.edge1, a.rb, a.omega,
                          1.0 - a.omega, a.n);
  g.store(a);
  T res[RPT][2];
  res_residual<T, RPT>(sh, buf, g.w, g.lane, g.e, g.ab, g.code, g.cells, a.beta, res);
  if (!g.own_col) return;
#pragma unroll
  for (int r = 0; r < RPT; r += 2) {
    const int jj = g.j + r;
    if (jj < g.oy0 || jj >= g.oy1 || !SG_IN_BOUNDS(jj + 1 < a.H && g.i + 1 < a.W)) continue;
    a.bc[(int64_t)(jj >> 1) * (a.W >> 1) + (g.i >> 1)] = mg_restrict<T, RPT>(res, g.cells, r, a.divisor);
  }
}

template <typename T, bool SOR>
__global__ void __launch_bounds__(kResThreads) k_mg_up(const __grid_constant__ MgLevelArgs<T> a) {
  constexpr int RPT = kMgRows;
  __shared__ ResEdges<T> sh;
  MgRegion<T, RPT> g;
  g.load(a);
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (g.cells >> (2 * r + q) & 1)
        g.e[r][q] = g.e[r][q] + mg_prolong(a.ec, a.W >> 1, a.H >> 1, a.W >> 1, g.j + r, g.i + q);
  int buf = 0;
  res_sweeps<T, SOR, RPT>(sh, buf, g.w, g.lane, g.e, g.ab, g.code, g.plain, g.edge0, g.edge1, a.rb, a.omega,
                          1.0 - a.omega, a.n);
  g.store(a);
}

template <typename T>
struct MgTailArgs {
  int levels;
  int H[kMgMaxLevels], W[kMgMaxLevels], off[kMgMaxLevels];  // off: the level's first cell in the shared arrays
  const uint8_t* code[kMgMaxLevels];
  int off_code[kMgMaxLevels];  // bytes, even
  double alpha[kMgMaxLevels], omega[kMgMaxLevels];
  int cells;        // of all levels
  const T* pin;     // the first level's pressure, null: 0
  int64_t ldin;
  T* pout;
  int64_t ldout;
  const T* b;
  int64_t ldb;
  double rb, beta;
  int n, n_coarsest;
};

template <typename T>
struct MgTailShared {
  T* p;            // pressures of all levels
  T* b;            // right-hand sides of the levels below the first
  uint8_t* code;   // codes of all levels
};

// One visit of level l: up, down or (the last level) its coarsest sweeps, in RPT rows a thread.
template <typename T, bool SOR, int RPT>
__device__ __forceinline__ void mg_tail_visit(const MgTailArgs<T>& a, const MgTailShared<T>& t, ResEdges<T>& sh, int l,
                                              bool up, bool coarsest) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int j = w * RPT, i = 2 * lane;
  const int H = a.H[l], W = a.W[l], o = a.off[l];
  const int threads = 32 * ((H + RPT - 1) / RPT);
  if (j >= H) return;
  const double alpha = a.alpha[l], omega = a.omega[l];
  int buf = 0;
  T e[RPT][2];
  double ab[RPT][2];
  uint32_t code[(RPT + 1) / 2], cells = 0;
#pragma unroll
  for (int r = 0; r < (RPT + 1) / 2; ++r) code[r] = 0;
  bool all = i + 1 < W;
#pragma unroll
  for (int r = 0; r < RPT; ++r) {
    const int jj = j + r;
    const uint32_t kk = mg_codes(t.code + a.off_code[l], H, W, jj, i, r, cells);
    all = all && res_is_plain(kk & K_ALL, i, W) && res_is_plain(kk >> 5, i + 1, W);
    code[r >> 1] |= kk << (10 * (r & 1));
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int ii = i + q;
      e[r][q] = (T)0;
      ab[r][q] = 0.0;
      if (jj >= H || ii >= W || !SG_IN_BOUNDS(o + jj * W + ii < a.cells)) continue;
      const int c = o + jj * W + ii;
      if (up)
        e[r][q] = t.p[c];
      else if (l == 0 && a.pin)
        e[r][q] = a.pin[(int64_t)jj * a.ldin + ii];
      ab[r][q] = alpha * (double)(l == 0 ? a.b[(int64_t)jj * a.ldb + ii] : t.b[c]);
    }
  }
  if (up) {
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int q = 0; q < 2; ++q)
        e[r][q] = e[r][q] + pick(cells >> (2 * r + q) & 1,
                                 mg_prolong((const T*)t.p + a.off[l + 1], W >> 1, H >> 1, W >> 1, j + r, i + q), (T)0);
  }
  const bool plain = __all_sync(0xffffffffu, all);
  res_sweeps<T, SOR, RPT, true>(sh, buf, w, lane, e, ab, code, plain, i == 0, i + 1 == W - 1, a.rb, omega,
                                1.0 - omega, coarsest ? a.n_coarsest : a.n, threads);
  const bool last = l == 0 && (up || coarsest);
  // a thread stores the cells it alone has read
#pragma unroll
  for (int r = 0; r < RPT; ++r)
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int jj = j + r, ii = i + q;
      if (jj >= H || ii >= W || !SG_IN_BOUNDS(o + jj * W + ii < a.cells)) continue;
      if (last)
        a.pout[(int64_t)jj * a.ldout + ii] = e[r][q];
      else
        t.p[o + jj * W + ii] = e[r][q];
    }
  if (up || coarsest) return;
  T res[RPT][2];
  res_residual<T, RPT, true>(sh, buf, w, lane, e, ab, code, cells, a.beta, res, threads);
#pragma unroll
  for (int r = 0; r < RPT; r += 2)
    if (j + r + 1 < H && i + 1 < W &&
        SG_IN_BOUNDS(a.off[l + 1] + ((j + r) >> 1) * (W >> 1) + (i >> 1) < a.cells))
      t.b[a.off[l + 1] + ((j + r) >> 1) * (W >> 1) + (i >> 1)] = mg_restrict<T, RPT>(res, cells, r, (T)a.alpha[l + 1]);
}

// The warps whose rows lie beyond a level wait for the others at the visit's end, and levels
// of at most 32 rows take two rows a thread, so twice the warps: what a small level costs is
// the length of one warp's instruction stream. (64^2 down to 8^2 with 30 coarsest SOR sweeps,
// float32: 50 us with all 16 warps in every half sweep and the codes formed from the masks,
// 38 us with idle warps left out and codes from global memory, 25 us so.)
template <typename T, bool SOR>
__global__ void __launch_bounds__(kResThreads) k_mg_tail(const __grid_constant__ MgTailArgs<T> a) {
  extern __shared__ __align__(16) unsigned char mg_smem[];
  __shared__ ResEdges<T> sh;
  MgTailShared<T> t;
  t.p = reinterpret_cast<T*>(mg_smem);
  t.b = t.p + a.cells;
  t.code = reinterpret_cast<uint8_t*>(t.b + a.cells);
  for (int l = 0; l < a.levels; ++l) {
    const int n = a.H[l] * (((a.W[l] + 1) & ~1) >> 1);  // pairs of codes
    const uint16_t* src = reinterpret_cast<const uint16_t*>(a.code[l]);
    uint16_t* dst = reinterpret_cast<uint16_t*>(t.code + a.off_code[l]);
    for (int q = threadIdx.x; q < n; q += kResThreads) dst[q] = src[q];
  }
  __syncthreads();
  // down to the last level, its sweeps, and up again
  for (int s = 0; s < 2 * a.levels - 1; ++s) {
    const bool up = s >= a.levels, coarsest = s == a.levels - 1;
    const int l = up ? 2 * a.levels - 2 - s : s;
    if (a.H[l] <= 2 * kResWarps)
      mg_tail_visit<T, SOR, 2>(a, t, sh, l, up, coarsest);
    else
      mg_tail_visit<T, SOR, 4>(a, t, sh, l, up, coarsest);
    __syncthreads();
  }
}

// ------------------------------------------------------------------ host side
struct MgPlan {  // offsets (bytes) of the levels' arrays in the workspace
  int tail;      // first level of the tail, n when the coarsest runs as resident sweeps
  int64_t pa[kMgMaxLevels], pb[kMgMaxLevels], rhs[kMgMaxLevels];
  int64_t code, xchg, bytes;  // code: level 0's
};

static int64_t code_pitch(int64_t W) { return (W + 1) & ~(int64_t)1; }

// false: a level or sweep count these kernels do not take
static bool mg_plan(int64_t elem, int n, const sg_mg_level* lv, int sor, int sweeps, MgPlan* p) {
  const int half = sor ? 2 * sweeps : sweeps;
  if (n < 1 || n > kMgMaxLevels || half > 8) return false;  // the down halo, half + 1 rounded up to even, is at most 10
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    const int64_t o = off;
    off = (off + bytes + 255) & ~(int64_t)255;
    return o;
  };
  p->tail = n;
  for (int k = 0; k < n; ++k) {
    if (lv[k].H < 1 || lv[k].W < 1 || lv[k].H > (1 << 15) || lv[k].W > (1 << 15)) return false;
    if (k + 1 < n && (lv[k + 1].H * 2 != lv[k].H || lv[k + 1].W * 2 != lv[k].W)) return false;
    if (p->tail == n && lv[k].H <= kMgTailRows && lv[k].W <= kMgTailCols) p->tail = k;
    const int64_t bytes = lv[k].H * lv[k].W * elem;
    p->pa[k] = k > 0 ? take(bytes) : 0;   // level 0 works on the caller's pressure and rhs
    p->rhs[k] = k > 0 ? take(bytes) : 0;
    p->pb[k] = k + 1 < n ? take(bytes) : 0;
  }
  p->code = take(lv[0].H * code_pitch(lv[0].W));
  p->xchg = off;
  if (p->tail == n) {
    const int64_t x = resident_workspace_bytes(elem, lv[n - 1].H, lv[n - 1].W);
    if (x == 0) return false;
    take(x);
  }
  p->bytes = off;
  return true;
}

static Masks level_masks(const sg_mg_level& L) {
  return make_masks(SG_MASK_PLANES, L.H, L.W, (const uint8_t*)L.face_mask_u, L.W + 1, (const uint8_t*)L.face_mask_v,
                    L.W, nullptr, 0);
}

template <typename T, bool SOR>
static int mg_vcycles(int n, const sg_mg_level* lv, const MgPlan& P, T* p, int64_t ldp, const T* div, int64_t ldd,
                      double rb, int cycles, int sweeps, int coarsest, bool from_zero, char* ws, cudaStream_t s) {
  const int half = SOR ? 2 * sweeps : sweeps;
  const double beta = 1.0 / rb;
  auto at = [&](int64_t o) { return (T*)(ws + o); };
  // level 0's codes of this call: its planes are the caller's, who may edit them between calls
  uint8_t* const code0 = (uint8_t*)(ws + P.code);
  if (cycles > 0 && (n > 1 || P.tail < n)) {
    const int ld = (int)code_pitch(lv[0].W);
    SG_LAUNCH(k_mg_codes<<<grid2d(ld, lv[0].H), block2d(), 0, s>>>((int)lv[0].H, (int)lv[0].W, level_masks(lv[0]),
                                                                  (const uint8_t*)lv[0].code, code0, ld));
  }
  auto level = [&](int k, bool down, bool zero) {
    MgLevelArgs<T> a{};
    a.H = (int)lv[k].H;
    a.W = (int)lv[k].W;
    a.code = k == 0 ? code0 : (const uint8_t*)lv[k].code;
    a.alpha = lv[k].alpha;
    a.omega = lv[k].omega;
    a.rb = rb;
    a.beta = beta;
    a.n = half;
    a.halo = (half + (down ? 1 : 0) + 1) & ~1;
    T* pa = k == 0 ? p : at(P.pa[k]);
    const int64_t lda = k == 0 ? ldp : a.W;
    a.b = k == 0 ? div : at(P.rhs[k]);
    a.ldb = k == 0 ? ldd : a.W;
    if (down) {  // pa (level 0) or zero -> pb
      a.pin = k == 0 && !zero ? p : nullptr;
      a.ldin = ldp;
      a.pout = at(P.pb[k]);
      a.ldout = a.W;
      a.bc = at(P.rhs[k + 1]);
      a.divisor = (T)lv[k + 1].alpha;
    } else {     // pb and the next level's correction -> pa
      a.pin = at(P.pb[k]);
      a.ldin = a.W;
      a.pout = pa;
      a.ldout = lda;
      a.ec = at(P.pa[k + 1]);
    }
    const dim3 g((unsigned)res_tiles(a.W, kResCols, a.halo), (unsigned)res_tiles(a.H, kResWarps * kMgRows, a.halo));
    if (down)
      SG_LAUNCH((k_mg_down<T, SOR><<<g, kResThreads, 0, s>>>(a)));
    else
      SG_LAUNCH((k_mg_up<T, SOR><<<g, kResThreads, 0, s>>>(a)));
  };
  MgTailArgs<T> t{};
  size_t smem = 0;
  int codes = 0;
  if (P.tail < n) {
    t.levels = n - P.tail;
    for (int q = 0; q < t.levels; ++q) {
      const sg_mg_level& L = lv[P.tail + q];
      t.H[q] = (int)L.H;
      t.W[q] = (int)L.W;
      t.off[q] = t.cells;
      t.cells += (int)(L.H * L.W);
      t.code[q] = P.tail + q == 0 ? code0 : (const uint8_t*)L.code;
      t.off_code[q] = codes;
      codes += (int)(L.H * code_pitch(L.W));
      t.alpha[q] = L.alpha;
      t.omega[q] = L.omega;
    }
    t.ldin = ldp;
    t.pout = P.tail == 0 ? p : at(P.pa[P.tail]);
    t.ldout = P.tail == 0 ? ldp : t.W[0];
    t.b = P.tail == 0 ? div : at(P.rhs[P.tail]);
    t.ldb = P.tail == 0 ? ldd : t.W[0];
    t.rb = rb;
    t.beta = beta;
    t.n = half;
    t.n_coarsest = SOR ? 2 * coarsest : coarsest;
    smem = (size_t)t.cells * 2 * sizeof(T) + (size_t)codes;
    // set on every call: the limit belongs to the function in the current device's context
    cudaError_t e = cudaFuncSetAttribute(k_mg_tail<T, SOR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(SG_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  } else {
    cudaError_t e = cudaMemsetAsync(ws + P.xchg, 0, (size_t)(P.bytes - P.xchg), s);
    if (e != cudaSuccess) return fail(SG_ERR_CUDA, "memset: %s", cudaGetErrorString(e));
  }
  uint32_t tag = 1;
  for (int c = 0; c < cycles; ++c) {
    const bool zero = from_zero && c == 0;  // level 0 starts from p = 0 without reading it
    for (int k = 0; k < P.tail && k < n - 1; ++k) level(k, true, zero);
    if (P.tail < n) {
      t.pin = P.tail == 0 && !zero ? p : nullptr;
      SG_LAUNCH((k_mg_tail<T, SOR><<<1, kResThreads, smem, s>>>(t)));
    } else {
      const sg_mg_level& L = lv[n - 1];
      T* pc = n == 1 ? p : at(P.pa[n - 1]);
      const bool fresh = n > 1 || zero;
      if (coarsest == 0 && fresh) {
        cudaError_t e = cudaMemset2DAsync(pc, sizeof(T) * (size_t)(n == 1 ? ldp : L.W), 0, sizeof(T) * (size_t)L.W,
                                          (size_t)L.H, s);
        if (e != cudaSuccess) return fail(SG_ERR_CUDA, "memset: %s", cudaGetErrorString(e));
      }
      SG_CHECK(resident_sweeps<T>(SOR, 0, (int)L.H, (int)L.W, pc, nullptr, n == 1 ? ldp : L.W,
                                  n == 1 ? div : at(P.rhs[n - 1]), nullptr, n == 1 ? ldd : L.W, level_masks(L),
                                  L.alpha, rb, L.omega, coarsest, fresh, ws + P.xchg, &tag, s));
    }
    for (int k = std::min(P.tail, n - 1) - 1; k >= 0; --k) level(k, false, false);
  }
  return check_launch("sg_mg_vcycles");
}

}  // namespace sg

using namespace sg;

extern "C" {

int64_t sg_mg_codes_bytes(int64_t H, int64_t W) { return H < 1 || W < 1 ? -1 : H * code_pitch(W); }

int sg_mg_codes(int64_t H, int64_t W, const uint8_t* fmu, const uint8_t* fmv, uint8_t* code, void* stream) {
  SG_REQUIRE(H >= 1 && W >= 1 && H <= (1 << 15) && W <= (1 << 15) && fmu && fmv && code, "bad grid or planes");
  const Masks m = make_masks(SG_MASK_PLANES, H, W, fmu, W + 1, fmv, W, nullptr, 0);
  const int ld = (int)code_pitch(W);
  SG_LAUNCH(k_mg_codes<<<grid2d(ld, H), block2d(), 0, as_stream(stream)>>>((int)H, (int)W, m, nullptr, code, ld));
  return check_launch("sg_mg_codes");
}

int64_t sg_mg_vcycles_workspace_bytes(int dtype, int n_levels, const sg_mg_level* levels, int sor, int sweeps) {
  MgPlan P;
  if ((dtype != SG_F32 && dtype != SG_F64) || !levels || sweeps < 0) return -1;
  return mg_plan(dtype == SG_F32 ? 4 : 8, n_levels, levels, sor, sweeps, &P) ? std::max<int64_t>(P.bytes, 256) : 0;
}

int sg_mg_vcycles(int dtype, int n_levels, const sg_mg_level* levels, void* p, int64_t ld_p, const void* div,
                  int64_t ld_div, double reciprocal_beta, int sor, int cycles, int sweeps, int coarsest_sweeps,
                  int from_zero, void* workspace, int64_t workspace_bytes, void* stream) {
  SG_REQUIRE(levels && p && div && n_levels >= 1, "null level table or fields");
  SG_REQUIRE(cycles >= (from_zero ? 1 : 0) && sweeps >= 0 && coarsest_sweeps >= 0,
             "counts must be >= 0, and cycles >= 1 from zero");
  SG_REQUIRE(reciprocal_beta != 0.0, "reciprocal_beta must be non-zero");
  SG_REQUIRE(dtype == SG_F32 || dtype == SG_F64, "unsupported dtype code %d", dtype);
  MgPlan P;
  if (coarsest_sweeps > (1 << 29) || !mg_plan(dtype == SG_F32 ? 4 : 8, n_levels, levels, sor, sweeps, &P))
    return fail(SG_ERR_CAPACITY, "these levels or sweeps do not fit the fused V-cycle");
  SG_REQUIRE(ld_p >= levels[0].W && ld_div >= levels[0].W, "row stride below row length");
  for (int k = 0; k < n_levels; ++k)
    SG_REQUIRE(levels[k].face_mask_u && levels[k].face_mask_v && levels[k].code && !((uintptr_t)levels[k].code & 1) &&
                   levels[k].alpha != 0.0, "level %d: masks, codes or alpha", k);
  SG_REQUIRE(workspace && !((uintptr_t)workspace & 255) && workspace_bytes >= P.bytes,
             "workspace must be 256-byte aligned and hold %lld bytes", (long long)P.bytes);
  SG_DISPATCH(dtype, {
    if (sor)
      return (mg_vcycles<T, true>(n_levels, levels, P, (T*)p, ld_p, (const T*)div, ld_div, reciprocal_beta, cycles,
                                  sweeps, coarsest_sweeps, from_zero != 0, (char*)workspace, as_stream(stream)));
    return (mg_vcycles<T, false>(n_levels, levels, P, (T*)p, ld_p, (const T*)div, ld_div, reciprocal_beta, cycles,
                                 sweeps, coarsest_sweeps, from_zero != 0, (char*)workspace, as_stream(stream)));
  });
}

}  // extern "C"

SG_BOUNDS_ACCESSOR(vcycle)
