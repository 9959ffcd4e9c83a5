// Lexicographic Gauss-Seidel (gauss_seidel.py:8-26) with the sweeps of a call following one
// another down the grid. Every update evaluates the reference's expression in the reference's
// order, so the iterates are those of one sweep after the other bit for bit. Compiled with
// -fmad=false like the other operator units.
#include <algorithm>

#include "sweep_region.cuh"
#include "waits.cuh"

namespace sg {

// ------------------------------------------------------------------ lexicographic Gauss-Seidel
// Cell (j, i) of anti-diagonal d = j + i reads d - 1 (this sweep) and d + 1 (the sweep before),
// so sweep s may work on diagonal t - 2 s at step t: sweeps run down the grid behind one
// another, and n of them take H + W - 1 + 2 (n - 1) steps instead of n (H + W - 1).
//
// The sweeps in flight are split over a chain of blocks, K to a block, one thread a cell of the
// diagonal that its sweep is at, and the block's last Mp threads load the diagonals to come
// (warps of their own where the block has room for them). A block holds the 2 K + 2 diagonals
// it works on in a shared-memory ring (entry x of a diagonal is the cell with coordinate x
// along the shorter axis: neighbours are entries x, x -+ 1 of the rows beside it, unit stride,
// no conflicts) and takes one barrier a step. A thread stays on its x, so two of the four
// neighbours and the old value are in its registers from the step before and its codes are
// read ahead of the barrier. A block's last sweep's diagonals go to
// the next block through a ring of kGsRing diagonals in global memory, as words that carry 32
// bits of the value and the diagonal's number: they say themselves when they are there. The
// chain runs one way, so a block that waited once stays that far behind and finds its loads,
// issued kGsAhead steps ahead, filled. A consumer tells every kGsCredit diagonals how far it
// has read, which is all that a producer ever waits for.
//
// What bounds it: the chain of steps, each a barrier and one update's latency (0.25 us with one
// sweep a block, 0.30 with four, 0.57 with eight, when loaders and updates share warps), and
// 4.5 us for each block of the chain to get under way. Hence about kGsCells updates a step
// (40 sweeps, float32, blocks for 256 / 512 / 896 cells: 97 x 161 142 / 130 / 143 us, 180 x 180
// 207 / 182 / 186). 97 x 161: 0.64 ms with one block for all sweeps, 11.0 ms one sweep after
// the other; 512 x 512 7.1 -> 0.69 ms.
constexpr int kGsThreads = 1024;
constexpr int kGsAhead = 4;
constexpr int kGsMaxSmem = 220 * 1024;
constexpr int kGsRing = 128;   // diagonals between two blocks
constexpr int kGsCredit = 16;  // diagonals between two credits
constexpr int kGsLine = 16;    // words from one block's credit to the next
constexpr int kGsCells = 512;  // updates a step for a block of a chain
constexpr int kGsSpins = 1 << 21;  // polls of about a microsecond each

template <typename T>
struct GsWords {  // a cell on its way to the next block
  static constexpr int N = sizeof(T) / 4;
  uint64_t w[N];
};
__device__ __forceinline__ void gs_put(uint64_t* o, float v, uint32_t tag) {
  const uint64_t a = ((uint64_t)tag << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(o), "l"(a) : "memory");
}
__device__ __forceinline__ void gs_put(uint64_t* o, double v, uint32_t tag) {
  const uint64_t t = (uint64_t)tag << 32;
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(o), "l"(t | (uint32_t)__double2loint(v)),
               "l"(t | (uint32_t)__double2hiint(v))
               : "memory");
}
__device__ __forceinline__ void gs_get(const uint64_t* o, GsWords<float>& g) {
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(g.w[0]) : "l"(o) : "memory");
}
__device__ __forceinline__ void gs_get(const uint64_t* o, GsWords<double>& g) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(g.w[0]), "=l"(g.w[1]) : "l"(o) : "memory");
}
__device__ __forceinline__ bool gs_there(const GsWords<float>& g, uint32_t tag) { return (uint32_t)(g.w[0] >> 32) == tag; }
__device__ __forceinline__ bool gs_there(const GsWords<double>& g, uint32_t tag) {
  return (uint32_t)(g.w[0] >> 32) == tag && (uint32_t)(g.w[1] >> 32) == tag;
}
__device__ __forceinline__ float gs_value(const GsWords<float>& g) { return __uint_as_float((uint32_t)g.w[0]); }
__device__ __forceinline__ double gs_value(const GsWords<double>& g) {
  return __hiloint2double((int)(uint32_t)g.w[1], (int)(uint32_t)g.w[0]);
}

__host__ __device__ inline int gs_pitch(int M) { return (M + 31) & ~31; }

// K * gs_pitch(min(H, W)) <= blockDim.x, a multiple of the pitch. xchg: the credits of
// gridDim.x blocks, kGsLine words apart, then their rings; zeroed. Null with one block, which
// then does all iterations (at most K).
template <typename T>
struct GsArgs {
  int H, W;
  T* p;
  int64_t ldp;
  const T* div;
  int64_t ldd;
  Masks m;
  double alpha, rb;
  int iterations, K;
  uint64_t* xchg;
};

// What a loader has on its way for its entry of one diagonal.
template <typename T, bool PLANES>
struct GsSlot {
  T p, d;
  GsWords<T> g;
  uint8_t f[4];  // face masks left, right, down, up
};

// FIRST: the chain's first block, which starts from p. ROLE: 0 a thread that updates and
// loads, 1 updates only, 2 loads only (a warp has one role; each role's registers are its own).
template <typename T, bool PLANES, bool FIRST, int ROLE>
__device__ __forceinline__ void gs_run(const GsArgs<T>& g, int* s_lost, unsigned char* smem) {
  const bool rows = g.H <= g.W;  // x is the row, else the column
  const int M = rows ? g.H : g.W, N = rows ? g.W : g.H;
  const int D = M + N - 1;
  const int Mp = gs_pitch(M);
  const int K = g.K, R = 2 * K + 2;
  double* sa = reinterpret_cast<double*>(smem);       // [R][Mp] alpha * divergence
  T* sp = reinterpret_cast<T*>(sa + (size_t)R * Mp);  // [R][Mp] iterate
  uint8_t* sc = reinterpret_cast<uint8_t*>(sp + (size_t)R * Mp);  // [R][Mp] codes
  const int tid = threadIdx.x;
  const int k = min(K, g.iterations - (int)blockIdx.x * K);
  const bool last = blockIdx.x == gridDim.x - 1;
  const int ring = kGsRing * Mp * GsWords<T>::N;
  uint64_t* out = g.xchg + (int64_t)gridDim.x * kGsLine + (int64_t)blockIdx.x * ring;
  const uint64_t* in = out - ring;
  uint32_t* credit_out = reinterpret_cast<uint32_t*>(g.xchg + (int64_t)blockIdx.x * kGsLine);  // of the next block
  uint32_t* credit_in = credit_out - 2 * kGsLine;  // this block's, to the one before
  auto slot = [&](int d, int x) { return ((d & (kGsRing - 1)) * Mp + x) * GsWords<T>::N; };

  // ---- loading: entry lx (the last Mp threads) of one diagonal after the other, always from
  // some valid address (y held to the grid) and without a branch, so that nothing waits for a
  // load before its diagonal's turn
  const int lx = tid - ((int)blockDim.x - Mp), lc = min(max(lx, 0), M - 1);
  GsSlot<T, PLANES> q[kGsAhead];
  const T* fp = g.p + (rows ? (int64_t)lc * g.ldp : lc);
  const T* fd = g.div + (rows ? (int64_t)lc * g.ldd : lc);
  const uint8_t* fu = g.m.fmu + (rows ? (int64_t)lc * g.m.ldu : lc);
  const uint8_t* fv = g.m.fmv + (rows ? (int64_t)lc * g.m.ldv : lc);
  int fy = -lc;  // y of the next diagonal to fetch
  // whether the pointer lies on a plane of h rows of w values, ld apart
  auto on_plane = [&](auto* at, auto* base, int h, int w, int64_t ld) {
    return at >= base && (at - base) / ld < h && (at - base) % ld < w;
  };
  auto fetch = [&](int d, int u) {
    if (FIRST)
      q[u].p = SG_IN_BOUNDS(on_plane(fp, (const T*)g.p, g.H, g.W, g.ldp)) ? *fp : (T)0;
    else if (SG_IN_BOUNDS(slot(d, lc) >= 0 && slot(d, lc) + GsWords<T>::N <= ring))
      gs_get(in + slot(d, lc), q[u].g);
    q[u].d = SG_IN_BOUNDS(on_plane(fd, g.div, g.H, g.W, g.ldd)) ? *fd : (T)0;
    if (PLANES && SG_IN_BOUNDS(on_plane(fu, g.m.fmu, g.H, g.W, g.m.ldu) && on_plane(fv, g.m.fmv, g.H, g.W, g.m.ldv))) {
      q[u].f[0] = fu[0];
      q[u].f[1] = fu[1];
      q[u].f[2] = fv[0];
      q[u].f[3] = fv[g.m.ldv];
    }
    const bool on = fy >= 0 && fy < N - 1;
    if (FIRST) fp += !on ? 0 : rows ? 1 : g.ldp;
    fd += !on ? 0 : rows ? 1 : g.ldd;
    if (PLANES) {
      fu += !on ? 0 : rows ? 1 : g.m.ldu;
      fv += !on ? 0 : rows ? 1 : g.m.ldv;
    }
    ++fy;
  };
  // codes of an open box or a ring of solid cells (e = 1) from a part for x and one for y
  const int e = g.m.mode == SG_MASK_RING ? 1 : 0;
  const uint32_t xlo = rows ? K_D : K_L, xhi = rows ? K_U : K_R, ylo = rows ? K_L : K_D, yhi = rows ? K_R : K_U;
  const bool xin = lx >= e && lx <= M - 1 - e;
  const uint32_t xc = (lx > e ? xlo : 0u) | (lx < M - 1 - e ? xhi : 0u);
  auto keep = [&](int row, int d, int u) {
    if (ROLE == 2 || lx >= 0) {
      const int y = d - lx;
      const bool on = lx < M && y >= 0 && y < N;
      T v = q[u].p;
      if (!FIRST) {
        if (on && !gs_there(q[u].g, (uint32_t)d + 1)) {
          int spins = 0;
          do {
            if (++spins > kGsSpins) *(volatile int*)s_lost = 1;
            gs_get(in + slot(d, lc), q[u].g);
          } while (!gs_there(q[u].g, (uint32_t)d + 1) && *(volatile int*)s_lost == 0);
        }
        // a block that never came (waits.cuh) leaves no usable iterate: say so in p, down the chain
        const bool lose = lose_waits(blockIdx.x);
        if (lose) *(volatile int*)s_lost = 1;
        v = gs_there(q[u].g, (uint32_t)d + 1) && !lose ? gs_value(q[u].g) : (T)__int_as_float(0x7fc00000);
      }
      uint32_t c;
      if (PLANES) {
        const uint8_t* f = q[u].f;
        c = faces_code(f[0] != 0, f[1] != 0, f[2] != 0, f[3] != 0, g.H, g.W, rows ? lx : y, rows ? y : lx);
      } else {
        c = xc | (y > e ? ylo : 0u) | (y < N - 1 - e ? yhi : 0u);
        c = xin && y >= e && y <= N - 1 - e && c ? c | K_FLUID : 0u;
      }
      const int o = row * Mp + lx;
      if (SG_IN_BOUNDS(row >= 0 && row < R && lx >= 0 && lx < Mp)) {
        sp[o] = on ? v : (T)0;
        sa[o] = g.alpha * (double)q[u].d;
        sc[o] = (uint8_t)(on ? c : 0);
      }
    }
    __syncwarp();  // the lanes leave the polls at different times
  };

  // ---- updating: entry cx of the diagonal that sweep cs is at
  const int cs = tid / Mp, cx = tid - cs * Mp;
  const bool own = cs < k && cx < M;
  const int xm = cx > 0 ? -1 : 0, xp = cx < M - 1 ? 1 : 0;
  T* const px = g.p + (rows ? (int64_t)cx * g.ldp : cx);
  const int64_t py = rows ? 1 : g.ldp;
  // ring entries of this thread's cell on diagonals d - 1, d, d + 1 (d = t - 2 cs)
  int o = (cs ? R - 2 * cs : 0) * Mp + cx, om = o >= Mp ? o - Mp : o + (R - 1) * Mp, op = o;
  T v = (T)0, m0 = (T)0;
  double a = 0.0;
  uint32_t c = 0;

  // ring row of diagonal d is d mod R; diagonals 0 and 1 first, 2 .. kGsAhead + 1 on the way
  if (ROLE != 1) {
    fetch(0, 0);
    keep(0, 0, 0);
    fetch(1, 0);
    keep(1, 1, 0);
#pragma unroll
    for (int u = 0; u < kGsAhead; ++u) fetch(2 + u, u);
  }
  __syncthreads();
  if (ROLE != 2 && own) {
    v = sp[o];
    a = sa[o];
    c = sc[o];
  }
  const int steps = D + 2 * (k - 1);
  int rn = 2;    // ring row of diagonal t + 2
  int read = 0;  // diagonals that the next block is known to have read
  for (int t0 = 0; t0 < steps; t0 += kGsAhead) {  // the last round may run past the last step: nothing is on the grid
    if (ROLE != 2 && !last) {
      const int need = min(t0 + kGsAhead - 2 * (k - 1), D) - kGsRing;  // read before this round's diagonals go out
      int spins = 0;
      while (read < need && *(volatile int*)s_lost == 0) {
        if (++spins > kGsSpins) *(volatile int*)s_lost = 1;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(read) : "l"(credit_out) : "memory");
      }
      __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < kGsAhead; ++u) {
      const int t = t0 + u;
      if (ROLE != 2) {
        op += Mp;
        op -= op >= R * Mp ? R * Mp : 0;
        if (own && SG_IN_BOUNDS(om + xm >= 0 && om < R * Mp && o >= 0 && o < R * Mp && op >= 0 && op + xp < R * Mp)) {
          const int d = t - 2 * cs, y = d - cx;
          const T m1 = sp[om + xm], p0 = sp[op], p1 = sp[op + xp];
          const double an = sa[op];
          const uint32_t cn = sc[op];
          // no branch before the store: as ternaries around the loads, the four faces were
          // branches taken apart by the edge cells
          const T l = pick(c & K_L, rows ? m0 : m1, v);
          const T r = pick(c & K_R, rows ? p0 : p1, v);
          const T dn = pick(c & K_D, rows ? m1 : m0, v);
          const T up = pick(c & K_U, rows ? p1 : p0, v);
          T sum = l + r;
          sum = sum + dn;
          sum = sum + up;
          m0 = pick(c & K_FLUID, (T)(((double)sum + a) * g.rb), v);
          if (y >= 0 && y < N) {
            sp[o] = m0;
            if (cs == k - 1) {
              if (last)
                px[(int64_t)y * py] = m0;
              else
                gs_put(out + slot(d, cx), m0, (uint32_t)d + 1);
            }
          }
          v = p0;
          a = an;
          c = cn;
        }
        om = o;
        o = op;
      }
      if (ROLE != 1) {
        // diagonal t + 2 takes the ring row of t - 2 K, which no sweep reads any more
        keep(rn, t + 2, u);
        fetch(t + 2 + kGsAhead, u);
        if (++rn == R) rn = 0;
      }
      __syncthreads();
      // diagonals to t + 2 have left the ring in global memory
      if (ROLE != 1 && !FIRST && lx == 0 && ((t + 3) & (kGsCredit - 1)) == 0)
        asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(credit_in), "r"(t + 3) : "memory");
    }
  }
}

template <typename T, bool PLANES>
__global__ void __launch_bounds__(kGsThreads, 1) k_gauss_seidel_wave(__grid_constant__ const GsArgs<T> g) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  __shared__ int s_lost;
  if (threadIdx.x == 0) s_lost = 0;
  __syncthreads();
  const int Mp = gs_pitch(min(g.H, g.W));
  const bool apart = g.K * Mp < (int)blockDim.x;  // the loaders are warps of their own
  const bool loader = (int)threadIdx.x >= (int)blockDim.x - Mp;
  if (apart && !loader)
    gs_run<T, PLANES, false, 1>(g, &s_lost, gs_smem);
  else if (apart && blockIdx.x == 0)
    gs_run<T, PLANES, true, 2>(g, &s_lost, gs_smem);
  else if (apart)
    gs_run<T, PLANES, false, 2>(g, &s_lost, gs_smem);
  else if (blockIdx.x == 0)
    gs_run<T, PLANES, true, 0>(g, &s_lost, gs_smem);
  else
    gs_run<T, PLANES, false, 0>(g, &s_lost, gs_smem);
  count_lost_wait(s_lost);  // every step ends with a barrier
}

// ------------------------------------------------------------------ host side
struct GsPlan {
  int K, blocks, threads;  // sweeps a block, blocks a launch
};

template <typename T>
static size_t gs_smem_bytes(int M, int K) {
  return (size_t)(2 * K + 2) * gs_pitch(M) * (sizeof(double) + sizeof(T) + 1);
}

template <typename T>
static GsPlan gs_plan(int M, int iterations, int blocks) {
  GsPlan g{0, 0, 0};
  if (M > kGsThreads || iterations <= 0 || blocks <= 0) return g;
  const int Mp = gs_pitch(M);
  const int most = std::min(kGsThreads / Mp, (int)(kGsMaxSmem / gs_smem_bytes<T>(M, 0)) - 1);
  if (most <= 0) return g;
  const int want = blocks == 1 ? most : std::min(most, std::max(1, kGsCells / Mp));
  const int passes = (int)(((int64_t)iterations + (int64_t)most * blocks - 1) / ((int64_t)most * blocks));
  const int per_pass = (iterations + passes - 1) / passes;
  g.blocks = std::min(blocks, (per_pass + want - 1) / want);
  g.K = (per_pass + g.blocks - 1) / g.blocks;
  g.blocks = (per_pass + g.K - 1) / g.K;
  g.threads = std::min(kGsThreads / Mp, g.K + 1) * Mp;
  return g;
}

template <typename T>
int64_t gauss_seidel_workspace(int M, int iterations) {
  const GsPlan g = gs_plan<T>(M, iterations, sm_count());
  if (g.blocks <= 1) return 0;
  return (int64_t)g.blocks * 8 * (kGsLine + (int64_t)kGsRing * gs_pitch(M) * GsWords<T>::N);
}
template int64_t gauss_seidel_workspace<float>(int, int);
template int64_t gauss_seidel_workspace<double>(int, int);

template <typename T>
int gauss_seidel_wave(int H, int W, T* p, int64_t ldp, const T* div, int64_t ldd, const Masks& m, double alpha,
                      double rb, int iterations, void* workspace, bool* ran, cudaStream_t s) {
  const int M = std::min(H, W);
  const GsPlan g = gs_plan<T>(M, iterations, workspace ? sm_count() : 1);
  *ran = g.K > 0;
  if (g.K <= 0) return SG_OK;
  const size_t smem = gs_smem_bytes<T>(M, g.K);
  const void* f = m.mode == SG_MASK_PLANES ? (const void*)k_gauss_seidel_wave<T, true>
                                           : (const void*)k_gauss_seidel_wave<T, false>;
  cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kGsMaxSmem);
  if (e != cudaSuccess) return fail(SG_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  for (int done = 0; done < iterations; done += g.K * g.blocks) {
    const int n = std::min(iterations - done, g.K * g.blocks);
    const int blocks = (n + g.K - 1) / g.K;
    GsArgs<T> a{H, W, p, ldp, div, ldd, m, alpha, rb, n, g.K, (uint64_t*)workspace};
    void* args[] = {&a};
    if (blocks == 1) {
      e = cudaLaunchKernel(f, dim3(1), dim3(g.threads), args, smem, s);
    } else {  // the blocks wait for one another, so they have to be on the chip together
      e = cudaMemsetAsync(workspace, 0, (size_t)gauss_seidel_workspace<T>(M, iterations), s);
      if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(f, dim3(blocks), dim3(g.threads), args, smem, s);
    }
    note_launch();
    if (e != cudaSuccess) return fail(SG_ERR_CUDA, "Gauss-Seidel: %s", cudaGetErrorString(e));
  }
  return check_launch("Gauss-Seidel");
}
template int gauss_seidel_wave<float>(int, int, float*, int64_t, const float*, int64_t, const Masks&, double, double,
                                      int, void*, bool*, cudaStream_t);
template int gauss_seidel_wave<double>(int, int, double*, int64_t, const double*, int64_t, const Masks&, double,
                                       double, int, void*, bool*, cudaStream_t);

}  // namespace sg

SG_BOUNDS_ACCESSOR(gauss_seidel)
SG_WAITS_ACCESSOR(gauss_seidel)
