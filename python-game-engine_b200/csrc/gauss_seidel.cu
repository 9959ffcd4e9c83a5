// Lexicographic Gauss-Seidel (gauss_seidel.py:8-26) with the sweeps of a call following one
// another down the grid. Every update evaluates the reference's expression in the reference's
// order, so the iterates are those of one sweep after the other bit for bit. Compiled with
// -fmad=false like the other operator units.
#include <algorithm>

#include "sweeps.cuh"

namespace sg {

// ------------------------------------------------------------------ lexicographic Gauss-Seidel
// Cell (j, i) of anti-diagonal d = j + i reads d - 1 (this sweep) and d + 1 (the sweep before),
// so sweep s may work on diagonal t - 2 s at step t: up to K sweeps run down the grid behind
// one another and a pass of K sweeps takes H + W - 1 + 2 (K - 1) steps, one block barrier
// each, instead of K (H + W - 1). One block; the 2 K + 2 diagonals in use lie in a shared-
// memory ring, entry x of a diagonal being the cell with coordinate x along the shorter axis
// (neighbours then are entries x, x -+ 1 of the rows beside it: unit stride, no conflicts).
// Diagonals are read from global memory kGsAhead steps before they are used and written once,
// by the pass's last sweep. 97 x 161 float32, 40 sweeps: 11.0 -> 0.80 ms. What bounds it: the chain of steps, each a barrier and (for many
// sweeps in flight) the issue of up to K x min(H, W) updates by one SM.
constexpr int kGsThreads = 1024;
constexpr int kGsAhead = 4;
constexpr int kGsMaxSmem = 220 * 1024;

template <typename T>
__global__ void __launch_bounds__(kGsThreads, 1) k_gauss_seidel_wave(int H, int W, T* p, int64_t ldp,
                                                                     const T* __restrict__ div, int64_t ldd, Masks m,
                                                                     double alpha, double rb, int iterations, int K) {
  extern __shared__ __align__(16) unsigned char gs_smem[];
  const bool rows = H <= W;  // x is the row, else the column
  const int M = rows ? H : W, N = rows ? W : H;
  const int D = H + W - 1;
  const int Mp = (M + 31) & ~31;
  const int R = 2 * K + 2;
  double* sa = reinterpret_cast<double*>(gs_smem);   // [R][Mp] alpha * divergence
  T* sp = reinterpret_cast<T*>(sa + (size_t)R * Mp);  // [R][Mp] iterate
  uint8_t* sc = reinterpret_cast<uint8_t*>(sp + (size_t)R * Mp);  // [R][Mp] codes
  const int tid = threadIdx.x;
  const int lx = rows ? 0 : 1, dx = rows ? 1 : 0;  // entry shift of the left / down neighbour
  const int tk = kGsThreads / Mp, tx = kGsThreads - tk * Mp;  // one pass over the threads, in (sweep, entry)
  T pv[kGsAhead];
  T dv[kGsAhead];
  uint32_t cv[kGsAhead];
  // entry tid of diagonal d into register slot u (nothing off the grid)
  auto fetch = [&](int d, int u) {
    cv[u] = 0;
    pv[u] = dv[u] = (T)0;
    const int y = d - tid;
    if (tid < M && y >= 0 && y < N && d < D) {
      const int j = rows ? tid : y, i = rows ? y : tid;
      pv[u] = p[(int64_t)j * ldp + i];
      dv[u] = div[(int64_t)j * ldd + i];
      cv[u] = cell_code(m, H, W, j, i);
    }
  };
  auto keep = [&](int row, int u) {
    if (tid < Mp) {
      sp[(size_t)row * Mp + tid] = pv[u];
      sa[(size_t)row * Mp + tid] = alpha * (double)dv[u];
      sc[(size_t)row * Mp + tid] = (uint8_t)cv[u];
    }
  };
  for (int done = 0; done < iterations; done += K) {
    const int k = iterations - done < K ? iterations - done : K;
    // ring row of diagonal d is d mod R; diagonals 0 and 1 first, 2 .. kGsAhead + 1 on the way
    fetch(0, 0);
    keep(0, 0);
    fetch(1, 0);
    keep(1, 0);
#pragma unroll
    for (int u = 0; u < kGsAhead; ++u) fetch(2 + u, u);
    __syncthreads();
    const int steps = D + 2 * (k - 1);
    int rt = 0;  // ring row of diagonal t
    for (int t0 = 0; t0 < steps; t0 += kGsAhead) {
#pragma unroll
      for (int u = 0; u < kGsAhead; ++u) {
        const int t = t0 + u;
        if (t >= steps) break;
        int s = tid / Mp, x = tid - s * Mp;
        while (s < k) {
          const int d = t - 2 * s;
          const int y = d - x;
          if (d >= 0 && x < M && y >= 0 && y < N) {
            int rd = rt - 2 * s;
            if (rd < 0) rd += R;
            const int rm = (rd == 0 ? R - 1 : rd - 1) * Mp, rp = (rd == R - 1 ? 0 : rd + 1) * Mp;
            const int o = rd * Mp + x;
            const uint32_t c = sc[o];
            if (c & K_FLUID) {
              const T v = sp[o];
              const T l = (c & K_L) ? sp[rm + x - lx] : v;
              const T r = (c & K_R) ? sp[rp + x + lx] : v;
              const T dn = (c & K_D) ? sp[rm + x - dx] : v;
              const T up = (c & K_U) ? sp[rp + x + dx] : v;
              T q = l + r;
              q = q + dn;
              q = q + up;
              const T n = (T)(((double)q + sa[o]) * rb);
              sp[o] = n;
              if (s == k - 1) p[rows ? (int64_t)x * ldp + y : (int64_t)y * ldp + x] = n;
            }
          }
          s += tk;
          x += tx;
          if (x >= Mp) {
            x -= Mp;
            ++s;
          }
        }
        // diagonal t + 2 takes the ring row of t - 2 K, which no sweep reads any more
        int rn = rt + 2;
        if (rn >= R) rn -= R;
        keep(rn, u);
        fetch(t + 2 + kGsAhead, u);
        if (++rt == R) rt = 0;
        __syncthreads();
      }
    }
  }
}

template <typename T>
static size_t gs_smem_bytes(int M, int K) {
  return (size_t)(2 * K + 2) * ((M + 31) & ~31) * (sizeof(double) + sizeof(T) + 1);
}

// Sweeps in flight per pass that the ring has room for, spread evenly over the passes; 0: the
// shorter side is too long.
template <typename T>
static int gs_in_flight(int M, int iterations) {
  if (M > kGsThreads) return 0;
  int k = iterations;
  while (k > 0 && gs_smem_bytes<T>(M, k) > kGsMaxSmem) --k;
  if (k <= 0) return 0;
  const int passes = (iterations + k - 1) / k;
  return (iterations + passes - 1) / passes;
}

template <typename T>
int gauss_seidel_wave(int H, int W, T* p, int64_t ldp, const T* div, int64_t ldd, const Masks& m, double alpha,
                      double rb, int iterations, bool* ran, cudaStream_t s) {
  const int M = std::min(H, W);
  const int k = gs_in_flight<T>(M, iterations);
  *ran = k > 0;
  if (k <= 0) return SG_OK;
  const size_t smem = gs_smem_bytes<T>(M, k);
  cudaError_t e = cudaFuncSetAttribute(k_gauss_seidel_wave<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return fail(SG_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
  SG_LAUNCH(k_gauss_seidel_wave<T><<<1, kGsThreads, smem, s>>>(H, W, p, ldp, div, ldd, m, alpha, rb, iterations, k));
  return check_launch("sg_gauss_seidel_solve");
}
template int gauss_seidel_wave<float>(int, int, float*, int64_t, const float*, int64_t, const Masks&, double, double,
                                      int, bool*, cudaStream_t);
template int gauss_seidel_wave<double>(int, int, double*, int64_t, const double*, int64_t, const Masks&, double,
                                       double, int, bool*, cudaStream_t);

}  // namespace sg
