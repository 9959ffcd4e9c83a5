// Transfer weights and relaxation reciprocals shared by the multigrid kernels of gmg.cu and
// batch.cu (included inside namespace sg).
#pragma once

// The fields and scale of a solve, in device memory (GmgState): the kernels of a solve's graph
// take them from here, so that one instantiated graph serves every pressure and divergence.
struct SolveFields {
  void* p;
  int64_t ldp;
  const void* div;
  int64_t ldd;
  double alpha;
  double bmean;  // mean of alpha div over the fluid cells (when the plan removes it)
};

// 1-D prolongation weight of fine index i onto coarse index I (grid of n coarse cells).
__device__ __forceinline__ float w1(int i, int I, int n) {
  int h = i >> 1;
  int x = h + ((i & 1) ? 1 : -1);
  x = x < 0 ? 0 : (x > n - 1 ? n - 1 : x);
  return (h == I ? 0.75f : 0.0f) + (x == I ? 0.25f : 0.0f);
}

// a where k has a bit of `bits`, else b; a select, never a branch
__device__ __forceinline__ float pick_bits(uint32_t k, uint32_t bits, float a, float b) {
  float o;
  asm("{.reg .pred p; .reg .b32 t; and.b32 t, %1, %2; setp.ne.u32 p, t, 0; selp.f32 %0, %3, %4, p;}"
      : "=f"(o) : "r"(k), "r"(bits), "f"(a), "f"(b));
  return o;
}
__device__ __forceinline__ double pick_bits(uint32_t k, uint32_t bits, double a, double b) {
  double o;
  asm("{.reg .pred p; .reg .b32 t; and.b32 t, %1, %2; setp.ne.u32 p, t, 0; selp.f64 %0, %3, %4, p;}"
      : "=d"(o) : "r"(k), "r"(bits), "d"(a), "d"(b));
  return o;
}

// 1 / (number of open faces), n in 1..4.
template <typename T>
__device__ __forceinline__ T rcp_open(int n) {
  return n == 4 ? (T)0.25 : (n == 3 ? (T)(1.0 / 3.0) : (n == 2 ? (T)0.5 : (T)1.0));
}
