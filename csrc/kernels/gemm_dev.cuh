// Device helpers that the tcgen05 GEMM kernels share.
#pragma once
#include "gemm_bf16.cuh"

#include "../common/sm100.cuh"

namespace oxb {

namespace {

__device__ __forceinline__ void red_add_v4_f32(float* p, float a, float b, float c, float d) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(a), "f"(b), "f"(c),
               "f"(d)
               : "memory");
}
// SiLU / tanh-GELU on the special-function unit (approximate reciprocal and tanh: the result is
// rounded to bf16 anyway); a full-precision divide and tanhf cost tens of instructions per value in
// an epilogue that only one warp per scheduler runs.
__device__ __forceinline__ float act_fn(float x, int act) {
  if (act == 0) return __fdividef(x, 1.f + __expf(-x));
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.7978845608028654f * (x + 0.044715f * x * x * x)));
  return 0.5f * x * (1.f + t);
}

// NG groups of 32 accumulator columns of this thread's TMEM lane: all loads are issued before the
// one wait (a load-wait pair costs a few hundred cycles).
template <int NG>
__device__ __forceinline__ void tmem_load_cols(uint32_t taddr, float (&a)[NG * 32]) {
  uint32_t r[NG][32];
#pragma unroll
  for (int g = 0; g < NG; ++g) tmem_ld_32x32b_x32(taddr + g * 32, r[g]);
  tmem_ld_wait();
#pragma unroll
  for (int g = 0; g < NG; ++g)
#pragma unroll
    for (int j = 0; j < 32; ++j) a[g * 32 + j] = __uint_as_float(r[g][j]);
}

// First tile of every group (tiles of `tile_rows` rows) and its row count, by one warp: starts[n_groups] is the sum.
__device__ __forceinline__ void group_tiles(const GemmParams& p, int tile_rows, int lane, int* starts, int* rows) {
  int acc = 0;
  for (int e0 = 0; e0 < p.n_groups; e0 += 32) {
    const int e = e0 + lane;
    const int n = e >= p.n_groups ? 0 : (p.group_counts != nullptr ? static_cast<int>(__ldcg(p.group_counts + e)) : p.M);
    const int tiles = (n + tile_rows - 1) / tile_rows;
    int incl = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (e < p.n_groups) {
      starts[e] = acc + incl - tiles;
      rows[e] = n;
    }
    acc += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) starts[p.n_groups] = acc;
}

}  // namespace

}  // namespace oxb
