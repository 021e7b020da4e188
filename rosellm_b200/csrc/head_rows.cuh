// A warp's share of a per-head product of at most 16 rows on mma.sync m16n8k16, operands straight from memory into registers:
// out[t, n] = sum_k in[t, k] w[n, k] for eight columns n and KB blocks of 64 elements of K.  Lane (g = lane / 4, j = lane % 4)
// holds elements 16 j ... 16 j + 15 of row g of W and of rows g and g + 8 of the input, block by block: K is permuted alike in
// both, so that every load is 16 bytes.  The weights are asked for by a call of their own: where no kernel ahead
// writes them, before the wait for those.
#pragma once
#include "common.cuh"

namespace rl {

template <int KB>
struct HeadRowsWeights {
  uint4 w[KB][2];
  // row: this lane's row of W (column n0 + g), from the warp's first element of K on
  __device__ __forceinline__ void load(const __nv_bfloat16* row) {
    const int j = threadIdx.x & 3;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb) {
      const uint4* src = reinterpret_cast<const uint4*>(row + kb * 64 + 16 * j);
      w[kb][0] = src[0];
      w[kb][1] = src[1];
    }
  }
  // c0, c1: row g, columns 2j and 2j + 1 of the eight; c2, c3: row g + 8.  lo, hi: this lane's two rows of the input (rows
  // that do not exist repeat one that does and are not stored).
  __device__ __forceinline__ void multiply(const __nv_bfloat16* lo, const __nv_bfloat16* hi, float (&c)[4]) const {
    const int j = threadIdx.x & 3;
    uint4 a[KB][2], b[KB][2];
#pragma unroll
    for (int kb = 0; kb < KB; ++kb)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        a[kb][s] = load_in_order(reinterpret_cast<const uint4*>(lo + kb * 64 + 16 * j) + s);
        b[kb][s] = load_in_order(reinterpret_cast<const uint4*>(hi + kb * 64 + 16 * j) + s);
      }
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
    for (int kb = 0; kb < KB; ++kb)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        step(c, a[kb][s].x, b[kb][s].x, a[kb][s].y, b[kb][s].y, w[kb][s].x, w[kb][s].y);
        step(d, a[kb][s].z, b[kb][s].z, a[kb][s].w, b[kb][s].w, w[kb][s].z, w[kb][s].w);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += d[i];
  }
  static __device__ __forceinline__ void step(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
  }
};

}  // namespace rl
