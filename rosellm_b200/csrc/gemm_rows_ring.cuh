// The interface of gemm_rows_ring.cu to gemm_rows_mma.cu.
#pragma once
#include "gemm_epilogue.cuh"

namespace rl {

// LayerNorm of float32 rows as the product's input (x == nullptr: off; K <= 1024, M <= 16):
// a = (x - mean) * rsqrt(var + eps) * gamma + beta with two-pass float32 statistics
// (rosellm/rosetrainer/fused_layernorm.py:99-120), rounded to bfloat16 as the separate kernel
// stores it.  Every block normalises the few rows itself, after it has issued its first weight
// loads: that costs less than a kernel of its own between two products.
struct NormArgs {
  const float* x;
  long ldx;
  const float* gamma;
  const float* beta;
  float eps;
};

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

namespace ring {

struct Args {
  const __nv_bfloat16* a;  // [M, K], row stride lda (norm.x == nullptr)
  long lda;
  NormArgs norm;
  const __nv_bfloat16* w;  // [N, K]
  const float* bias;       // [N] or nullptr
  void* out;               // [M, N] bfloat16 or float32, row stride ldo
  long ldo;
  int M, N, K, act, residual, out_f32;
  KvScatter kv;
  int* status;
  SampleArgs sample;       // out_ids != nullptr: the rows' next tokens instead of `out` (nullptr then)
};

// Whether the kernel takes this product (sizes and alignments; see gemm_rows_ring.cu).
bool takes(const Args& p);
// Launches it; 0 or the error of the launch.
int run(const Args& p, cudaStream_t stream);

}  // namespace ring
}  // namespace rl
