// The interface of gemm_f32_tc.cu to gemm_simt.cu.
#pragma once
#include "common.cuh"

namespace rl {
namespace f32tc {

// Shorter sums stay on the CUDA cores: what the accumulators cut off is about two units in a sum's last place however long it is,
// the roundings of FMAs grow with its length, and by 256 elements are the larger (csrc/gemm_f32_tc.cu).
constexpr int MIN_K = 256;
// Whether operands lie as the kernel's copies need them: on 16-byte boundaries, rows of a whole number of 16-byte pieces.
bool takes(const void* a, long lda, const void* w, int K, const int* status);
// What a product is expected to take, in microseconds, in the tile width that takes the least (*width).
double time_us(int M, int N, int K, int* width);
// Launches it; 0 or the error of the launch (or of the tensor maps).
int run(const float* a, long lda, const float* w, const float* bias, float* out, long ldo, int M, int N, int K, int act, int residual,
        int width, int* status, cudaStream_t stream);

}  // namespace f32tc
}  // namespace rl
