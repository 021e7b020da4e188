// The interface of gemm_f32_tc.cu to gemm_simt.cu.
#pragma once
#include "common.cuh"

namespace rl {
namespace f32tc {

// Shorter sums stay on the CUDA cores, where they take no longer.
constexpr int MIN_K = 256;
// Which products of many rows run here: by their columns and inner size alone, never by their rows, so that a row's result does not
// depend on the rows beside it (the CUDA cores add in another order).  From 736 columns on (inner sizes below 768: from 1024) this kernel is ahead
// from 129 rows on; below that the CUDA cores keep all of a product's rows.  Measured, us, CUDA cores / here, at 65, 129 and 1,752 rows:
// 768 x 768 18.6 / 22.2, 22.2 / 22.4, 65 / 39; 768 x 3072 69.5 / 75, 83 / 74, 248 / 122; 1024 x 256 8.3 / 10.0, 11.5 / 10.0, 33 / 18; 2304 x 768 35 / 22, 57 / 23, 157
// / 70; and of the others 704 x 768 18.4 / 22.3, 22.5 / 22.6 (192 rows 21.6 / 22.6), 65 / 38; 768 x 256 7.4 / 9.9, 8.8 / 10.2, 25 / 19; 512 x 512
// 12.0 / 16.0, 13.9 / 16.2, 44 / 20; 256 x 1024 21.7 / 28, 21.6 / 28, 78 / 29.
inline bool ahead(int N, int K) { return K >= MIN_K && (N >= 1024 || (N >= 736 && K >= 768)); }
// Whether operands lie as the kernel's copies need them: on 16-byte boundaries, rows of a whole number of 16-byte pieces, none over another.
bool takes(const void* a, long lda, const void* w, int K, const int* status);
// The tile width that is expected to take the least time.
int width_for(int M, int N, int K);
// Launches it; 0, the error of the launch, or -10 or -11 where a tensor map could not be made (nothing is launched then).
int run(const float* a, long lda, const float* w, const float* bias, float* out, long ldo, int M, int N, int K, int act, int residual,
        int width, int* status, cudaStream_t stream);

}  // namespace f32tc
}  // namespace rl
