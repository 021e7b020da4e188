// One small product per head: out[t, h, :] = in[t, h, :] W_h, for every token t and head h.
//
// Mixers that cache a latent instead of keys and values move the keys' and values'
// per-head up-projections to the query and to the output (see latent_attention.cu): the query
// of head h becomes q_plain W_uk,h (a [dim] row times a [dim, rank] matrix) and the head's
// output (sum of probabilities x latents) W_uv,h^T (a [rank] row times [rank, vdim]).  Both
// are this kernel; the weight of head h is reached by three strides (head, inner index, output
// index), so either storage order can be read.  float32: IEEE multiply-adds on 64 x 64 tiles
// (tile_gemm.cuh).  bfloat16 with the weight's inner index contiguous: the tensor cores
// (mma_tile.cuh), float32 accumulation; any other bfloat16 layout takes the float32 tiles.
// An output gate may ride on the epilogue (fused): out[t, h, n] *= sigmoid(gate[t, h, n]) with float32 logits
// reached by strides of their own (a column stride of 0: one logit a head), so a mixer that gates its merged heads needs
// no kernel for it.
#include "head_rows.cuh"
#include "mma_tile.cuh"
#include "tile_gemm.cuh"

namespace rl {

template <typename T>
__global__ __launch_bounds__(256) void head_linear_kernel(const T* __restrict__ in, long in_tok, long in_head,
                                                          const T* __restrict__ w, long w_head, long w_k, long w_n,
                                                          T* __restrict__ out, long out_tok, long out_head,
                                                          int n_tokens, int k_total, int n_total,
                                                          const float* __restrict__ gate, long gate_tok, long gate_head,
                                                          long gate_n) {
  __shared__ TileGemmSmem s;
  pdl_begin();
  const int h = blockIdx.z;
  const int m0 = blockIdx.x * TG_M, n0 = blockIdx.y * TG_N;
  const T* in_h = in + (size_t)h * in_head;
  const T* w_h = w + (size_t)h * w_head;
  float acc[4][4] = {};
  tile_gemm(
      acc, k_total,
      [&](int m, int k) {
        return (m0 + m < n_tokens && k < k_total) ? to_f32(in_h[(size_t)(m0 + m) * in_tok + k]) : 0.f;
      },
      [&](int k, int n) {
        return (n0 + n < n_total && k < k_total) ? to_f32(w_h[(size_t)k * w_k + (size_t)(n0 + n) * w_n]) : 0.f;
      },
      s);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= n_tokens) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < n_total) {
        float v = acc[i][j];
        if (gate != nullptr) v *= 1.0f / (1.0f + expf(-gate[(size_t)m * gate_tok + (size_t)h * gate_head + n * gate_n]));
        out[(size_t)m * out_tok + (size_t)h * out_head + n] = from_f32<T>(v);
      }
    }
  }
}

// bfloat16 on the tensor cores; the weight's inner index is contiguous (w_k == 1).
template <bool VEC>
__global__ __launch_bounds__(128) void head_linear_mma_kernel(const __nv_bfloat16* __restrict__ in, long in_tok,
                                                              long in_head, const __nv_bfloat16* __restrict__ w,
                                                              long w_head, long w_n, __nv_bfloat16* __restrict__ out,
                                                              long out_tok, long out_head, int n_tokens, int k_total,
                                                              int n_total, const float* __restrict__ gate,
                                                              long gate_tok, long gate_head, long gate_n) {
  __shared__ __align__(16) MmaTileSmem s;
  pdl_begin();
  const int h = blockIdx.z;
  const int m0 = blockIdx.x * MT_M, n0 = blockIdx.y * MT_N;
  const __nv_bfloat16* in_h = in + (size_t)h * in_head;
  const __nv_bfloat16* w_h = w + (size_t)h * w_head;
  float acc[2][4][4] = {};
  mma_tile<VEC>(
      acc, k_total, [&](int m) { return m0 + m < n_tokens ? in_h + (size_t)(m0 + m) * in_tok : nullptr; },
      [&](int n) { return n0 + n < n_total ? w_h + (size_t)(n0 + n) * w_n : nullptr; }, s);
  if (gate == nullptr && (((uintptr_t)out & 3) | (uintptr_t)((out_tok | out_head | n_total) & 1)) == 0) {
    // neighbouring columns together: single bfloat16 stores were what a prompt's product waited for
    mma_for_each(acc, [&](int m, int n, int mi, int ni, int c) {
      if ((c & 1) == 0 && m0 + m < n_tokens && n0 + n < n_total)
        *reinterpret_cast<__nv_bfloat162*>(out + (size_t)(m0 + m) * out_tok + (size_t)h * out_head + n0 + n) =
            __floats2bfloat162_rn(acc[mi][ni][c], acc[mi][ni][c + 1]);
    });
    return;
  }
  mma_for_each(acc, [&](int m, int n, int mi, int ni, int c) {
    if (m0 + m < n_tokens && n0 + n < n_total) {
      float v = acc[mi][ni][c];
      if (gate != nullptr) v *= 1.0f / (1.0f + expf(-gate[(size_t)(m0 + m) * gate_tok + (size_t)h * gate_head + (n0 + n) * gate_n]));
      out[(size_t)(m0 + m) * out_tok + (size_t)h * out_head + n0 + n] = __float2bfloat16_rn(v);
    }
  });
}

// At most 16 rows of bfloat16 (a decode step of few requests): eight warps a block, each eight columns and KB blocks of 64
// elements of K; `parts` warps share columns, their sums meeting in shared memory in a fixed order.  What bounds it is latency:
// one round trip for the input's rows after the wait.  Eight rows, 16 heads, 512 to 128 columns: 10.3 us on 64 x 64
// tiles (32 blocks, sixteen steps of K one after the other).
constexpr int HR_WARPS = 8, HR_MAX_K = 4 * 64 * HR_WARPS;
template <int KB>
__global__ __launch_bounds__(32 * HR_WARPS) void head_rows_kernel(const __nv_bfloat16* in, long in_tok, long in_head,
                                                                  const __nv_bfloat16* __restrict__ w, long w_head, long w_n,
                                                                  __nv_bfloat16* __restrict__ out, long out_tok, long out_head,
                                                                  int n_tokens, int n_total, int parts, const float* gate,
                                                                  long gate_tok, long gate_head, long gate_n, int w_settled) {
  __shared__ float part_s[HR_WARPS][32][4];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, j = lane & 3;
  const int h = blockIdx.y, per_block = HR_WARPS / parts;
  const int part = warp / per_block, n0 = (blockIdx.x * per_block + warp % per_block) * 8, k0 = part * KB * 64;
  HeadRowsWeights<KB> weights;
  if (!w_settled) asm volatile("griddepcontrol.wait;" ::: "memory");  // the caller promises nothing
  weights.load(w + (size_t)h * w_head + (size_t)min(n0 + g, n_total - 1) * w_n + k0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const __nv_bfloat16* in_h = in + (size_t)h * in_head + k0;
  float c[4];
  weights.multiply(in_h + (size_t)min(g, n_tokens - 1) * in_tok, in_h + (size_t)min(g + 8, n_tokens - 1) * in_tok, c);
  if (parts > 1) {
    *reinterpret_cast<float4*>(part_s[warp][lane]) = make_float4(c[0], c[1], c[2], c[3]);
    __syncthreads();
    if (part != 0) return;
    for (int q = 1; q < parts; ++q) {
      const float4 o = *reinterpret_cast<const float4*>(part_s[q * per_block + warp][lane]);
      c[0] += o.x, c[1] += o.y, c[2] += o.z, c[3] += o.w;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = g + (i >> 1) * 8, n = n0 + 2 * j + (i & 1);
    if (t < n_tokens && n < n_total) {
      float v = c[i];
      if (gate != nullptr) v *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_tok + (size_t)h * gate_head + n * gate_n]));
      out[(size_t)t * out_tok + (size_t)h * out_head + n] = __float2bfloat16_rn(v);
    }
  }
}

}  // namespace rl

// in: element (t, h, k) at in + t*in_tok + h*in_head + k; w: element (h, k, n) at
// w + h*w_head + k*w_k + n*w_n; out: element (t, h, n) at out + t*out_tok + h*out_head + n.
// gate: null, or float32 logits, element (t, h, n) at gate + t*gate_tok + h*gate_head + n*gate_n: out *=
// sigmoid(gate).  w_settled: w was written by work that was over before the kernel preceding this call on the stream began (weights);
// the kernel of up to 16 rows then asks for it before its wait for the kernels ahead.
RL_EXPORT int rl_head_linear(int dtype, const void* in, long in_tok, long in_head, const void* w, long w_head, long w_k,
                             long w_n, void* out, long out_tok, long out_head, int n_tokens, int n_heads, int k_total,
                             int n_total, const float* gate, long gate_tok, long gate_head, long gate_n, int w_settled,
                             cudaStream_t stream) {
  if (n_tokens <= 0) return 0;
  if (n_heads <= 0 || n_heads > 65535 || k_total <= 0 || n_total <= 0) return -2;
  const dim3 grid((n_tokens + rl::TG_M - 1) / rl::TG_M, (n_total + rl::TG_N - 1) / rl::TG_N, n_heads);
  if (grid.y > 65535) return -2;
  if (dtype == RL_F32)
    rl::launch_pdl(rl::head_linear_kernel<float>, grid, 256, 0, stream, (const float*)in, in_tok, in_head,
                   (const float*)w, w_head, w_k, w_n, (float*)out, out_tok, out_head, n_tokens, k_total, n_total, gate,
                   gate_tok, gate_head, gate_n);
  else if (w_k == 1) {
    const bool vec = k_total % 8 == 0 && in_tok % 8 == 0 && in_head % 8 == 0 && w_head % 8 == 0 && w_n % 8 == 0 &&
                     ((uintptr_t)in % 16) == 0 && ((uintptr_t)w % 16) == 0;
    const int kbs = k_total / 64;
    if (vec && n_tokens <= 16 && k_total % 64 == 0 && k_total <= rl::HR_MAX_K) {
      // two blocks of 64 a warp while eight warps reach that far, else four; a power of two of warps along K
      int parts = 1;
      while (parts < rl::HR_WARPS && parts * 2 < kbs) parts *= 2;
      const int kb = kbs / parts;
      if (kb * parts == kbs && (kb == 1 || kb == 2 || kb == 4)) {
        const int columns = 8 * (rl::HR_WARPS / parts);
        auto kernel = kb == 1 ? rl::head_rows_kernel<1> : kb == 2 ? rl::head_rows_kernel<2> : rl::head_rows_kernel<4>;
        rl::launch_pdl(kernel, dim3((n_total + columns - 1) / columns, n_heads), 32 * rl::HR_WARPS, 0, stream, (const __nv_bfloat16*)in,
                       in_tok, in_head, (const __nv_bfloat16*)w, w_head, w_n, (__nv_bfloat16*)out, out_tok, out_head, n_tokens, n_total,
                       parts, gate, gate_tok, gate_head, gate_n, w_settled);
        RL_CHECK_LAUNCH();
        return 0;
      }
    }
    auto kernel = vec ? rl::head_linear_mma_kernel<true> : rl::head_linear_mma_kernel<false>;
    rl::launch_pdl(kernel, grid, 128, 0, stream, (const __nv_bfloat16*)in, in_tok, in_head, (const __nv_bfloat16*)w,
                   w_head, w_n, (__nv_bfloat16*)out, out_tok, out_head, n_tokens, k_total, n_total, gate, gate_tok, gate_head, gate_n);
  } else
    rl::launch_pdl(rl::head_linear_kernel<__nv_bfloat16>, grid, 256, 0, stream, (const __nv_bfloat16*)in, in_tok,
                   in_head, (const __nv_bfloat16*)w, w_head, w_k, w_n, (__nv_bfloat16*)out, out_tok, out_head, n_tokens,
                   k_total, n_total, gate, gate_tok, gate_head, gate_n);
  RL_CHECK_LAUNCH();
  return 0;
}
