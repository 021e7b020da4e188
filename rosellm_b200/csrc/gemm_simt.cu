// Matrix products on the CUDA cores: out[M,N] = A[M,K] * W[N,K]^T, with the epilogues the
// model needs fused in: + bias[N]; GELU; and accumulation into a float32 residual stream.
//
// This is the matrix path of the 32-bit mode (IEEE float32 FMA; products of many rows whose columns and inner size
// are large go to gemm_f32_tc.cu, which holds its operands in full and rounds less often), and the small-batch path of the bfloat16
// mode, where a product streams the weights once and is bound by memory, not arithmetic.  The formulas fused here:
//   y = a W + b                           rosellm/rosetrainer/model.py:95, 220, 334-337
//   gelu_tanh(u) = 0.5 u (1 + tanh(sqrt(2/pi) (u + 0.044715 u^3)))   model.py:274-277,
//                                                                    fused_mlp.py:79-89
//   gelu_erf(u)  = 0.5 u (1 + erf(u / sqrt 2))                       model.py:345-346 (F.gelu)
//   x = x + y (residual)                  model.py:412-413, 424-428; fused_mlp.py:91-113
#include "gemm_epilogue.cuh"
#include "gemm_f32_tc.cuh"

namespace rl {

// Tiles of bfloat16: 64x64 output tile per block of 256 threads, 4x4 outputs per thread, K in steps of 16.
// Each output's sum runs over k in ascending order whatever M is, so a row's result does
// not depend on which other rows share the launch.
template <typename TIn, typename TOut>
__global__ __launch_bounds__(256) void gemm_tile_kernel(
    const TIn* __restrict__ A, long lda, const TIn* __restrict__ W, const float* __restrict__ bias,
    TOut* __restrict__ out, long ldo, int M, int N, int K, int act, int residual) {
  constexpr int BM = 64, BN = 64, BK = 16;
  pdl_begin();
  __shared__ __align__(16) float As[BK][BM + 4];
  __shared__ __align__(16) float Ws[BK][BN + 4];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float ra[4], rw[4];
  auto fetch = [&](int k0) {
    const int k = k0 + lk;
    const int m = m0 + lrow, n = n0 + lrow;
    if (m < M && k < K) load4(A + (size_t)m * lda + k, ra);
    else { ra[0] = ra[1] = ra[2] = ra[3] = 0.f; }
    if (n < N && k < K) load4(W + (size_t)n * K + k, rw);
    else { rw[0] = rw[1] = rw[2] = rw[3] = 0.f; }
  };
  fetch(0);
  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      As[lk + i][lrow] = ra[i];
      Ws[lk + i][lrow] = rw[i];
    }
    __syncthreads();
    if (k0 + BK < K) fetch(k0 + BK);
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 b4 = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
      const float a[4] = {a4.x, a4.y, a4.z, a4.w};
      const float b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias != nullptr) v += bias[n];
      v = apply_act(v, act);
      store_out<TOut>(out, (size_t)m * ldo + n, v, residual);
    }
  }
}

// Tiles of float32.  BM x BN output tile per block, TM x TN outputs per thread (rows and columns of a thread lie a
// thread grid apart), K in steps of 16 that travel by cp.async, as they lie in memory, through a ring of three buffers of
// shared memory (rows 80 bytes apart: the eight rows of a 16-byte access phase hit different banks).
// Each output's sum runs over k in ascending order whatever M is and whatever the tile is, so a row's result does
// not depend on which other rows share the launch (nor does it hang on M whether a product of many rows comes here: f32tc::ahead).  What bounds it: reads of shared memory, 12 pieces of 16 bytes a thread for 128
// FMAs with 8 x 4 outputs (about 19 of the 37.2 TFMA/s; the form before, 64 x 64 tiles of 4 x 4 outputs transposed through registers with
// two barriers a step, 9 to 16).  Pairs of FMAs in one instruction (fma.rn.f32x2) measured the same and add up in another order.
template <int BM, int BN, int TM, int TN>
__global__ __launch_bounds__((BM / TM) * (BN / TN)) void gemm_tile_f32_kernel(
    const float* __restrict__ A, long lda, const float* __restrict__ W, const float* __restrict__ bias,
    float* __restrict__ out, long ldo, int M, int N, int K, int act, int residual) {
  constexpr int BK = 16, STAGES = 3, LD = 20;  // floats between two rows in shared memory
  constexpr int GX = BN / TN, GY = BM / TM, THREADS = GX * GY;
  constexpr int PIECES = (BM + BN) * 4 / THREADS;  // 16-byte pieces of a step a thread copies
  static_assert((BM + BN) * 4 % THREADS == 0, "pieces are shared evenly");
  extern __shared__ __align__(16) float tile_s[];  // [STAGES][BM + BN][LD]: rows of A, then of W
  const int tid = threadIdx.x, tx = tid % GX, ty = tid / GX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int steps = (K + BK - 1) / BK;
  const float* src[PIECES];
  uint32_t dst[PIECES];
  bool there[PIECES];
#pragma unroll
  for (int q = 0; q < PIECES; ++q) {
    const int i = tid + THREADS * q, row = i >> 2, piece = i & 3;
    const bool of_a = row < BM;
    const int r = of_a ? m0 + row : n0 + row - BM;
    there[q] = r < (of_a ? M : N);
    src[q] = (of_a ? A + (size_t)(there[q] ? r : 0) * lda : W + (size_t)(there[q] ? r : 0) * K) + 4 * piece;
    dst[q] = (uint32_t)__cvta_generic_to_shared(tile_s + row * LD + 4 * piece);
  }
  auto copy = [&](int step) {  // what lies outside the matrices arrives as zeros
    const uint32_t at = (uint32_t)(step % STAGES) * ((BM + BN) * LD * 4);
#pragma unroll
    for (int q = 0; q < PIECES; ++q) {
      const bool in = there[q] && step * BK + 4 * (int)(tid & 3) < K;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst[q] + at), "l"(src[q] + (in ? step * BK : 0)),
                   "r"(in ? 16 : 0)
                   : "memory");
    }
  };
  pdl_begin();
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) copy(s);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // the step's pieces are there for all, and all have left the buffer that is filled now
    if (step + STAGES - 1 < steps) copy(step + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* a_s = tile_s + (step % STAGES) * ((BM + BN) * LD) + ty * LD;
    const float* w_s = tile_s + (step % STAGES) * ((BM + BN) * LD) + (BM + tx) * LD;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      float4 w[TN];
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(w_s + j * GX * LD + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(a_s + i * GY * LD + kk);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + i * GY + ty;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + j * GX + tx;
      if (n >= N) continue;
      float v = acc[i][j];
      if (bias != nullptr) v += bias[n];
      v = apply_act(v, act);
      store_out<float>(out, (size_t)m * ldo + n, v, residual);
    }
  }
}

// Few rows of float32 (decoded tokens).  PARTS of a block's eight warps share a group of COLS output columns, ROWS rows at a
// time: they take the chunks of 128 elements of K in turn, a lane four elements of each, so that every piece of the weights that a
// lane holds meets all the rows in registers.  A lane's weights travel by cp.async into a ring of its own in shared memory (it
// reads back only what it copied itself, so no barrier is needed), two chunks ahead, and the first of them before the wait
// for the kernels ahead.  The COLS * ROWS sums of a lane are added over the lanes by halving exchanges (each lane gives away half
// of what it has left), then over the group's warps in shared memory: in an order that is the same for every row whatever M is.
constexpr int ROWS_COLS = 4, ROWS_STAGES = 3;
template <int ROWS, int PARTS>
__global__ __launch_bounds__(256, 2) void gemm_rows_f32_kernel(const float* A, long lda, const float* __restrict__ W,
                                                               const float* __restrict__ bias, float* __restrict__ out, long ldo,
                                                               int M, int N, int K, int act, int residual, KvScatter kv) {
  constexpr int COLS = ROWS_COLS, STAGES = ROWS_STAGES, VALUES = COLS * ROWS, AHEAD = STAGES - 1, GROUPS = 8 / PARTS;
  extern __shared__ __align__(128) float4 rows_ring[];  // [warp][stage][column][lane]
  __shared__ __align__(128) float part_s[2][GROUPS][PARTS][VALUES];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mine = warp / PARTS, part = warp % PARTS;
  const int groups = (N + COLS - 1) / COLS, chunks = (K + 127) / 128, stride = (int)gridDim.x * GROUPS;
  float4* ring = rows_ring + (size_t)warp * STAGES * COLS * 32 + lane;
  const uint32_t ring_addr = (uint32_t)__cvta_generic_to_shared(ring);
  // what the warp copies next: of a group its chunks, those once for every ROWS rows, then its next group
  int c_group = part < chunks ? (int)blockIdx.x * GROUPS + mine : groups, c_chunk = part, c_m0 = 0, c_stage = 0;
  auto copy = [&]() {
    if (c_group < groups) {
      const int k = c_chunk * 128 + 4 * lane;
#pragma unroll
      for (int c = 0; c < COLS; ++c)  // beyond K: zeros
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring_addr + (uint32_t)(c_stage * COLS + c) * 512),
                     "l"(W + (size_t)min(c_group * COLS + c, N - 1) * K + (k < K ? k : 0)), "r"(k < K ? 16 : 0)
                     : "memory");
      if (++c_stage == STAGES) c_stage = 0;
      if ((c_chunk += PARTS) >= chunks) {
        c_chunk = part;
        if ((c_m0 += ROWS) >= M) c_m0 = 0, c_group += stride;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
#pragma unroll
  for (int s = 0; s < AHEAD; ++s) copy();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  int buf = 0, stage = 0;
  // the epilogue's thread: a column of a row of one of the groups
  const int e_mine = tid / VALUES, e_value = tid % VALUES;
  for (int first = (int)blockIdx.x * GROUPS; first < groups; first += stride) {
    const bool there = first + mine < groups;
    const int n = (first + e_mine) * COLS + e_value % COLS;
    const bool n_there = e_mine < GROUPS && n < N;
    const float b = n_there && bias != nullptr ? bias[n] : 0.f;
    for (int m0 = 0; m0 < M; m0 += ROWS, buf ^= 1) {
      float acc[VALUES];  // [row][column]
#pragma unroll
      for (int i = 0; i < VALUES; ++i) acc[i] = 0.f;
      if (there)
        for (int chunk = part; chunk < chunks; chunk += PARTS) {
          copy();  // into the stage that was read last
          asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD) : "memory");
          float4 w[COLS];
#pragma unroll
          for (int c = 0; c < COLS; ++c) w[c] = ring[(stage * COLS + c) * 32];
          if (++stage == STAGES) stage = 0;
          const int k = chunk * 128 + 4 * lane;
#pragma unroll
          for (int r = 0; r < ROWS; ++r) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            if (k < K) a = *reinterpret_cast<const float4*>(A + (size_t)min(m0 + r, M - 1) * lda + k);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
              float& t = acc[r * COLS + c];
              t = fmaf(a.x, w[c].x, t);
              t = fmaf(a.y, w[c].y, t);
              t = fmaf(a.z, w[c].z, t);
              t = fmaf(a.w, w[c].w, t);
            }
          }
        }
      // after the exchange over lane bit o, a lane keeps the half of its values whose index has that bit as its own;
      // with one value left the lanes add it up
#pragma unroll
      for (int o = 16, half = VALUES / 2; o > 0; o >>= 1, half >>= 1) {
        const bool upper = (lane & o) != 0;
        if (half == 0) {
          acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], o);
          continue;
        }
#pragma unroll
        for (int i = 0; i < VALUES / 2; ++i) {
          if (i >= half) break;
          const float give = upper ? acc[i] : acc[i + half];
          const float keep = upper ? acc[i + half] : acc[i];
          acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
      }
      part_s[buf][mine][part][lane / (32 / VALUES)] = acc[0];  // fewer values than lanes: neighbours hold the same one
      __syncthreads();  // the other buffer takes the next sums, so one barrier is enough
      const int m = m0 + e_value / COLS;
      if (n_there && m < M) {
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < PARTS; ++q) v += part_s[buf][e_mine][q][e_value];
        v = apply_act(v + b, act);
        if (!scatter_kv<float>(kv, m, n, v)) store_out<float>(out, (size_t)m * ldo + n, v, residual);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// Few rows of bfloat16.  A block of four warps computes 4 / KSPLIT output columns for all
// rows: KSPLIT warps share a column, each taking a contiguous part of K, and their partial
// sums meet in shared memory in a fixed order.  Lanes split a warp's part of K in 16-byte
// pieces and four pieces of the weight row are in flight per lane before any is used, so that
// a weight matrix is streamed from memory once, with enough loads outstanding to keep the
// memory system busy even when the matrix has few rows of its own.
template <typename TIn, typename TOut, int MB, int KSPLIT>
__global__ __launch_bounds__(128) void gemm_rows_kernel(
    const TIn* __restrict__ A, long lda, const TIn* __restrict__ W,
    const float* __restrict__ bias, TOut* __restrict__ out, long ldo, int M, int N, int K, int act,
    int residual, KvScatter kv) {
  constexpr int VEC = Vec16<TIn>::N;
  constexpr int U = 4;
  constexpr int COLS = 4 / KSPLIT;
  extern __shared__ __align__(16) uint8_t rows_smem[];
  float* part_s = reinterpret_cast<float*>(rows_smem);          // [4][MB]
  pdl_begin();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * COLS + warp / KSPLIT;
  const int part = warp % KSPLIT;
  const int k_part = ((K + KSPLIT - 1) / KSPLIT + VEC - 1) / VEC * VEC;
  const int k_begin = part * k_part;
  const int k_end = min(K, k_begin + k_part);
  const bool active = n < N;
  const TIn* w = W + (size_t)(active ? n : 0) * K;
  const float b = (bias != nullptr && active) ? bias[n] : 0.f;
  for (int m0 = 0; m0 < M; m0 += MB) {
    float acc[MB];
#pragma unroll
    for (int i = 0; i < MB; ++i) acc[i] = 0.f;
    if (active) {
      for (int k0 = k_begin + lane * VEC; k0 < k_end; k0 += 32 * VEC * U) {
        float wv[U][VEC];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int k = k0 + u * 32 * VEC;
          if (k < k_end) {
            Vec16<TIn>::load(w + k, wv[u]);
          } else {
#pragma unroll
            for (int v = 0; v < VEC; ++v) wv[u][v] = 0.f;
          }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const int k = k0 + u * 32 * VEC;
          if (k >= k_end) break;
#pragma unroll
          for (int i = 0; i < MB; ++i) {
            if (m0 + i < M) {
              float av[VEC];
              Vec16<TIn>::load(A + (size_t)(m0 + i) * lda + k, av);
#pragma unroll
              for (int v = 0; v < VEC; ++v) acc[i] = fmaf(av[v], wv[u][v], acc[i]);
            }
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < MB; ++i) acc[i] = warp_sum(acc[i]);
    if (KSPLIT > 1) {
      __syncthreads();  // part_s may still be read for the previous group of rows
      if (lane == 0) {
#pragma unroll
        for (int i = 0; i < MB; ++i) part_s[warp * MB + i] = acc[i];
      }
      __syncthreads();
      if (lane == 0 && part == 0) {
#pragma unroll
        for (int i = 0; i < MB; ++i) {
          float t = 0.f;
#pragma unroll
          for (int q = 0; q < KSPLIT; ++q) t += part_s[(warp + q) * MB + i];
          acc[i] = t;
        }
      }
    }
    if (lane == 0 && part == 0 && active) {
#pragma unroll
      for (int i = 0; i < MB; ++i) {
        if (m0 + i < M) {
          const float v = apply_act(acc[i] + b, act);
          if (!scatter_kv<TIn>(kv, m0 + i, n, v)) store_out<TOut>(out, (size_t)(m0 + i) * ldo + n, v, residual);
        }
      }
    }
  }
}

template <typename TIn, typename TOut, int MB>
static void launch_rows(const TIn* a, long lda, const TIn* w, const float* bias, TOut* o,
                        long ldo, int M, int N, int K, int act, int residual, const KvScatter& kv,
                        cudaStream_t stream) {
  // enough warps to keep loads in flight on every SM: split K among warps while columns are few
  constexpr int VEC = Vec16<TIn>::N;
  int ks = 1;
  while (ks < 4 && (long)N * ks < 3000 && K / (ks * 2) >= 32 * VEC && (M <= 4 || N <= 1024)) ks *= 2;
  const size_t smem = 4 * MB * sizeof(float);
  const int cols = 4 / ks;
  const int blocks = (N + cols - 1) / cols;
#define RL_ROWS(KS)                                                                                       \
  do {                                                                                                    \
    if (smem > 48 * 1024)                                                                                 \
      cudaFuncSetAttribute(gemm_rows_kernel<TIn, TOut, MB, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                           (int)smem);                                                                    \
    launch_pdl(gemm_rows_kernel<TIn, TOut, MB, KS>, blocks, 128, smem, stream, a, lda, w, bias, o, ldo, \
               M, N, K, act, residual, kv);                                                               \
  } while (0)
  if (ks == 1) RL_ROWS(1);
  else if (ks == 2) RL_ROWS(2);
  else RL_ROWS(4);
#undef RL_ROWS
}

static int simt_sm_count() {
  static int n_sms = 0;
  if (n_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (n_sms <= 0) n_sms = 1;
  }
  return n_sms;
}

template <int BM, int BN, int TM, int TN>
static void launch_tile_f32_form(const float* a, long lda, const float* w, const float* bias, float* o, long ldo, int M, int N, int K,
                                 int act, int residual, cudaStream_t stream) {
  constexpr size_t smem = 3 * (size_t)(BM + BN) * 20 * 4;
  static bool attr_set = false;
  if (!attr_set) {
    if (smem > 48 * 1024)
      note_launch(cudaFuncSetAttribute(gemm_tile_f32_kernel<BM, BN, TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = true;
  }
  launch_pdl(gemm_tile_f32_kernel<BM, BN, TM, TN>, dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3((BM / TM) * (BN / TN)), smem,
             stream, a, lda, w, bias, o, ldo, M, N, K, act, residual);
}

// What a form of tile takes at K 768 (us) by how many of its tiles fall to an SM, measured in a chain of products and straight in
// between; another K scales all forms alike.  A block alone is bound by its own chain of steps, and up to four, four and
// six blocks an SM run beside one another; already from a third of the SMs on some SMs are given two (the next
// launch's blocks are placed while the one ahead still runs).
struct TileTime {
  double tiles, us;
};
constexpr TileTime TIME_64X64[] = {{0.33, 32.2}, {0.6, 44.4}, {0.85, 69.8}, {1.1, 79.3}, {2.5, 90.1}, {4, 94.5}, {5, 128}, {8, 180}, {11, 250}};
constexpr TileTime TIME_32X64[] = {{0.35, 20.6}, {0.65, 30.8}, {0.85, 35.4}, {1.1, 51.3}, {1.5, 52.7}, {2, 58.5}, {4.5, 63.8}, {5.2, 78.1},
                                   {8, 104.6}, {14, 174.5}};
constexpr TileTime TIME_32X32[] = {{0.5, 17.1}, {0.8, 21.7}, {1.2, 29.5}, {1.7, 38.5}, {2.1, 51.1}, {3, 52.4}, {4, 61.5}, {6.4, 61.5},
                                   {8, 69.4}, {14, 109.7}, {30, 225.7}};

template <int POINTS>
static double tile_time(const TileTime (&time)[POINTS], double tiles) {
  if (tiles <= time[0].tiles) return time[0].us;
  int i = 1;
  while (i < POINTS - 1 && tiles > time[i].tiles) ++i;
  return time[i - 1].us + (time[i].us - time[i - 1].us) * (tiles - time[i - 1].tiles) / (time[i].tiles - time[i - 1].tiles);
}

// The tile that ends first.  Over 161 products of 65 to 2048 rows (64 to 4096 columns, K 256 to 6400) the choice is 1% behind the
// fastest form on average; by counting rounds of tiles it was 7%, up to 45% (1600 x 1600 at 300 rows: 146, 99 and 120 us on 64 x 64,
// 32 x 64 and 32 x 32; 768 x 768 at 600 rows 66, 56 and 59).  128 x 64, and 8 x 8 outputs a thread, measured slower throughout.
static dim3 tile_f32_for(int M, int N) {
  const int sms = simt_sm_count();
  auto cost = [&](int bm, int bn, const auto& time) {
    const long down = (M + bm - 1) / bm, tiles = down * ((N + bn - 1) / bn);
    if (down > 65535) return 1e30;  // the limit of a grid's second extent: the tiles of 64 rows go furthest
    return tile_time(time, (double)tiles / sms);
  };
  const double large = cost(64, 64, TIME_64X64), middle = cost(32, 64, TIME_32X64), small = cost(32, 32, TIME_32X32);
  return large <= middle && large <= small ? dim3(64, 64) : middle <= small ? dim3(32, 64) : dim3(32, 32);
}

static void launch_tile_f32(const float* a, long lda, const float* w, const float* bias, float* o, long ldo, int M, int N, int K,
                            int act, int residual, cudaStream_t stream) {
  const dim3 tile = tile_f32_for(M, N);  // rows, columns
  if (tile.x == 64) launch_tile_f32_form<64, 64, 8, 4>(a, lda, w, bias, o, ldo, M, N, K, act, residual, stream);
  else if (tile.y == 64) launch_tile_f32_form<32, 64, 4, 4>(a, lda, w, bias, o, ldo, M, N, K, act, residual, stream);
  else launch_tile_f32_form<32, 32, 4, 2>(a, lda, w, bias, o, ldo, M, N, K, act, residual, stream);
}

template <int ROWS, int PARTS>
static void launch_rows_f32_parts(const float* a, long lda, const float* w, const float* bias, float* o, long ldo, int M, int N, int K,
                                  int act, int residual, const KvScatter& kv, int blocks, cudaStream_t stream) {
  constexpr size_t smem = 8 * ROWS_STAGES * ROWS_COLS * 512;  // the rings of eight warps
  static bool attr_set = false;
  if (!attr_set) {  // with the kernel's static part above 48 KB
    note_launch(cudaFuncSetAttribute(gemm_rows_f32_kernel<ROWS, PARTS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set = true;
  }
  launch_pdl(gemm_rows_f32_kernel<ROWS, PARTS>, blocks, 256, smem, stream, a, lda, w, bias, o, ldo, M, N, K, act, residual, kv);
}

template <int ROWS>
static void launch_rows_f32_form(const float* a, long lda, const float* w, const float* bias, float* o, long ldo, int M, int N, int K,
                                 int act, int residual, const KvScatter& kv, cudaStream_t stream) {
  // Warps that share a group, by the rounds of groups and what a round takes: a part that does not change with K and one for each chunk
  // a warp walks (in 8 rows about 1 us and 0.75).  Measured, 8 rows, us, two / four / eight warps: 768 x 768 3.6 / 2.9 / 2.4, 2304 x 768
  // 4.1 / 3.3 / 4.0, 3072 x 768 4.5 / 5.5 / 5.7, 4096 x 1024 5.5 / 6.2 / 7.6, 1600 x 1600 7.0 / 5.1 / 5.3, 4800 x 1600 12.2 / 11.2 / 10.8,
  // 6400 x 1600 13.4 / 12.3 / 14.2, 1600 x 6400 20.5 / 13.0 / 15.1, 50257 x 768 35.7 / 49.6 / 68.7 (43.0 with a warp a group).
  const int groups = (N + ROWS_COLS - 1) / ROWS_COLS, chunks = (K + 127) / 128, places = 2 * simt_sm_count();
  int parts = 8, turns = groups;
  float least = 0.f;
  for (int p = 8; p >= 2; p /= 2) {
    const int t = (groups + 8 / p - 1) / (8 / p);
    const float cost = (float)((t + places - 1) / places) * (1.f + 0.75f * (float)((chunks + p - 1) / p));
    if (p == 8 || cost < 0.95f * least) parts = p, turns = t, least = cost;
  }
#define RL_PARTS(PARTS) \
  launch_rows_f32_parts<ROWS, PARTS>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, min(turns, places), stream)
  if (parts == 2) RL_PARTS(2);
  else if (parts == 4) RL_PARTS(4);
  else RL_PARTS(8);
#undef RL_PARTS
}

static void launch_rows_f32(const float* a, long lda, const float* w, const float* bias, float* o, long ldo, int M, int N, int K,
                            int act, int residual, const KvScatter& kv, cudaStream_t stream) {
  if (M == 1) launch_rows_f32_form<1>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
  else if (M == 2) launch_rows_f32_form<2>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
  else if (M <= 4) launch_rows_f32_form<4>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
  else launch_rows_f32_form<8>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
}

template <typename TIn, typename TOut>
static int launch_gemm(const void* A, long lda, const void* W, const float* bias, void* out,
                       long ldo, int M, int N, int K, int act, int residual, int rows_limit,
                       const KvScatter& kv, cudaStream_t stream) {
  const TIn* a = (const TIn*)A;
  const TIn* w = (const TIn*)W;
  TOut* o = (TOut*)out;
  if (M <= rows_limit) {
    if constexpr (sizeof(TIn) == 4) {
      launch_rows_f32(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
    } else {
      if (M == 1) launch_rows<TIn, TOut, 1>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
      else if (M == 2) launch_rows<TIn, TOut, 2>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
      else if (M <= 4) launch_rows<TIn, TOut, 4>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
      else launch_rows<TIn, TOut, 8>(a, lda, w, bias, o, ldo, M, N, K, act, residual, kv, stream);
    }
  } else {
    if (kv.pool != nullptr) return -5;  // the cache scatter is fused only into the row kernel
    if constexpr (sizeof(TIn) == 4) {
      launch_tile_f32(a, lda, w, bias, o, ldo, M, N, K, act, residual, stream);
    } else {
      dim3 grid((N + 63) / 64, (M + 63) / 64);
      launch_pdl(gemm_tile_kernel<TIn, TOut>, grid, 256, 0, stream, a, lda, w, bias, o, ldo, M, N, K, act, residual);
    }
  }
  return 0;
}

}  // namespace rl

// in_dtype / out_dtype: RL_F32 or RL_BF16; out may be float32 with bfloat16 inputs.
// residual != 0: out (float32) += result.  rows_limit: up to this many rows the streaming
// kernel runs, above it the tiled one.  kv_pool != nullptr (streaming kernel): output columns
// from kv_q_width on are scattered into cache pages as keys and values.
RL_EXPORT int rl_gemm_simt(int in_dtype, int out_dtype, const void* A, long lda, const void* W,
                           const float* bias, void* out, long ldo, int M, int N, int K, int act,
                           int residual, int rows_limit, void* kv_pool,
                           const int* kv_block_table, int kv_bt_stride, const int* kv_positions,
                           const int* kv_req_of_token, const int* kv_slots, int kv_q_width, int kv_width,
                           int kv_head_dim, int kv_page_size, int kv_heads, int kv_max_pos, int* status,
                           cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 8 != 0 || lda % 8 != 0) return -2;
  if (residual && out_dtype != RL_F32) return -3;
  rl::KvScatter kv{kv_pool, kv_block_table, kv_bt_stride, kv_positions, kv_req_of_token, kv_slots,
                   kv_q_width, kv_width, kv_head_dim, kv_page_size, kv_heads, kv_max_pos, status};
  int rc;
  if (in_dtype == RL_F32 && out_dtype == RL_F32 && M > rows_limit && kv_pool == nullptr && rl::f32tc::ahead(N, K) &&
      rl::f32tc::takes(A, lda, W, K, status)) {
    rc = rl::f32tc::run((const float*)A, lda, (const float*)W, bias, (float*)out, ldo, M, N, K, act, residual,
                        rl::f32tc::width_for(M, N, K), status, stream);
    if (rc != -10 && rc != -11) return rc;  // without tensor maps: the CUDA cores
  }
  if (in_dtype == RL_F32 && out_dtype == RL_F32)
    rc = rl::launch_gemm<float, float>(A, lda, W, bias, out, ldo, M, N, K, act, residual, rows_limit, kv, stream);
  else if (in_dtype == RL_BF16 && out_dtype == RL_BF16)
    rc = rl::launch_gemm<__nv_bfloat16, __nv_bfloat16>(A, lda, W, bias, out, ldo, M, N, K, act, residual, rows_limit, kv, stream);
  else if (in_dtype == RL_BF16 && out_dtype == RL_F32)
    rc = rl::launch_gemm<__nv_bfloat16, float>(A, lda, W, bias, out, ldo, M, N, K, act, residual, rows_limit, kv, stream);
  else
    return -4;
  if (rc != 0) return rc;
  RL_CHECK_LAUNCH();
  return 0;
}

// The tile that a float32 product of so many rows and columns runs in: 100 x its rows + its columns.
RL_EXPORT int rl_gemm_tile_f32_for(int M, int N) {
  const dim3 tile = rl::tile_f32_for(M, N);
  return (int)(100 * tile.x + tile.y);
}
