// float32 products of many rows (prompt portions of the 32-bit mode) on the tensor cores of sm_100a:
//
//   out[M,N] = A[M,K] * W[N,K]^T  (+ bias[N]) (GELU) (or out += ..., the float32 residual stream)
//
// the products and epilogues of gemm_simt.cu (rosellm/rosetrainer/model.py:95, 220, 334-337; fused_mlp.py:79-113).  An
// operand is the sum of three bfloat16 numbers, x = hi + mid + lo, each the nearest to what is left: 8 + 8 + 8 bits hold all 24 of a
// float32 number, and its range is bfloat16's, so nothing is left out.  Eight of the nine products of the parts are
// made, each exact in the multiplier; lo lo is left out, at most 2^-34 of the product.  What costs a sum on this unit its bits is the
// accumulator, which cuts off instead of rounding: so hi hi (16 bits a product) and the seven small products have an accumulator each.  The
// first is drained after CHUNK K blocks of 32 and added in registers with ordinary float32 additions, one rounding a drain as an FMA has
// one a product; the small one, of 2^-8 of its size, is drained after SPAN K blocks and at the end.  (Two parts of eleven bits, in tf32, are 6 to
// 16% faster and leave out up to 2^-21 of a product: a sum of one product was up to 7.4 x 2^-24 off, an FMA is 1.0, this 1.0.)
//
// One block per SM walks tiles of 128 rows x BN columns.  Its warps:
//   warp 0      one lane copies tiles of A and W (K blocks of 32 floats = 128 bytes, 128-byte swizzle) by TMA into a ring of
//               stages; those of W for the first stages before the wait for the kernels ahead;
//   warps 2-9   cut what arrived: the 128 bytes of a row take its hi (64 bytes) and its mid behind them, the first half of a
//               row of 128 bytes in the stage's second half its lo, all in the swizzle of the copy;
//   warp 1      one lane issues tcgen05.mma kind::f16 (bfloat16), sixteen of K 16 a K block;
//   warps 10-17 drain the accumulators (two of each in turn) and write the tile.
// What bounds it: a K block goes through four roles, each with a wait on the one before; no unit is full.  Of 3072 x 768 at 1,752
// rows (ncu, 128 columns): tensor pipe 40%, shared memory's pipe 57% (a K block of 128 x 128 is read once and written one and a half times by the
// cutting warps and read eight times in parts by the products), issue slots 46%.  A K block takes 1.04 us where the tensor pipe needs 0.55; narrow
// tiles are all chain, 0.75 us a K block.
//
// Measured on B200 in chains of products, 1,752 rows, us (the CUDA-core tiles, this kernel): 2304 x 768 157, 70; 3072 x 768 218, 103; 768 x 768
// 65, 38; 768 x 3072 247, 116; 1600 x 6400 932, 428.  129 rows: 768 x 768 22.2, 22.5; 2304 x 768 56.6, 22.7; 1600 x 1600 73, 41.
// Error against 64 bits (2-norm of the difference over that of the FMAs' difference): dense sums 0.25 (K 256), 0.21 (768), 0.19 (3072); sums
// of one product 1.00, of two to sixteen 0.5 to 1.1; of positive numbers 0.26 to 0.19.
//
// Sums that are not finite are worked out again with FMAs from memory, in the order of the CUDA-core kernels, each by itself: those with an
// infinity or NaN among their operands, those that overflow on the way (a product of hi parts does before the FMA with it does), and
// those with an operand that three parts do not hold (above 3.39e38, or with bits below 2^-133), which becomes NaN in the cutting.
// Every wait on a barrier is bounded (status bit, abort flag), as in gemm_tc.cu.
#include "gemm_epilogue.cuh"
#include "gemm_f32_tc.cuh"
#include "tc_common.cuh"

namespace rl {
namespace f32tc {

constexpr int BM = 128, BK = 32;
constexpr int CUT_WARPS = 8, EPI_WARPS = 8, THREADS = 32 * (2 + CUT_WARPS + EPI_WARPS);
constexpr int CHUNK = 1;  // K blocks between two additions in registers
constexpr int SPAN = 128;  // K blocks between two drains of the small products' accumulator; a multiple of CHUNK
constexpr int MAX_STAGES = 4;
constexpr int A_BYTES = BM * BK * 4;
__host__ __device__ constexpr int operand_bytes(int bn) { return A_BYTES + bn * BK * 4; }
__host__ __device__ constexpr int stages_of(int bn) {
  const int fit = (227 * 1024 - 2048) / (2 * operand_bytes(bn));
  return fit > MAX_STAGES ? MAX_STAGES : fit;
}
// 1024 for alignment | stages of (hi, in x's place | lo) | barriers full, cut, empty [MAX_STAGES], acc_full, acc_empty [2],
// the tensor-memory address and the abort flag
__host__ __device__ constexpr int smem_bytes(int bn) { return 1024 + stages_of(bn) * 2 * operand_bytes(bn) + (3 * MAX_STAGES + 4) * 8 + 16; }

struct Args {
  const float* a;
  long lda;
  const float* w;
  const float* bias;
  float* out;
  long ldo;
  int M, N, K, act, residual;
  int* status;
};

// Two neighbouring numbers' nearest bfloat16 ones, the first in the lower half, and what is left of the numbers (exactly).
__device__ __forceinline__ uint32_t take_part(float& x, float& y) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const uint32_t bits = *reinterpret_cast<const uint32_t*>(&h);
  x -= __uint_as_float(bits << 16);
  y -= __uint_as_float(bits & 0xffff0000u);
  return bits;
}
// A call, not sixteen inlined copies, of four values at a time: one after the other their latencies would add up.
__device__ __noinline__ float4 act_call(float4 v, int act) {
  return make_float4(apply_act(v.x, act), apply_act(v.y, act), apply_act(v.z, act), apply_act(v.w, act));
}

// A sum of the product by FMAs in ascending order, as the CUDA-core kernels add (K a multiple of 4, both on 16-byte boundaries).
__device__ __noinline__ float sum_of_fmas(const float* a, const float* w, int K) {
  float t = 0.f;
  for (int k = 0; k < K; k += 32) {
    float4 x[8], y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {  // beyond K: the first numbers again, and not used
      const int at = k + 4 * i < K ? k + 4 * i : 0;
      x[i] = *reinterpret_cast<const float4*>(a + at);
      y[i] = *reinterpret_cast<const float4*>(w + at);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (k + 4 * i < K) t = fmaf(x[i].w, y[i].w, fmaf(x[i].z, y[i].z, fmaf(x[i].y, y[i].y, fmaf(x[i].x, y[i].x, t))));
  }
  return t;
}

template <int BN>
__global__ __launch_bounds__(THREADS, 1) void gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                 const __grid_constant__ CUtensorMap map_w, const Args p) {
  constexpr int OPERANDS = operand_bytes(BN), STAGE = 2 * OPERANDS, STAGES = stages_of(BN);
  constexpr uint32_t TMEM_COLS = 4 * BN;  // two accumulators of hi hi, two of the small products
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t smem_base = tc::smem_u32(smem), bar_base = smem_base + STAGES * STAGE;
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto cut_bar = [&](int s) { return bar_base + 8u * (MAX_STAGES + s); };
  auto empty_bar = [&](int s) { return bar_base + 8u * (2 * MAX_STAGES + s); };
  auto acc_full = [&](int b) { return bar_base + 8u * (3 * MAX_STAGES + b); };
  auto acc_empty = [&](int b) { return bar_base + 8u * (3 * MAX_STAGES + 2 + b); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + STAGES * STAGE + (3 * MAX_STAGES + 4) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int m_tiles = (p.M + BM - 1) / BM, units = m_tiles * ((p.N + BN - 1) / BN), kbs = (p.K + BK - 1) / BK;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      tc::mbar_init(full_bar(s), 1);
      tc::mbar_init(cut_bar(s), CUT_WARPS);
      tc::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(acc_full(b), 1);
      tc::mbar_init(acc_empty(b), EPI_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc::tma_prefetch_map(&map_a);
    tc::tma_prefetch_map(&map_w);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(tmem_slot)), "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  // The copying and the issuing warp walk their loops whole, with values that are the same in all lanes; one lane issues.
  if (warp == 0) {
    int ahead = 0;  // stages whose W tiles are asked for before the kernels ahead have ended
    if ((int)blockIdx.x < units) {
      ahead = kbs < STAGES ? kbs : STAGES;
      const int n0 = ((int)blockIdx.x / m_tiles) * BN;
      for (int s = 0; s < ahead; ++s)
        if (tc::elect_one()) {
          tc::mbar_expect_tx(full_bar(s), OPERANDS);
          tc::tma_load_2d(smem_base + s * STAGE + A_BYTES, &map_w, full_bar(s), s * BK, n0);
        }
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int it = 0, s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const int m0 = (unit % m_tiles) * BM, n0 = (unit / m_tiles) * BN;
      for (int kb = 0; kb < kbs; ++kb, ++it) {
        if (it >= ahead) {
          ok = tc::mbar_wait_warp(empty_bar(s), ph ^ 1u, abort_flag, p.status);  // a stage's first use: passes at once
          if (!ok) break;
        }
        if (tc::elect_one()) {
          if (it >= ahead) {
            tc::mbar_expect_tx(full_bar(s), OPERANDS);
            tc::tma_load_2d(smem_base + s * STAGE + A_BYTES, &map_w, full_bar(s), kb * BK, n0);
          }
          tc::tma_load_2d(smem_base + s * STAGE, &map_a, full_bar(s), kb * BK, m0);
        }
        __syncwarp();
        if (++s == STAGES) s = 0, ph ^= 1u;
      }
    }
    if (*abort_flag)
      for (int k = it > STAGES ? it - STAGES : 0; k < it; ++k) tc::mbar_wait_quiet(full_bar(k % STAGES), (uint32_t)(k / STAGES) & 1u);
  } else if (warp == 1) {
    constexpr uint32_t idesc = tc::instr_desc(BN);
    const uint64_t desc0 = tc::smem_desc(smem_base);
    // (an accumulator of the small products is written again two spans on, when the chunk after the one it was drained with has been
    // drained as well: the wait for the main accumulator says so)
    int s = 0, chunk = 0, span = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x)
      for (int kb0 = 0; kb0 < kbs && ok; kb0 += CHUNK, ++chunk) {
        const int buf = chunk & 1;
        ok = tc::mbar_wait_warp(acc_empty(buf), ((uint32_t)(chunk >> 1) & 1u) ^ 1u, abort_flag, p.status);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t main = tmem_base + (uint32_t)(buf * BN), small = tmem_base + (uint32_t)((2 + (span & 1)) * BN);
        for (int kb = kb0; kb < min(kb0 + CHUNK, kbs); ++kb) {
          ok = tc::mbar_wait_warp(cut_bar(s), ph, abort_flag, p.status);
          if (!ok) break;
          const uint64_t a = desc0 + (uint64_t)(s * (STAGE >> 4)), w = a + (A_BYTES >> 4);
          if (tc::elect_one()) {
            // the parts of a row: descriptors count 16-byte units, a K step of 16 numbers is two of them
            constexpr uint32_t HI = 0, MID = 4, LO = OPERANDS >> 4;
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) {
              const uint32_t more = kb > kb0 || k > 0 ? 1u : 0u, small_more = kb % SPAN != 0 || k > 0 ? 1u : 0u;
              tc::mma_f16(small, a + LO + 2 * k, w + MID + 2 * k, idesc, small_more);
              tc::mma_f16(small, a + MID + 2 * k, w + LO + 2 * k, idesc, 1u);
              tc::mma_f16(small, a + LO + 2 * k, w + HI + 2 * k, idesc, 1u);
              tc::mma_f16(small, a + HI + 2 * k, w + LO + 2 * k, idesc, 1u);
              tc::mma_f16(small, a + MID + 2 * k, w + MID + 2 * k, idesc, 1u);
              tc::mma_f16(small, a + MID + 2 * k, w + HI + 2 * k, idesc, 1u);
              tc::mma_f16(small, a + HI + 2 * k, w + MID + 2 * k, idesc, 1u);
              tc::mma_f16(main, a + HI + 2 * k, w + HI + 2 * k, idesc, more);
            }
            tc::mma_commit(empty_bar(s));
          }
          __syncwarp();
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
        if (ok && tc::elect_one()) tc::mma_commit(acc_full(buf));
        __syncwarp();
        if ((kb0 + CHUNK) % SPAN == 0 || kb0 + CHUNK >= kbs) ++span;
      }
  } else if (warp < 2 + CUT_WARPS) {
    // A warp cuts eight rows at a time, lane (r = lane / 4, c = lane % 4) the numbers 8 c ... 8 c + 7 of row r: the 16-byte pieces 2 c and
    // 2 c + 1 of its 128 bytes, which become piece c of hi, of mid (piece 4 + c) and of lo; piece p of row r lies at p ^ r.  Odd rows store mid
    // first, so that eight lanes' stores meet all banks.
    constexpr int GROUPS = (BM + BN) / 8, TURNS = (GROUPS + CUT_WARPS - 1) / CUT_WARPS;
    const int r = lane >> 2, c = lane & 3, first = r & 1 ? 4 : 0;
    int s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x)
      for (int kb = 0; kb < kbs; ++kb) {
        ok = tc::mbar_wait_warp(full_bar(s), ph, abort_flag, p.status);
        if (!ok) break;
        uint8_t* rows = smem + s * STAGE + (size_t)((warp - 2) * 8 + r) * 128;
        float4 v[TURNS][2];
#pragma unroll
        for (int i = 0; i < TURNS; ++i)
          if (warp - 2 + i * CUT_WARPS < GROUPS)
#pragma unroll
            for (int h = 0; h < 2; ++h) v[i][h] = *reinterpret_cast<const float4*>(rows + i * CUT_WARPS * 1024 + (((2 * c + h) ^ r) << 4));
        __syncwarp();  // all of the warp's rows have been read: they are written over
#pragma unroll
        for (int i = 0; i < TURNS; ++i)
          if (warp - 2 + i * CUT_WARPS < GROUPS) {
            float x[8] = {v[i][0].x, v[i][0].y, v[i][0].z, v[i][0].w, v[i][1].x, v[i][1].y, v[i][1].z, v[i][1].w};
            uint32_t part[3][4];
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
              for (int e = 0; e < 4; ++e) part[q][e] = take_part(x[2 * e], x[2 * e + 1]);
            uint8_t* row = rows + i * CUT_WARPS * 1024;
            const uint4 hi = make_uint4(part[0][0], part[0][1], part[0][2], part[0][3]);
            const uint4 mid = make_uint4(part[1][0], part[1][1], part[1][2], part[1][3]);
            *reinterpret_cast<uint4*>(row + (((first + c) ^ r) << 4)) = first ? mid : hi;
            *reinterpret_cast<uint4*>(row + (((4 - first + c) ^ r) << 4)) = first ? hi : mid;
            uint4* lo = reinterpret_cast<uint4*>(row + OPERANDS + ((c ^ r) << 4));
            *lo = make_uint4(part[2][0], part[2][1], part[2][2], part[2][3]);
            // a rest that is not finite, or left beyond bfloat16's least number (else all are +0): NaN in its place, so that the row's sums
            // are worked out anew
            uint32_t rest = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) rest |= __float_as_uint(x[e]);
            if (rest != 0) lo->x = 0x7fff7fffu;
          }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(cut_bar(s)) : "memory");
        if (++s == STAGES) s = 0, ph ^= 1u;
      }
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int COLS = BN / 2;                    // of a thread: its row's, in one half of the tile
    constexpr int STEP = 16;
    const int quarter = warp & 3, part = (warp - 2 - CUT_WARPS) >> 2;
    const bool vec = p.ldo % 4 == 0 && (uintptr_t)p.out % 16 == 0;
    int chunk = 0, span = 0;
    bool ok = true;
    for (int unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
      const int row = (unit % m_tiles) * BM + quarter * 32 + lane, n0 = (unit / m_tiles) * BN + part * COLS;
      float acc[COLS];
#pragma unroll
      for (int i = 0; i < COLS; ++i) acc[i] = 0.f;
      for (int kb0 = 0; kb0 < kbs; kb0 += CHUNK, ++chunk) {
        const int buf = chunk & 1;
        ok = tc::mbar_wait_warp(acc_full(buf), (uint32_t)(chunk >> 1) & 1u, abort_flag, p.status);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t mine = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * COLS);
        auto add = [&](uint32_t from) {
#pragma unroll
          for (int c = 0; c < COLS; c += STEP) {
            uint32_t r[STEP];
            tc::tmem_load16(from + c, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < STEP; ++i) acc[c + i] += __uint_as_float(r[i]);
          }
        };
        add(mine + (uint32_t)(buf * BN));
        if ((kb0 + CHUNK) % SPAN == 0 || kb0 + CHUNK >= kbs) add(mine + (uint32_t)((2 + (span++ & 1)) * BN));
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty(buf)) : "memory");
      }
      if (!ok) break;
      uint32_t again[(COLS + 31) / 32] = {};  // columns whose sums are not finite
      float* out = p.out + (size_t)row * p.ldo + n0;
      if (row < p.M) {
#pragma unroll
        for (int c = 0; c < COLS; c += 4) {
          if (n0 + c >= p.N) break;
          float v[4];
          uint32_t odd = 0;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            v[i] = acc[c + i];
            if (n0 + c + i >= p.N) continue;
            odd |= (uint32_t)((__float_as_uint(v[i]) & 0x7f800000u) == 0x7f800000u) << i;
            if (p.bias != nullptr) v[i] += p.bias[n0 + c + i];
          }
          again[c / 32] |= odd << (c % 32);
          if (p.act != RL_ACT_NONE) {
            const float4 t = act_call(make_float4(v[0], v[1], v[2], v[3]), p.act);
            v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
          }
          if (vec && odd == 0 && n0 + c + 3 < p.N) {
            float4 t = make_float4(v[0], v[1], v[2], v[3]);
            if (p.residual) {
              const float4 old = *reinterpret_cast<const float4*>(out + c);
              t.x += old.x, t.y += old.y, t.z += old.z, t.w += old.w;
            }
            *reinterpret_cast<float4*>(out + c) = t;
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n0 + c + i < p.N && (odd >> i & 1) == 0) out[c + i] = p.residual ? out[c + i] + v[i] : v[i];
          }
        }
      }
      // a row at a time, its columns over the lanes
      uint32_t any = again[0];
      if constexpr (COLS > 32) any |= again[1];
      for (unsigned rows = __ballot_sync(0xffffffffu, any != 0); rows != 0; rows &= rows - 1) {
        const int src = __ffs(rows) - 1;
        const size_t there = (size_t)(row - lane + src);
#pragma unroll
        for (int h = 0; h < (COLS + 31) / 32; ++h) {
          const uint32_t columns = __shfl_sync(0xffffffffu, again[h], src);
          if (columns >> lane & 1) {
            const int n = n0 + 32 * h + lane;
            float v = sum_of_fmas(p.a + there * p.lda, p.w + (size_t)n * p.K, p.K);
            if (p.bias != nullptr) v += p.bias[n];
            v = act_call(make_float4(v, 0.f, 0.f, 0.f), p.act).x;
            float* at = p.out + there * p.ldo + n;
            *at = p.residual ? *at + v : v;
          }
        }
      }
      __syncwarp();
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
}

static int sm_count() {
  static int n_sms = 0;
  if (n_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (n_sms <= 0) n_sms = 1;
  }
  return n_sms;
}

template <int BN>
static int launch(const Args& p, cudaStream_t stream) {
  CUtensorMap ma, mw;
  int rc = tc::tensor_map(p.a, p.M, p.K, p.lda, BM, &ma, BK, 4);
  if (rc == 0) rc = tc::tensor_map(p.w, p.N, p.K, p.K, BN, &mw, BK, 4);
  if (rc != 0) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    note_launch(cudaFuncSetAttribute(gemm_f32_tc_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes(BN)));
    attr_set = true;
  }
  const int n_sms = sm_count();
  const long units = (long)((p.M + BM - 1) / BM) * ((p.N + BN - 1) / BN);
  launch_pdl_split(false, gemm_f32_tc_kernel<BN>, dim3((unsigned)(units < n_sms ? units : n_sms)), dim3(THREADS), smem_bytes(BN), stream, ma,
                   mw, p);
  return take_launch_error();
}

bool takes(const void* a, long lda, const void* w, int K, const int* status) {
  return K > 0 && K % 4 == 0 && lda >= K && lda % 4 == 0 && (uintptr_t)a % 16 == 0 && (uintptr_t)w % 16 == 0 && status != nullptr &&
         tc::encode_fn() != nullptr;
}

// A tile: a fixed time (launch, first copies, the epilogue) and one a K block; a round of tiles more costs its epilogue too.
struct WidthTime {
  int bn;
  double fixed, kb, round;
};
constexpr WidthTime WIDTHS[] = {{32, 4.6, 0.75, 1.3}, {64, 6.3, 0.82, 3.8}, {128, 10.3, 1.04, 9.0}};

int width_for(int M, int N, int K) {
  const long down = ((long)M + BM - 1) / BM;
  const int kbs = (K + BK - 1) / BK, sms = sm_count();
  double best = 1e30;
  int width = 128;
  for (const WidthTime& w : WIDTHS) {
    const long tiles = down * ((N + w.bn - 1) / w.bn), rounds = (tiles + sms - 1) / sms;
    const double us = w.fixed + rounds * kbs * w.kb + (rounds - 1) * w.round;
    if (us < best && tiles <= 0x7fffffff) {
      best = us;
      width = w.bn;
    }
  }
  return width;
}

int run(const float* a, long lda, const float* w, const float* bias, float* out, long ldo, int M, int N, int K, int act, int residual,
        int width, int* status, cudaStream_t stream) {
  const Args p{a, lda, w, bias, out, ldo, M, N, K, act, residual, status};
  return width == 32 ? launch<32>(p, stream) : width == 64 ? launch<64>(p, stream) : launch<128>(p, stream);
}

}  // namespace f32tc
}  // namespace rl

// float32 A [M, K] (row stride lda) and W [N, K], out float32; residual != 0: out += result.  tile_width: 0 = chosen here, else
// the columns of a tile (32, 64 or 128; for tests and measurements).  Operands on 16-byte boundaries, K and lda multiples of 4.
RL_EXPORT int rl_gemm_f32_tc(const float* A, long lda, const float* W, const float* bias, float* out, long ldo, int M, int N, int K,
                             int act, int residual, int tile_width, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (!rl::f32tc::takes(A, lda, W, K, status)) return -2;
  const int width = tile_width == 0 ? rl::f32tc::width_for(M, N, K) : tile_width;
  if (width != 32 && width != 64 && width != 128) return -2;
  return rl::f32tc::run(A, lda, W, bias, out, ldo, M, N, K, act, residual, width, status, stream);
}
