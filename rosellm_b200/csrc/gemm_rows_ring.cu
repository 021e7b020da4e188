// bfloat16 products of at most 16 rows (a decode step of few requests):
//   out[M,N] = A[M,K] * W[N,K]^T (+ bias) (GELU) (or out += ..., the float32 residual stream), the
// input given as rows or as the LayerNorm of float32 rows (rosellm/rosetrainer/model.py:95, 220, 334-337).
//
// Such a product is its weight stream and, in a step, the wait for the kernel ahead.  One block an
// SM owns some groups of eight output columns (and, for an `out += ...`, perhaps a part of K).  The
// weight rows of a group, up to 1024 elements of each at a time, are brought by TMA (one box of eight rows
// a piece: cp.async.bulk.tensor; a bulk copy a row measured 19.7 us where this takes 13) into a ring of stages in shared memory,
// and the first of them before the block waits for the kernels ahead, since no kernel writes weights.  A block's shared
// memory is kept below half of an SM's, and where a warp holds one piece of eight rows its registers too, so
// that the next product's block stands beside this one and its weights arrive while this one computes: in a chain of
// products the memory is busy through the kernel boundaries.  Short rows of W stay with gemm_rows_mma.cu (short_rows).
// Eight warps share K (blocks of 64 elements in turn), so that a warp's part of the rows of A, as mma.sync
// fragments, stays in its registers for all of the block's columns: the rows are read (and normalised,
// through shared memory) once a block.  A ninth warp keeps the ring full.  The loop over the pieces is kept to some tens of
// instructions a warp: with two warps a scheduler, a piece of 13 KB lasts as long as its instructions take to
// issue (with 250 of them, 320 ns; the memory brings it in 290).  Weight pieces of 16 bytes a lane
// feed two m16n8k16 steps (A and W permuted alike along K); a block of 64 elements lies in shared memory as eight
// rows of 128 bytes, swizzled as TMA does it, and lane j of a row takes its 16-byte pieces 2j and 2j + 1, so
// that the two rows of an access phase hit different banks.  After at most four groups of columns the
// warps' partial sums meet in shared memory, added in a fixed order.
//
// Measured on B200, us (the register-fed kernel of gemm_rows_mma.cu before, now): 8 rows: 6400 x 1600 9.5, 6.9; +=
// 1600 x 1600 5.4, 2.5; += 1600 x 6400 11.4, 6.1; 3072 x 1024 with the LayerNorm 6.8, 3.9; 16384 x 2048 23.6, 12.9
// (5.2 TB/s of weights); 2048 x 8192 11.1, 7.8; 4800 x 1600 5.9, 5.5.  16 rows: += 1600 x 6400 14.0, 6.6.  A layer of a decode
// step as a chain, 512 cached tokens, width 1600: 39.4 -> 28.0 at batch 1, 48.9 -> 35.6 at 8, 55.5 -> 38.4 at 16.
#include "gemm_rows_ring.cuh"
#include "sampling_key.cuh"
#include "tc_common.cuh"

namespace rl {
namespace ring {

constexpr int WARPS = 8;
constexpr int THREADS = 32 * (WARPS + 1);    // and a warp that copies
constexpr int SLOTS = 2;                     // blocks of 64 elements of K a warp takes of a piece, at most
constexpr int MAX_PIECE = SLOTS * WARPS;     // blocks of 64 elements of K in a piece of the weight stream, at most
constexpr int ROUND = 4;                     // groups of eight columns between two meetings of the warps
constexpr int MAX_STAGES = 15;
constexpr int SMEM_TARGET = 112 * 1024;      // a block's shared memory at most: two blocks fit an SM

// How a product is cut (all in blocks of 64 elements where K is meant).
struct Cut {
  int blocks_n;  // thread blocks that share the groups of columns
  int parts;     // parts of K, one a thread block
  int kpart;     // of a part
  int piece;     // of a piece of the weight stream: eight columns of that many
  int stages;    // pieces that the ring holds
  int fixed;     // bytes of shared memory before the ring
};

__host__ __device__ inline int piece_bytes(int piece) { return piece * 8 * 128; }
// Bytes between two normalised rows in shared memory: 16 beyond a multiple of 128, so that the eight lanes of a
// 16-byte access phase (two rows, four pieces each, 32 bytes apart) hit different banks.
__host__ __device__ inline int row_pitch(int K) { return 2 * K + 16; }
// Shared memory: barriers (512) | partial sums [2][ROUND][8 warps][H][8 rows][8 columns] f32, and in their place
// before the first of them gamma and beta [K] f32 and the normalised rows [M] (NORM) | the ring
__host__ __device__ inline int fixed_bytes(int M, bool norm, int K) {
  const int part = 2 * ROUND * WARPS * (M <= 8 ? 1 : 2) * 64 * 4, rows = norm ? 8 * K + M * row_pitch(K) : 0;
  return (512 + (part > rows ? part : rows) + 1023) / 1024 * 1024;
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
__device__ __forceinline__ uint4 read_shared(uint32_t addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void consumers_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// HALVES: 1 for up to eight rows, 2 for up to sixteen.  PIECES: pieces of a group whose fragments of A a warp holds
// at once (a longer K takes them in turn).  Registers: within half an SM's where a warp holds one piece of eight rows; with
// more the 96 that this leaves a thread cost more than the neighbour gives (8 rows, 1600 x 6400: 7.9 us with them, 6.1 without).
// SAMPLE: the rows' next tokens are chosen from the sums (SampleArgs) and nothing else is written: the same sums in the same
// order as the form that writes them, so that a token is the one that the sampling kernel chooses from those logits.
template <int HALVES, int PIECES, bool NORM, bool SAMPLE>
__global__ __launch_bounds__(THREADS, HALVES * PIECES == 1 ? 2 : 1) void gemm_rows_ring_kernel(
    const __grid_constant__ CUtensorMap wmap, Args p, Cut cut) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, j = lane & 3;
  const int groups = (p.N + 7) / 8;
  const int first = (int)((long)blockIdx.x * groups / cut.blocks_n);
  const int last = (int)((long)(blockIdx.x + 1) * groups / cut.blocks_n);
  const int kb0 = (int)blockIdx.y * cut.kpart;
  const int kbs = min(cut.kpart, p.K / 64 - kb0);  // > 0: the host cuts no empty part
  const int held = PIECES * cut.piece;
  // shared memory's first 512 bytes: barriers of the stages (filled, read by all), of gamma and beta; the flag of a wait
  // that gave up
  const uint32_t full0 = tc::smem_u32(smem), empty0 = full0 + 8 * MAX_STAGES, bar_gb = full0 + 16 * MAX_STAGES;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + 16 * MAX_STAGES + 8);
  float* part_s = reinterpret_cast<float*>(smem + 512);
  const uint32_t ring0 = full0 + cut.fixed;
  const int stage_bytes = piece_bytes(cut.piece);

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (tid == 0) {
    for (int s = 0; s < cut.stages; ++s) {
      tc::mbar_init(full0 + 8 * s, 1);
      tc::mbar_init(empty0 + 8 * s, WARPS);
    }
    if (NORM) tc::mbar_init(bar_gb, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == WARPS) {
    // The weight stream, piece by piece in the order of their use: rounds of ROUND groups; in a round the parts of K
    // whose fragments are held together; in those the groups; in a group its pieces along K.
    if (lane != 0) return;
    if (NORM) {
      const uint32_t bytes = (uint32_t)p.K * 4;
      tc::mbar_expect_tx(bar_gb, p.norm.beta != nullptr ? 2 * bytes : bytes);
      bulk_copy(tc::smem_u32(part_s), p.norm.gamma, bytes, bar_gb);
      if (p.norm.beta != nullptr) bulk_copy(tc::smem_u32(part_s) + bytes, p.norm.beta, bytes, bar_gb);
    }
    int stage = 0, lap = 0;
    bool ok = true;
    for (int g0 = first; g0 < last && ok; g0 += ROUND)
      for (int kh = 0; kh < kbs && ok; kh += held)
        for (int gi = g0; gi < min(g0 + ROUND, last) && ok; ++gi)
          for (int kb = kh; kb < min(kh + held, kbs); kb += cut.piece) {
            if (lap > 0) {
              ok = tc::mbar_wait(empty0 + 8 * stage, (uint32_t)(lap - 1) & 1u, abort_flag, p.status);
              if (!ok) break;
              // the stage was read by ordinary loads, the copy writes through the async proxy
              asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            }
            tc::mbar_expect_tx(full0 + 8 * stage, (uint32_t)stage_bytes);
            tma_load_3d(ring0 + stage * stage_bytes, &wmap, full0 + 8 * stage, 0, 8 * gi, kb0 + kb);
            if (++stage == cut.stages) stage = 0, ++lap;
          }
    // what is still on its way arrives before the block ends, whatever became of the waits: every stage's last copy
    for (int s = 0; s < cut.stages; ++s) {
      const int laps = s < stage ? lap + 1 : lap;
      if (laps > 0) tc::mbar_wait_quiet(full0 + 8 * s, (uint32_t)(laps - 1) & 1u);
    }
    if (NORM) tc::mbar_wait_quiet(bar_gb, 0);
    return;
  }

  // The epilogue's thread: one pair of columns of one row of one group a round.
  const int e_lane = lane, e_half = HALVES == 2 ? (warp & 1) : 0, e_group = HALVES == 2 ? warp >> 1 : warp;
  const bool e_thread = e_group < ROUND;
  const int e_row = (e_lane >> 2) + 8 * e_half;
  // where the row's keys and values go (the step's description is written by none of its kernels)
  int kv_page = -1, kv_place = 0;
  if (p.kv.pool != nullptr && e_thread && e_row < p.M) {
    const int slot = p.kv.slots[p.kv.req_of_token[e_row]];
    const int pos = p.kv.positions[e_row];
    if (slot >= 0) {  // slot -1: padding of a fixed-size batch
      if (pos < 0 || pos >= p.kv.max_pos) {
        atomicOr(p.status, RL_STATUS_BAD_POSITION);
      } else {
        kv_page = p.kv.block_table[(size_t)slot * p.kv.bt_stride + pos / p.kv.page_size];
        kv_place = pos % p.kv.page_size;
        if (kv_page < 0) atomicOr(p.status, RL_STATUS_BAD_PAGE);
      }
    }
  }
  // Where a warp holds one piece of eight rows (and there is no norm or choice of tokens) the loop below is walked once before the wait
  // for the kernels ahead, over a kilobyte of the partial sums' place that nothing writes by
  // then (never the ring, which the copies fill) and to no effect: between other kernels its instructions would
  // have to be fetched once the rows are there.  A step of GPT-2 355M, one request, 481 -> 464 us with both numbers of pieces, a pass of
  // 8 requests of GPT-2 124M 19,313 -> 18,892, one of 1.5B 51,555 -> 51,213.  Two pieces gain less (one request of 1.5B 50,740) and lose where
  // a short kernel is ahead, and the lap comes too late (8 requests of the latent-attention model 14,635 -> 14,737); sixteen rows 5% slower in chains.
  constexpr bool DRY = !NORM && !SAMPLE && HALVES * PIECES == 1;
  constexpr int DRY_AT = WARPS * 64 * 4;  // beyond the sums that the lap itself stores; its reads end 1 KB behind, those of a second block WARPS KB on
  static_assert(!DRY || DRY_AT + (SLOTS - 1) * WARPS * 1024 + 1024 <= 2 * ROUND * WARPS * 64 * 4, "within the partial sums' place");
  if constexpr (!DRY) asm volatile("griddepcontrol.wait;" ::: "memory");

  // the row's sampling options, and its best entry so far
  float temp = 0.f;
  uint64_t seed = 0;
  uint32_t counter = 0;
  ArgMax best{-CUDART_INF_F, 0x7fffffff};
  if (SAMPLE && p.sample.temperature != nullptr && e_thread && e_row < p.M) {
    temp = p.sample.temperature[e_row];
    if (temp > 0.f) {
      seed = (uint64_t)p.sample.seeds[e_row];
      counter = (uint32_t)p.sample.counters[e_row];
    }
  }

  // A's fragments: of piece b, slot i, the block kh + b * piece + 8 i + warp of 64 elements, in two steps of 32: lane j
  // holds elements 16 j ... 16 j + 7 of it for the first step and the next eight for the second.
  uint4 af[PIECES][SLOTS][2][HALVES];
  bool ok = true;
  const int row_of[2] = {min(g, p.M - 1), min(g + 8, p.M - 1)};  // rows beyond M repeat the last: not stored
  auto load_rows = [&](const uint8_t* rows, size_t pitch, int kh) {
#pragma unroll
    for (int b = 0; b < PIECES; ++b)
#pragma unroll
      for (int i = 0; i < SLOTS; ++i) {
        const int in = WARPS * i + warp, kb = kh + b * cut.piece + in;
        const bool there = in < cut.piece && kb < kbs;  // of a block that is not there: the first, not used
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          const uint4* src = reinterpret_cast<const uint4*>(rows + row_of[h] * pitch + (kb0 + (there ? kb : 0)) * 128 + 32 * j);
          af[b][i][0][h] = src[0];
          af[b][i][1][h] = src[1];
        }
      }
  };
  const uint8_t* rows = reinterpret_cast<const uint8_t*>(p.a);
  size_t pitch = (size_t)p.lda * 2;
  if constexpr (NORM) {
    // A row a warp: pieces of four elements a lane, in registers between the two passes of the statistics.
    constexpr int Q = 8 * PIECES;  // 32 lanes x 4 elements x Q >= K
    const int n4 = p.K >> 2;
    rows = reinterpret_cast<const uint8_t*>(part_s + 2 * p.K);
    pitch = row_pitch(p.K);
    const float4* gamma = reinterpret_cast<const float4*>(part_s);
    const float4* beta = reinterpret_cast<const float4*>(part_s + p.K);
    for (int row = warp; row < p.M; row += WARPS) {
      const float4* xr = reinterpret_cast<const float4*>(p.norm.x + (size_t)row * p.norm.ldx);
      float4 r[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) r[q] = xr[lane + 32 * q < n4 ? lane + 32 * q : 0];
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        if (lane + 32 * q >= n4) r[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        sum[q & 3] += (r[q].x + r[q].y) + (r[q].z + r[q].w);
      }
      const float mean = warp_sum((sum[0] + sum[1]) + (sum[2] + sum[3])) / (float)p.K;
      float sq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (lane + 32 * q < n4) {
          const float a = r[q].x - mean, b = r[q].y - mean, cc = r[q].z - mean, dd = r[q].w - mean;
          sq[q & 3] += (a * a + b * b) + (cc * cc + dd * dd);
        }
      const float rstd = 1.0f / sqrtf(warp_sum((sq[0] + sq[1]) + (sq[2] + sq[3])) / (float)p.K + p.norm.eps);
      if (row == warp) ok = tc::mbar_wait(bar_gb, 0, abort_flag, p.status);
      uint8_t* dst = reinterpret_cast<uint8_t*>(part_s + 2 * p.K) + (size_t)row * pitch;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int e = lane + 32 * q;
        if (e < n4) {
          const float4 gm = gamma[e], bt = p.norm.beta != nullptr ? beta[e] : make_float4(0.f, 0.f, 0.f, 0.f);
          *reinterpret_cast<uint2*>(dst + 8 * e) =
              make_uint2(pack((r[q].x - mean) * rstd * gm.x + bt.x, (r[q].y - mean) * rstd * gm.y + bt.y),
                         pack((r[q].z - mean) * rstd * gm.z + bt.z, (r[q].w - mean) * rstd * gm.w + bt.w));
        }
      }
    }
    consumers_sync();
    load_rows(rows, pitch, 0);
    consumers_sync();  // the partial sums take the rows' place
  } else if constexpr (DRY) {
#pragma unroll
    for (int b = 0; b < PIECES; ++b)
#pragma unroll
      for (int i = 0; i < SLOTS; ++i)
#pragma unroll
        for (int h = 0; h < HALVES; ++h) af[b][i][0][h] = af[b][i][1][h] = make_uint4(0u, 0u, 0u, 0u);
  } else {
    load_rows(rows, pitch, 0);
  }

  // The lane's two 16-byte pieces of a block: 2 j and 2 j + 1 of the row's 128 bytes, swizzled by the row.
  const uint32_t w_at = ring0 + warp * 1024 + g * 128 + ((2 * j ^ g) << 4);
  int stage = 0, buf = 0;
  uint32_t parity = 0, w_stage = DRY ? tc::smem_u32(part_s) + DRY_AT + g * 128 + ((2 * j ^ g) << 4) : w_at;
#pragma unroll 1
  for (int g0 = DRY ? first - ROUND : first; g0 < last; g0 += ROUND, buf ^= 1) {
    const bool dry = DRY && g0 < first;
    if (DRY && g0 == first) {
      asm volatile("griddepcontrol.wait;" ::: "memory");
      load_rows(rows, pitch, 0);
      w_stage = w_at;
    }
    const int n_here = dry ? 1 : min(ROUND, last - g0);
    float* mine = part_s + buf * (ROUND * WARPS * HALVES * 64);
    const int n = 8 * (g0 + e_group) + 2 * j;
    const bool e_here = !dry && e_thread && e_group < n_here && e_row < p.M && n < p.N;
    float2 bias = make_float2(0.f, 0.f);
    if (e_here && p.bias != nullptr && blockIdx.y == 0) bias = *reinterpret_cast<const float2*>(p.bias + n);
    for (int kh = 0; kh < (dry ? 1 : kbs); kh += held) {
      if (!NORM && kbs > held && (kh > 0 || g0 > first)) load_rows(rows, pitch, kh);
      bool has[PIECES][SLOTS];  // the warp's blocks that are there
#pragma unroll
      for (int b = 0; b < PIECES; ++b)
#pragma unroll
        for (int i = 0; i < SLOTS; ++i) has[b][i] = WARPS * i + warp < min(cut.piece, kbs - kh - b * cut.piece);
      float2* slot = reinterpret_cast<float2*>(mine + warp * HALVES * 64) + lane;
#pragma unroll 1
      for (int gi = 0; gi < n_here; ++gi, slot += WARPS * HALVES * 32) {
        float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};  // two chains of products
#pragma unroll
        for (int b = 0; b < PIECES; ++b) {
          if (b > 0 && kh + b * cut.piece >= kbs) break;
          if (ok && !dry) ok = tc::mbar_wait(full0 + 8 * stage, parity, abort_flag, p.status);
          uint4 w[SLOTS][2];
#pragma unroll
          for (int i = 0; i < SLOTS; ++i)
            if (has[b][i]) {
              w[i][0] = read_shared(w_stage + i * WARPS * 1024);
              w[i][1] = read_shared((w_stage ^ 16u) + i * WARPS * 1024);
            }
#pragma unroll
          for (int i = 0; i < SLOTS; ++i)
            if (has[b][i])
#pragma unroll
              for (int s = 0; s < 2; ++s) {
                const uint4 lo = af[b][i][s][0];
                const uint4 hi = HALVES == 2 ? af[b][i][s][HALVES - 1] : make_uint4(0u, 0u, 0u, 0u);
                mma_bf16_16816(c, lo.x, hi.x, lo.y, hi.y, w[i][s].x, w[i][s].y);
                mma_bf16_16816(d, lo.z, hi.z, lo.w, hi.w, w[i][s].z, w[i][s].w);
              }
          __syncwarp();
          if (dry) continue;
          if (lane == 0) arrive(empty0 + 8 * stage);
          w_stage += stage_bytes;
          if (++stage == cut.stages) stage = 0, parity ^= 1u, w_stage = w_at;
        }
        // accumulators: c0, c1 = row g, columns 2j, 2j + 1; c2, c3 = row g + 8
#pragma unroll
        for (int h = 0; h < HALVES; ++h) {
          float2 t = make_float2(c[2 * h] + d[2 * h], c[2 * h + 1] + d[2 * h + 1]);
          if (kh > 0) {
            t.x += slot[32 * h].x;
            t.y += slot[32 * h].y;
          }
          slot[32 * h] = t;
        }
      }
    }
    // the warps' parts of K meet; the other buffer takes the next round's, so one barrier a round is enough
    consumers_sync();
    if (!(dry ? e_thread && e_group == 0 : e_here) || *abort_flag) continue;
    float2 sum = make_float2(0.f, 0.f);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) {
      const float2 v = *reinterpret_cast<const float2*>(mine + ((e_group * WARPS + w) * HALVES + e_half) * 64 + 2 * e_lane);
      sum.x += v.x; sum.y += v.y;
    }
    const float v0 = apply_act(sum.x + bias.x, p.act), v1 = apply_act(sum.y + bias.y, p.act);
    if (dry) {
      asm volatile("" ::"f"(v0), "f"(v1));
      continue;
    }
    if constexpr (SAMPLE) {
      float s0 = v0, s1 = v1;
      if (temp > 0.f) {
        const float inv_t = 1.0f / temp;
        s0 = sample_key(soft_capped(v0, p.sample.soft_cap), inv_t, seed, counter, (uint32_t)n);
        s1 = sample_key(soft_capped(v1, p.sample.soft_cap), inv_t, seed, counter, (uint32_t)(n + 1));
      }
      best = better(better(best, ArgMax{s0, n}), ArgMax{s1, n + 1});
      continue;
    }
    if (p.kv.pool != nullptr && n >= p.kv.q_width) {
      if (kv_page < 0) continue;
      const int cidx = n - p.kv.q_width;
      const int which = cidx / p.kv.kv_width;
      const int rem = cidx - which * p.kv.kv_width;
      const int head = rem / p.kv.head_dim, dd = rem - head * p.kv.head_dim;
      __nv_bfloat16* dst = (__nv_bfloat16*)p.kv.pool +
                           ((((size_t)kv_page * 2 + which) * p.kv.n_kv_heads + head) * p.kv.page_size + kv_place) * p.kv.head_dim + dd;
      *reinterpret_cast<__nv_bfloat162*>(dst) = __floats2bfloat162_rn(v0, v1);
    } else if (p.out_f32) {
      float* dst = (float*)p.out + (size_t)e_row * p.ldo + n;
      if (p.residual)  // one addition an element, or one a part of K (in no fixed order)
        asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(dst), "f"(v0), "f"(v1) : "memory");
      else if (((uintptr_t)dst & 7) == 0)
        *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
      else  // rows an odd number of elements apart
        dst[0] = v0, dst[1] = v1;
    } else {
      *reinterpret_cast<__nv_bfloat162*>((__nv_bfloat16*)p.out + (size_t)e_row * p.ldo + n) = __floats2bfloat162_rn(v0, v1);
    }
  }
  if constexpr (SAMPLE) {
    // the four lanes of a row agree, a warp's best per row is offered once; then one ticket a block
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      const ArgMax b{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
      best = better(best, b);
    }
    if (j == 0 && best.i != 0x7fffffff) {  // (only rows that are there have one)
      const unsigned long long word = ((unsigned long long)ordered_bits(best.v) << 32) | (unsigned long long)(~(uint32_t)best.i);
      if (word > __ldcg(p.sample.best + e_row)) {
        atomicMax(p.sample.best + e_row, word);
        __threadfence();
      }
    }
    consumers_sync();
    if (warp == 0) {
      int last_block = 0;
      if (lane == 0) last_block = atomicAdd(p.sample.ticket, 1) == (int)gridDim.x - 1;  // (K is not cut here)
      last_block = __shfl_sync(0xffffffffu, last_block, 0);
      if (last_block) sample_finish(p.sample, p.M, lane);
    }
  }
}

static int n_sms() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
  }
  return n;
}

// How a product is cut.  An `out += ...` (its parts meet by additions in memory) may cut K: the number
// of parts is the one whose busiest block has the fewest weights to read; a part more costs its
// additions, about what 2 KB of weights cost.
static Cut cut_for(const Args& p) {
  const int groups = (p.N + 7) / 8, kbs = p.K / 64;
  const bool may_cut = p.residual && p.norm.x == nullptr;
  Cut best{0, 0, 0, 0, 0, 0};
  long best_cost = 0;
  for (int parts = 1; parts <= (may_cut ? 8 : 1); ++parts) {
    const int kpart = (kbs + parts - 1) / parts;
    if (parts > 1 && (kpart < 4 || kpart * (parts - 1) >= kbs)) continue;
    const int blocks_n = min(groups, max(1, n_sms() / parts));
    const long per_block = (groups + blocks_n - 1) / blocks_n;
    const long cost = per_block * kpart * 1024 + 2048 * parts;
    if (best.parts == 0 || cost < best_cost) {
      best = Cut{blocks_n, parts, kpart, 0, 0, 0};
      best_cost = cost;
    }
  }
  const int per_group = (best.kpart + MAX_PIECE - 1) / MAX_PIECE;
  best.piece = (best.kpart + per_group - 1) / per_group;
  best.fixed = fixed_bytes(p.M, p.norm.x != nullptr, p.K);
  const int pieces = (groups + best.blocks_n - 1) / best.blocks_n * per_group;
  best.stages = min(min((SMEM_TARGET - best.fixed - 1024) / piece_bytes(best.piece), MAX_STAGES), max(pieces, 1));
  return best;
}

// Whether the rows of W are so short that the register-fed kernel of gemm_rows_mma.cu is ahead: a piece costs about
// 0.33 us (0.36 beyond eight rows) however short it is, which several groups of columns a block then pay one after the other,
// and some tenths of a microsecond more than the other kernel before the first.  Measured up to 512 elements (us, register-fed
// / here): 64 x 18944 at 8 rows 2.95 / 6.16, 64 x 2368 1.57 / 1.93; 256 x 9472 2.89 / 3.72 and 512 x 18944 6.15 / 6.40, but 256 x 7104 3.79 /
// 3.28 and 512 x 7104 3.96 / 3.32 (six groups a block); 16 rows 256 x 1184 1.90 / 2.14, 512 x 9472 at 9 rows 4.31 / 4.56.  Added into
// the stream only the shortest: 256 x 256 at 16 rows 2.3 / 1.9.  A LayerNorm of one or two rows costs the other
// kernel's warps little as well: 256 x 9472 3.89 / 4.58 at one, 128 x 4736 2.91 / 3.30 at two, 3.97 / 3.36 at four.  From 576
// elements on this kernel is ahead or level everywhere (576 x 37888 at 8 rows 12.86 / 11.81).
static bool short_rows(int M, int N, int K, bool residual, bool norm) {
  if (K > 512) return false;
  if (norm) return K <= 256 && (M == 1 || (M == 2 && K >= 128));
  return K < (residual ? 128 : 256) || (M > 8 && !residual) || (N + 7) / 8 > 6 * n_sms();
}

bool takes(const Args& p) {
  if (p.M < 1 || p.M > 16 || p.K % 64 != 0 || p.K < 64 || p.N % 2 != 0 || p.status == nullptr) return false;
  // pairs of outputs are stored together; float32 ones that are not added to, logits among them, singly where need be (whether
  // a head's tokens are asked for or its logits may not decide which kernel takes it)
  if ((p.residual || !p.out_f32) && (p.ldo % 2 != 0 || (uintptr_t)p.out % (p.out_f32 ? 8 : 4) != 0)) return false;
  if ((uintptr_t)p.w % 16 != 0 || (p.bias != nullptr && (uintptr_t)p.bias % 8 != 0))
    return false;
  if (p.norm.x == nullptr && (p.lda % 8 != 0 || (uintptr_t)p.a % 16 != 0)) return false;
  if (p.norm.x != nullptr && (p.K > MAX_PIECE * 64 || p.norm.ldx % 4 != 0 || (uintptr_t)p.norm.x % 16 != 0 ||
                              (uintptr_t)p.norm.gamma % 16 != 0 || (p.norm.beta != nullptr && (uintptr_t)p.norm.beta % 16 != 0)))
    return false;
  if (p.residual && (!p.out_f32 || p.act != RL_ACT_NONE || p.kv.pool != nullptr)) return false;
  if (p.kv.pool != nullptr && (p.out_f32 || p.act != RL_ACT_NONE || p.kv.head_dim % 8 != 0 || p.kv.q_width % 8 != 0 ||
                               p.kv.kv_width % 8 != 0))
    return false;
  if (short_rows(p.M, p.N, p.K, p.residual != 0, p.norm.x != nullptr)) return false;
  return tc::encode_fn() != nullptr;
}

// The weights as [K / 64][N][64]: a box is eight rows of `piece` blocks of 64 elements, a block's rows 128 bytes
// apart and swizzled; rows beyond N and blocks beyond K read as zeros.  Remembered by what they describe, as the other
// kernels' maps are (tc::tensor_map): a step of GPT-2 1.5B asks for 192.
static int weight_map(const Args& p, int piece, CUtensorMap* out) {
  static std::unordered_map<tc::MapKey, CUtensorMap, tc::MapKeyHash> cache;
  static std::mutex lock;
  const tc::MapKey key{p.w, p.N, p.K, p.K, 8, piece, 2};
  std::lock_guard<std::mutex> hold(lock);
  const auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  const cuuint64_t dim[3] = {64, (cuuint64_t)p.N, (cuuint64_t)(p.K / 64)};
  const cuuint64_t stride[2] = {(cuuint64_t)p.K * 2, 128};
  const cuuint32_t box[3] = {64, 8, (cuuint32_t)piece}, unit[3] = {1, 1, 1};
  const CUresult rc = tc::encode_fn()(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(p.w), dim, stride, box,
                                      unit, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) return -11;
  if (cache.size() > 8192) cache.clear();
  try {
    cache.emplace(key, *out);
  } catch (...) {  // no memory to remember it by: the caller is a C entry
  }
  return 0;
}

template <int HALVES, int PIECES, bool NORM, bool SAMPLE>
static void launch_form(const CUtensorMap& wmap, const Args& p, const Cut& cut, cudaStream_t stream) {
  constexpr auto kernel = gemm_rows_ring_kernel<HALVES, PIECES, NORM, SAMPLE>;
  static bool attr_set = false;
  if (!attr_set) {
    note_launch(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TARGET));
    note_launch(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    attr_set = true;
  }
  launch_pdl_split(false, kernel, dim3(cut.blocks_n, cut.parts), dim3(THREADS),
                   (size_t)cut.fixed + (size_t)cut.stages * piece_bytes(cut.piece), stream, wmap, p, cut);
}

template <int HALVES, int PIECES, bool NORM>
static void launch(const CUtensorMap& wmap, const Args& p, const Cut& cut, cudaStream_t stream) {
  if (p.sample.out_ids != nullptr) launch_form<HALVES, PIECES, NORM, true>(wmap, p, cut, stream);
  else launch_form<HALVES, PIECES, NORM, false>(wmap, p, cut, stream);
}

int run(const Args& p, cudaStream_t stream) {
  const Cut cut = cut_for(p);
  CUtensorMap wmap;
  const int rc = weight_map(p, cut.piece, &wmap);
  if (rc != 0) return rc;
  const bool norm = p.norm.x != nullptr, two = cut.kpart > MAX_PIECE;
  if (p.M <= 8) {
    if (norm) launch<1, 1, true>(wmap, p, cut, stream);
    else two ? launch<1, 2, false>(wmap, p, cut, stream) : launch<1, 1, false>(wmap, p, cut, stream);
  } else {
    if (norm) launch<2, 1, true>(wmap, p, cut, stream);
    else two ? launch<2, 2, false>(wmap, p, cut, stream) : launch<2, 1, false>(wmap, p, cut, stream);
  }
  return take_launch_error();
}

}  // namespace ring
}  // namespace rl

// Whether the sizes of a product of up to 16 rows are for this kernel (operands on the usual boundaries, even strides).
RL_EXPORT int rl_gemm_rows_ring_fits(int M, int N, int K, int residual, int norm) {
  return M >= 1 && M <= 16 && K % 64 == 0 && K >= 64 && N % 2 == 0 && !(norm && K > rl::ring::MAX_PIECE * 64) &&
         !rl::ring::short_rows(M, N, K, residual != 0, norm != 0);
}
