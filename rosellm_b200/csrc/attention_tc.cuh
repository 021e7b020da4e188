// Attention of prompt portions on tcgen05 (bfloat16, head size 64, no window): the same function
// as attn_mma_kernel (attention_mma.cuh; rosellm/rosetrainer/model.py:169-185 with the online
// softmax of rosellm/rosetrainer/paged_attention.py:80-109), with both products on the
// fifth-generation tensor cores and the scores in tensor memory.
//
// A block takes 128 consecutive queries of one request and head and walks the visible keys in
// tiles of 128, then (paired so that all blocks walk about as many tiles) 128 more queries of
// the same request and head.  Its warps have fixed roles:
//   warp 0     looks up the pages of each tile, a lane a page, and issues their TMA loads (a page
//              of one head is a contiguous [page size x 64] piece of the pool: one box a page)
//              for keys and values into a ring of three stages, and the load of the queries;
//   warp 1     allocates tensor memory (two score tiles of 128 columns, two P V tiles of 64); the
//              whole warp walks, one lane issues S = Q K^T (M=128, N=128, four steps of K=16) for the
//              next tile as soon as its keys have arrived, and P V (M=128, N=64, eight steps; V is
//              read as it lies in the cache, head dimension contiguous: the MN-major form of the B
//              operand) once the probabilities of the tile are in shared memory;
//   warps 2-17 softmax, two groups of eight warps on alternate key tiles, two threads a query row
//              (one for each half of a tile's keys and of the output's columns; tensor memory lets a
//              warp read only the lanes of its quarter): read the scores from tensor memory, mask by
//              position, agree on the row's maximum through shared memory, update the group's
//              maximum and sum in float32, write the probabilities as bfloat16 in the swizzled
//              K-major layout the second product reads, and, at the group's next tile, add
//              the P V (read back from tensor memory) to the row's output, which they keep in
//              registers and rescale there when the maximum rose.  At a turn's end the two
//              groups' outputs are added up through shared memory.
// What bounds it is the softmax's chain (a tile: scores ready, maximum 0.3 us, exponentials 1 us, product 0.4) and its
// arithmetic, not the tensor cores; hence the two chains side by side, 16 columns of scores on their way while the 16 before are
// worked on, and instructions that take two float32 values or three.
// Keys past the request's last visible key may hold anything (a partly filled page): their
// scores are masked by index, and their value rows are zeroed in shared memory before the
// second product, so that 0 * value stays 0.  Every wait on a barrier is bounded.
#pragma once
#include "attention_kernels.cuh"
#include "tc_common.cuh"

namespace rl {
namespace tc {

constexpr int ATT_Q = 128;       // queries per block
constexpr int ATT_KV = 128;      // keys per tile
constexpr int ATT_DH = 64;
constexpr int ATT_THREADS = 576;     // a TMA warp, an MMA warp, sixteen softmax warps
constexpr int ATT_SOFTMAX_THREADS = 512;
constexpr int ATT_Q_BYTES = ATT_Q * ATT_DH * 2;        // 16 KB
constexpr int ATT_KV_BYTES = ATT_KV * ATT_DH * 2;      // 16 KB: keys or values of a tile
constexpr int ATT_P_BYTES = ATT_Q * ATT_KV * 2;        // 32 KB: two K blocks of 64 keys
constexpr int ATT_PAIRED = 4;                          // pieces of 128 queries of a request that go in pairs where the grid leaves a choice
constexpr int ATT_STAGES = 3;                          // tiles of keys and values in shared memory
// The probabilities lie in two buffers: those of tile g are written while the P V of tile g - 1 may still read its own (only the
// P V of g - 2 has been waited for by then).  The block has its SM to itself either way.
constexpr int ATT_SMEM = 2 * ATT_Q_BYTES + ATT_STAGES * 2 * ATT_KV_BYTES + 2 * ATT_P_BYTES + 128 + 13 * ATT_Q * 4 + 1024;

// Instruction descriptor of kind::f16, bfloat16 x bfloat16 -> float32, M = 128; b_mn: the B
// operand has its N dimension contiguous in shared memory (values as they lie in the cache).
__host__ __device__ constexpr uint32_t att_instr_desc(int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(n >> 3) << 17) |
         ((uint32_t)(128 >> 4) << 24);
}

// Shared-memory descriptor of an MN-major tile with 128-byte swizzle: rows of 64 elements
// (one swizzle row) along N, groups of eight such rows (eight steps of K) 1024 bytes apart.
// With N = 64 there is one group across, so both strides name the step along K.
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(1024 >> 4) << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Waits of this kernel give up after about 50 ms (a tile takes microseconds) and leave in the
// status word's upper half which wait it was.
__device__ __forceinline__ bool att_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* status,
                                         int which) {
  const long long t0 = clock64();
  for (uint32_t it = 0;; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 0x3fu) == 0x3fu) {
      if (*abort_flag) return false;
      if (clock64() - t0 > 100000000LL) {
        *abort_flag = 1;
        atomicOr(status, RL_STATUS_WAIT_TIMEOUT | (1 << (16 + which)));
        return false;
      }
    }
  }
}

// Waits for tensor-memory loads, naming the registers that the last one fills: what is computed from them cannot move ahead.
__device__ __forceinline__ void att_loads_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]),
                 "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}
__device__ __forceinline__ float att_max3(float a, float b, float c) {
  float m;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
  return m;
}
// Two float32 values as one register pair, for the instructions that take two at a time.
__device__ __forceinline__ uint64_t att_pair(float lo, float hi) {
  return (uint64_t)__float_as_uint(lo) | ((uint64_t)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ uint64_t att_fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t att_add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float att_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float att_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

__device__ __forceinline__ float att_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The 128 queries of a block's turn: where they start in the request's portion, how many there
// are, the position of the first, one past the last key any of them sees, and the key tiles.
struct AttQueries {
  int t0, rows, first_pos, kv_hi, n_tiles;
};

// tiles: [n][2] = (request, first query of a 64-query tile within the request's portion).  The
// entries whose first query is a multiple of 128 name 128 consecutive queries; of a request's k
// such pieces, the block of piece i < k - 1 - i takes pieces k - 1 - i and i, one after the
// other (under the causal mask the first sees the most keys and the last the fewest: together
// every block walks about the same number of key tiles, and all blocks run in one round), the
// block of the middle piece takes it alone, and the others' blocks leave at once.
// singly (grid: heads, tiles): every piece has a block of its own, the pieces with the most keys of a request first, for
// grids whose pairs would need a second round of blocks (see launch_attn_tc); 2: those of requests of more than ATT_PAIRED pieces.
// map_q: the step's queries [tokens][heads * 64]; map_kv: this layer's pool as rows of 64
// [pages * 2 * kv heads * page size][64], a box being one page of one head.
__global__ __launch_bounds__(ATT_THREADS, 1) void attn_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                 const __grid_constant__ CUtensorMap map_kv,
                                                                 AttnParams p, const int* __restrict__ tiles, int singly) {
  extern __shared__ uint8_t att_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)att_smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t q_addr = smem_u32(smem);                            // [2 turns][128 queries]
  const uint32_t kv_addr = q_addr + 2 * ATT_Q_BYTES;                 // [stage][keys 16 KB, values 16 KB]
  const uint32_t p_addr = kv_addr + ATT_STAGES * 2 * ATT_KV_BYTES;   // [2 tiles][2 K blocks][128 rows][128 bytes]
  const uint32_t bar_base = p_addr + 2 * ATT_P_BYTES;
  const uint32_t q_full0 = bar_base, kv_full0 = bar_base + 16, kv_empty0 = bar_base + 40, s_full0 = bar_base + 64,
                 p_ready0 = bar_base + 80, pv_full0 = bar_base + 96;
  uint8_t* after_p = smem + 2 * ATT_Q_BYTES + ATT_STAGES * 2 * ATT_KV_BYTES + 2 * ATT_P_BYTES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(after_p + 112);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  // the warp's number as a value that the compiler knows to be the same in all lanes
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (!p.old_keys_settled) asm volatile("griddepcontrol.wait;" ::: "memory");  // the caller promises nothing of the table and the description
  const int tile = singly ? gridDim.y - 1 - blockIdx.y : gridDim.x - 1 - blockIdx.x;
  const int req = tiles[2 * tile], entry_t0 = tiles[2 * tile + 1];
  if (entry_t0 % ATT_Q != 0) return;  // the second half of a piece
  const int h = singly ? blockIdx.x : blockIdx.y;
  const int hkv = h / (p.n_heads / p.n_kv_heads);
  const int qs = p.q_start[req];
  const int q_len = p.q_start[req + 1] - qs;
  const int kv_len = p.kv_len[req];
  const int slot = p.slots[req];
  const int piece = entry_t0 / ATT_Q, n_pieces = (q_len + ATT_Q - 1) / ATT_Q;
  const bool alone = singly == 1 || (singly == 2 && n_pieces > ATT_PAIRED);
  if (!alone && piece > n_pieces - 1 - piece) return;  // taken by the block of its partner
  const int n_turns = !alone && piece < n_pieces - 1 - piece ? 2 : 1;
  auto queries_of = [&](int turn) {
    AttQueries q;
    q.t0 = (turn == 0 && !alone ? n_pieces - 1 - piece : piece) * ATT_Q;  // the longer walk first
    q.rows = min(ATT_Q, q_len - q.t0);
    q.first_pos = kv_len - q_len + q.t0;
    q.kv_hi = q.first_pos + q.rows;
    q.n_tiles = (q.kv_hi + ATT_KV - 1) / ATT_KV;
    return q;
  };
  RL_PHASE(0);

  if (threadIdx.x == 0) {
    mbar_init(q_full0, 1);
    mbar_init(q_full0 + 8, 1);
    for (int s = 0; s < ATT_STAGES; ++s) {
      mbar_init(kv_full0 + 8 * s, 1);
      mbar_init(kv_empty0 + 8 * s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full0 + 8 * s, 1);
      mbar_init(pv_full0 + 8 * s, 1);
      mbar_init(p_ready0 + 8 * s, ATT_SOFTMAX_THREADS / 64);  // one arrival a warp of the tile's group
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t tmem_pv = tmem_base + 256u;  // two tiles of 64 columns
  RL_PHASE(1);
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // the pages of the first tile (the block table is of earlier work, or has been waited for): looked up before the wait
  const int* bt = p.block_table + (size_t)slot * p.bt_stride;
  const int pages_per_tile = ATT_KV / p.page_size;
  auto pages_of_tile = [&](int kv_hi, int t) { return min(pages_per_tile, (kv_hi - t * ATT_KV + p.page_size - 1) / p.page_size); };
  auto entry_of_tile = [&](int kv_hi, int t) { return lane < pages_of_tile(kv_hi, t) ? bt[t * pages_per_tile + lane] : 0; };
  int next_page = 0;
  if (warp == 0) next_page = entry_of_tile(queries_of(0).kv_hi, 0);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  RL_PHASE(2);

  // Key tiles are counted through both turns (g): stages, score and P V buffers and the phases
  // of their barriers go by that count.
  if (warp == 0) {
    // The whole warp brings the tiles: lane i looks up page i of a tile and issues its two
    // copies (keys, values), so that a tile of sixteen pages costs one table read and one round of
    // issues, not sixteen of each in a row; the table entry of the next tile is asked for before
    // this tile's copies go out.
    if (lane == 0) {
      for (int turn = 0; turn < n_turns; ++turn) {
        mbar_expect_tx(q_full0 + 8 * turn, ATT_Q_BYTES);
        tma_load_2d(q_addr + turn * ATT_Q_BYTES, &map_q, q_full0 + 8 * turn, h * ATT_DH, qs + queries_of(turn).t0);
      }
    }
    const uint32_t page_bytes = (uint32_t)p.page_size * ATT_DH * 2;
    bool ok = true;
    int g = 0;
    for (int turn = 0; turn < n_turns && ok; ++turn) {
      const AttQueries q = queries_of(turn);
      for (int t = 0; t < q.n_tiles; ++t, ++g) {
        const int s = g % ATT_STAGES;
        const int n_pages = pages_of_tile(q.kv_hi, t);
        int page = next_page;
        if (t + 1 < q.n_tiles)
          next_page = entry_of_tile(q.kv_hi, t + 1);
        else if (turn + 1 < n_turns)
          next_page = entry_of_tile(queries_of(turn + 1).kv_hi, 0);
        ok = __all_sync(0xffffffffu, att_wait(kv_empty0 + 8 * s, ((g / ATT_STAGES) & 1u) ^ 1u, abort_flag, p.status, 0));
        if (!ok) break;
        if (lane == 0) mbar_expect_tx(kv_full0 + 8 * s, 2u * page_bytes * (uint32_t)n_pages);
        __syncwarp();
        if (lane < n_pages) {
          if (page < 0) {
            atomicOr(p.status, RL_STATUS_BAD_PAGE);
            page = 0;
          }
          const uint32_t k_dst = kv_addr + (uint32_t)s * 2u * ATT_KV_BYTES + (uint32_t)lane * page_bytes;
          const int row_k = ((page * 2) * p.n_kv_heads + hkv) * p.page_size;
          tma_load_2d(k_dst, &map_kv, kv_full0 + 8 * s, 0, row_k);
          tma_load_2d(k_dst + ATT_KV_BYTES, &map_kv, kv_full0 + 8 * s, 0, row_k + p.n_kv_heads * p.page_size);
        }
        if (g < 3) RL_PHASE(3 + g);
      }
    }
    if (lane == 0 && *abort_flag) {  // copies still in flight must land before the block leaves
      for (int turn = 0; turn < n_turns; ++turn) mbar_wait_quiet(q_full0 + 8 * turn, 0u);
      for (int k = max(0, g - ATT_STAGES); k < g; ++k) mbar_wait_quiet(kv_full0 + 8 * (k % ATT_STAGES), (k / ATT_STAGES) & 1u);
    }
  } else if (warp == 1) {
    // The whole warp walks, with values that are the same in all lanes (a product's operands are taken from uniform
    // registers); one lane issues.
    constexpr uint32_t idesc_s = att_instr_desc(ATT_KV, false);
    constexpr uint32_t idesc_o = att_instr_desc(ATT_DH, true);
    const int n_first = queries_of(0).n_tiles;
    const int n_all = n_first + (n_turns > 1 ? queries_of(1).n_tiles : 0);
    const uint64_t q_desc = smem_desc(q_addr), k_desc = smem_desc(kv_addr), p_desc = smem_desc(p_addr),
                   v_desc = smem_desc_mn(kv_addr + ATT_KV_BYTES);
    bool ok = true;
    auto wait = [&](uint32_t bar, uint32_t parity, int which) {
      return __all_sync(0xffffffffu, att_wait(bar, parity, abort_flag, p.status, which));
    };
    // S = Q K^T of tile g (of the turn it falls in), once its keys (and that turn's queries) have arrived
    auto issue_s = [&](int g) {
      const int turn = g < n_first ? 0 : 1;
      if (g == 0 || g == n_first) ok = wait(q_full0 + 8 * turn, 0u, 1);
      if (ok) ok = wait(kv_full0 + 8 * (g % ATT_STAGES), (g / ATT_STAGES) & 1u, 2);
      if (!ok) return;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // descriptors count 16-byte units; a K step of 32 bytes is +2
      const uint64_t kd = k_desc + (uint64_t)((g % ATT_STAGES) * (2 * ATT_KV_BYTES >> 4)), qd = q_desc + (uint64_t)(turn * (ATT_Q_BYTES >> 4));
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < ATT_DH / 16; ++k)
          mma_f16(tmem_base + (uint32_t)(g & 1) * 128u, qd + 2 * k, kd + 2 * k, idesc_s, k != 0 ? 1u : 0u);
        mma_commit(s_full0 + 8 * (g & 1));
      }
      __syncwarp();
    };
    if (n_all > 0) issue_s(0);
    RL_PHASE_OF(6, 32);
    for (int g = 0; g < n_all && ok; ++g) {
      // the scores of the next tile, while the softmax works on this one (its place was last
      // read for tile g - 1, whose probabilities have been waited for)
      if (g + 1 < n_all) {
        issue_s(g + 1);
        if (!ok) break;
      }
      ok = wait(p_ready0 + 8 * (g & 1), (g >> 1) & 1u, 3);
      if (!ok) break;
      if (g < 6) RL_PHASE_OF(10 + g, 32);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint64_t vd = v_desc + (uint64_t)((g % ATT_STAGES) * (2 * ATT_KV_BYTES >> 4)), pd = p_desc + (uint64_t)((g & 1) * (ATT_P_BYTES >> 4));
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < ATT_KV / 16; ++k)  // 16 keys a step: two groups of eight value rows
          mma_f16(tmem_pv + (uint32_t)(g & 1) * 64u, pd + (uint64_t)((k >> 2) * (ATT_Q * 128 >> 4) + (k & 3) * 2),
                  vd + (uint64_t)(k * (2048 >> 4)), idesc_o, k != 0 ? 1u : 0u);
        mma_commit(kv_empty0 + 8 * (g % ATT_STAGES));
        mma_commit(pv_full0 + 8 * (g & 1));
      }
      __syncwarp();
    }
  } else {
    // Two groups of eight warps take the key tiles in turn, each with a running maximum, sum and output of its own, so that
    // the chain of one tile (scores, maximum over the row, exponentials, probabilities to shared memory, their product) lies
    // under the other's; a turn's two results are added up at its end.  In a group two threads share a query row: warp w reads the
    // tensor-memory lanes of its quarter (w % 4); `half` says which 64 keys of a tile and which 32 columns of the output are
    // this thread's.  (With all sixteen warps on one tile the 2 x 1024 tokens of GPT-2 124M took 22.6 us a layer.)
    const int quarter = warp & 3, group = (warp - 2) >> 3, half = ((warp - 2) >> 2) & 1;
    const int row = quarter * 32 + lane;
    const int st = (threadIdx.x - 64) & (ATT_SOFTMAX_THREADS / 2 - 1);  // 0..255 in the group
    const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
    const float sl2 = p.scale * 1.4426950408889634f;  // scores in units of log 2
    float* mx_s = reinterpret_cast<float*>(after_p + 128);  // maxima [2 groups][2 tiles][2 halves][128]
    float* l_s = mx_s + 8 * ATT_Q;                           // at a turn's end: sums [2 groups][2 halves][128], then
    float* m_s = l_s + 4 * ATT_Q;                            // the second group's maxima [128]
    // this thread's 64 probabilities of a tile: the row's 128 bytes in K block `half` of the group's buffer
    uint8_t* p_row = smem + 2 * ATT_Q_BYTES + ATT_STAGES * 2 * ATT_KV_BYTES + (size_t)group * ATT_P_BYTES + (size_t)half * (ATT_Q * 128) +
                     (size_t)row * 128;
    // the second group's outputs at a turn's end, in the place of its probabilities: [16 pieces of four columns][128 rows] float4
    float4* o_s = reinterpret_cast<float4*>(smem + 2 * ATT_Q_BYTES + ATT_STAGES * 2 * ATT_KV_BYTES + ATT_P_BYTES);
    const int sw = row & 7;  // swizzle of 16-byte chunks
    auto group_sync = [&]() { asm volatile("bar.sync %0, 256;" ::"r"(1 + group) : "memory"); };
    auto all_sync = [&]() { asm volatile("bar.sync 3, 512;" ::: "memory"); };
    float o[ATT_DH / 2];
    // adds tile g's P V (this thread's 32 columns) to the row's output, after its product has finished
    auto take_pv = [&](int g) -> bool {
      const bool arrived = __all_sync(0xffffffffu, att_wait(pv_full0 + 8 * group, (g >> 1) & 1u, abort_flag, p.status, 5));
      if (!arrived) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < 32; c += 16) {
        uint32_t r[16];
        tmem_load16(tmem_pv + lane_base + (uint32_t)group * 64u + (uint32_t)half * 32u + (uint32_t)c, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int i = 0; i < 16; ++i) o[c + i] += __uint_as_float(r[i]);
      }
      return true;
    };
    // Every softmax thread passes its group's barrier once a tile of the group and the common one twice a turn, also
    // after a wait gave up (ok false): the work is skipped then, the barriers never.
    bool ok = true;
    int g0 = 0;  // tiles of the turns before
    for (int turn = 0; turn < n_turns; ++turn) {
      const AttQueries q = queries_of(turn);
      const bool row_ok = row < q.rows;
      const int qpos = q.first_pos + row;
      float m = -CUDART_INF_F, l = 0.f;  // l: the sum over this thread's keys
#pragma unroll
      for (int d = 0; d < ATT_DH / 2; ++d) o[d] = 0.f;
      int last = -1;  // the group's last tile of this turn
      for (int t = (group - g0) & 1; t < q.n_tiles; t += 2) {
        const int g = g0 + t;
        const int kt = t * ATT_KV + half * 64;  // first key of this thread's half of the tile
        if (ok) ok = __all_sync(0xffffffffu, att_wait(s_full0 + 8 * group, (g >> 1) & 1u, abort_flag, p.status, 4));
        if (g < 4) RL_PHASE_OF(16 + 4 * g, 64);
        const uint32_t s_addr = tmem_base + lane_base + (uint32_t)group * 128u + (uint32_t)half * 64u;
        // keys of this half the query sees: [0, n_vis); the whole warp sees all of them in every tile but the last ones
        const int n_vis = row_ok ? max(0, min(64, qpos - kt + 1)) : 0;
        const bool all_vis = __all_sync(0xffffffffu, n_vis == 64);
        float mx = -CUDART_INF_F;
        if (ok) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // sixteen columns at a time, the next on their way while these are looked at
          uint32_t r[2][16];
          tmem_load16(s_addr, r[0]);
          float m2[2] = {-CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            att_loads_wait(r[c & 1]);
            if (c < 3) tmem_load16(s_addr + (uint32_t)(c + 1) * 16u, r[(c + 1) & 1]);
            if (all_vis) {
#pragma unroll
              for (int i = 0; i < 16; i += 2)
                m2[(i >> 1) & 1] = att_max3(m2[(i >> 1) & 1], __uint_as_float(r[c & 1][i]), __uint_as_float(r[c & 1][i + 1]));
            } else {
#pragma unroll
              for (int i = 0; i < 16; ++i)
                if (c * 16 + i < n_vis) mx = fmaxf(mx, __uint_as_float(r[c & 1][i]));
            }
          }
          mx = fmaxf(mx, fmaxf(m2[0], m2[1]));
        }
        // the row's maximum over the two halves
        float* mx_t = mx_s + (group * 2 + ((g >> 1) & 1)) * 2 * ATT_Q + row;  // (written again two of the group's tiles on)
        mx_t[half * ATT_Q] = mx;
        group_sync();
        mx = fmaxf(mx_t[0], mx_t[ATT_Q]);
        if (g < 4) RL_PHASE_OF(17 + 4 * g, 64);
        const float m_new = fmaxf(m, mx * sl2);
        const float alpha = m_new == -CUDART_INF_F ? 1.f : att_ex2(m - m_new);
        const float neg_m = m_new == -CUDART_INF_F ? 0.f : -m_new;
        // the P V of the group's tile before: its probabilities lie where this tile's go
        if (ok && last >= 0) {
          ok = take_pv(last);
          if (ok && __any_sync(0xffffffffu, alpha != 1.f)) {
#pragma unroll
            for (int d = 0; d < ATT_DH / 2; ++d) o[d] *= alpha;
          }
        }
        last = g;
        if (!ok) continue;
        // probabilities of this thread's 64 keys, as bfloat16, into the operand of the second product (the scores are read again:
        // held from the first reading, they would not fit the registers beside the output)
        const uint64_t sl2_2 = att_pair(sl2, sl2), neg_m2 = att_pair(neg_m, neg_m);
        uint64_t sum2[2] = {0ull, 0ull};  // two chains of pairs of sums
        uint32_t r[2][16];
        tmem_load16(s_addr, r[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          att_loads_wait(r[c & 1]);
          if (c < 3) tmem_load16(s_addr + (uint32_t)(c + 1) * 16u, r[(c + 1) & 1]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {  // eight keys = a 16-byte chunk of the row
            uint32_t packed[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int k = 8 * e + 2 * i;
              const uint64_t x = att_fma2((uint64_t)r[c & 1][k] | ((uint64_t)r[c & 1][k + 1] << 32), sl2_2, neg_m2);
              float p0 = att_ex2(att_lo(x)), p1 = att_ex2(att_hi(x));
              if (!all_vis) {
                if (c * 16 + k >= n_vis) p0 = 0.f;
                if (c * 16 + k + 1 >= n_vis) p1 = 0.f;
              }
              sum2[i & 1] = att_add2(sum2[i & 1], att_pair(p0, p1));
              const __nv_bfloat162 hh = __floats2bfloat162_rn(p0, p1);
              packed[i] = *reinterpret_cast<const uint32_t*>(&hh);
            }
            *reinterpret_cast<uint4*>(p_row + (((c * 2 + e) ^ sw) << 4)) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
          }
        }
        const uint64_t both = att_add2(sum2[0], sum2[1]);
        const float sum = att_lo(both) + att_hi(both);
        l = l * alpha + sum;
        m = m_new;
        // value rows of keys no query of the turn sees: zero, so that 0 * value stays 0
        if (t * ATT_KV + ATT_KV > q.kv_hi) {
          // the values of this tile have arrived: the scores could not be there otherwise, and
          // keys and values come under one barrier
          uint8_t* v_s = smem + 2 * ATT_Q_BYTES + (size_t)(g % ATT_STAGES) * 2 * ATT_KV_BYTES + ATT_KV_BYTES;
          const int first_bad = q.kv_hi - t * ATT_KV;
          for (int i = st + first_bad * 8; i < ATT_KV * 8; i += ATT_SOFTMAX_THREADS / 2)
            *reinterpret_cast<uint4*>(v_s + (size_t)i * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_ready0 + 8 * group) : "memory");
        if (g < 4) RL_PHASE_OF(18 + 4 * g, 64);
      }
      g0 += q.n_tiles;
      if (ok && last >= 0) ok = take_pv(last);
      if (turn == 0) RL_PHASE_OF(7, 64);
      // the turn's end: the second group's outputs, maxima and sums to shared memory, the first group adds its own
      l_s[(group * 2 + half) * ATT_Q + row] = l;
      if (group == 1) {
#pragma unroll
        for (int i = 0; i < 8; ++i) o_s[(half * 8 + i) * ATT_Q + row] = make_float4(o[4 * i], o[4 * i + 1], o[4 * i + 2], o[4 * i + 3]);
        if (half == 0) m_s[row] = m;
      }
      all_sync();
      if (group == 0 && ok && row_ok) {
        const float m1 = m_s[row], top = fmaxf(m, m1);
        const float f0 = m == -CUDART_INF_F ? 0.f : att_ex2(m - top), f1 = m1 == -CUDART_INF_F ? 0.f : att_ex2(m1 - top);
        const float all = (l_s[row] + l_s[ATT_Q + row]) * f0 + (l_s[2 * ATT_Q + row] + l_s[3 * ATT_Q + row]) * f1;
        const float inv = all > 0.f ? 1.0f / all : 0.f;
        const float s0 = f0 * inv, s1 = f1 * inv;
        __nv_bfloat16* out = (__nv_bfloat16*)p.out + (size_t)(qs + q.t0 + row) * p.out_stride + h * ATT_DH + half * 32;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 u = o_s[(half * 8 + 2 * i) * ATT_Q + row], v = o_s[(half * 8 + 2 * i + 1) * ATT_Q + row];
          const __nv_bfloat162 a0 = __floats2bfloat162_rn(o[8 * i] * s0 + u.x * s1, o[8 * i + 1] * s0 + u.y * s1);
          const __nv_bfloat162 a1 = __floats2bfloat162_rn(o[8 * i + 2] * s0 + u.z * s1, o[8 * i + 3] * s0 + u.w * s1);
          const __nv_bfloat162 a2 = __floats2bfloat162_rn(o[8 * i + 4] * s0 + v.x * s1, o[8 * i + 5] * s0 + v.y * s1);
          const __nv_bfloat162 a3 = __floats2bfloat162_rn(o[8 * i + 6] * s0 + v.z * s1, o[8 * i + 7] * s0 + v.w * s1);
          *reinterpret_cast<uint4*>(out + i * 8) =
              make_uint4(*reinterpret_cast<const uint32_t*>(&a0), *reinterpret_cast<const uint32_t*>(&a1),
                         *reinterpret_cast<const uint32_t*>(&a2), *reinterpret_cast<const uint32_t*>(&a3));
        }
      }
      all_sync();  // the next turn's probabilities and maxima take their places
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  RL_PHASE(8);
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
  }
}

// Whether the tcgen05 kernel takes these sizes.
static inline bool attn_tc_fits(const AttnParams& p) {
  return p.head_dim == ATT_DH && p.window <= 0 && p.page_size >= 8 && p.page_size <= ATT_KV &&
         ATT_KV % p.page_size == 0 && (p.page_size & 7) == 0 && p.out_stride % 8 == 0 &&
         ((uintptr_t)p.out % 16) == 0;
}

// n_tokens: rows of the query matrix; n_pages: pages of this layer's pool.  Returns 0, or a
// negative code when a tensor map could not be made (the caller then takes the other kernel).
static inline int launch_attn_tc(const AttnParams& p, const int* tiles, int n_tiles, int n_tokens, long n_pages,
                                 cudaStream_t stream) {
  CUtensorMap mq, mkv;
  int rc = tensor_map(p.q, n_tokens, (long)p.n_heads * ATT_DH, p.q_stride, ATT_Q, &mq);
  if (rc != 0) return rc;
  rc = tensor_map(p.pool, n_pages * 2 * p.n_kv_heads * p.page_size, ATT_DH, ATT_DH, p.page_size, &mkv);
  if (rc != 0) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    cudaFuncSetAttribute(attn_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ATT_SMEM);
    attr_set = true;
  }
  // Pairs all walk about as many key tiles: a round of them is full to its end, and a last round of only a few blocks
  // costs as much as the first.  Where the rounds that the pairs (about a quarter of the 64-query tiles, for every head) take
  // would stand empty by a sixth or more, the pieces go singly, and an SM takes the next as soon as it is free (us, pairs / singly: 25
  // heads, 2 prompts of 1024, 200 pairs on 148 SMs 41.9 / 37.8, 4 of 512 29.8 / 27.9; 20 heads, 2048 tokens 64.0 / 44.8;
  // 40 heads, 2 of 1024 62.0 / 57.1).  Fuller rounds go in pairs: 32 heads, 256 pairs, 4 prompts of 512 32.3 / 34.0, 8 of 256 26.5 / 29.3.
  static int n_sms = 0;
  if (n_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (n_sms <= 0) n_sms = 1;
  }
  const long pairs = (long)(n_tiles + 3) / 4 * p.n_heads, places = (pairs + n_sms - 1) / n_sms * n_sms;
  // Pieces that all stand on the SMs at once go singly as well, and up to eight pieces to five SMs where a request has more than four: the
  // longest, started first, end before a pair of a long and a short piece does (us, pairs / singly: 12 heads, 2 prompts of 512 14.2 (the
  // form before) / 10.0, 2 of 1024 19.6 / 17.1, 2 of 896 18.2 / 14.4, 3 of 640 15.7 / 15.1, one of 2048 29.3 / 25.1); shorter
  // requests' pieces in a second round cost their blocks' start again: 4 of 512 14.8 / 16.7, 4 of 400 14.2 / 16.2.
  const bool round = pairs > n_sms && 5 * places > 6 * pairs;
  const int mode = n_tiles > 65535 ? 0 : (round || 2 * pairs <= n_sms) ? 1 : (2 * pairs * 5 <= 8 * n_sms) ? 2 : 0;  // (a grid's second extent)
  const bool singly = mode != 0;
  const dim3 grid = singly ? dim3(p.n_heads, n_tiles) : dim3(n_tiles, p.n_heads);
  launch_pdl_split(false, attn_tc_kernel, grid, ATT_THREADS, ATT_SMEM, stream, mq, mkv, p, tiles, mode);
  return 0;
}

}  // namespace tc
}  // namespace rl
