// bfloat16 products of 17 to 128 rows (a batch of decoded tokens, a short prompt portion) on
// tcgen05, with K split over the blocks of a thread-block cluster:
//
//   out[M,N] = A[M,K] * W[N,K]^T  (+ bias[N]) (GELU) (or out += ..., the float32 residual stream)
//
// the products of rosellm/rosetrainer/model.py:95, 220, 334-337 for the batch sizes between
// the weight-streaming kernel (gemm_rows_mma.cu, where every warp re-reads the rows of A) and
// the tiled kernel for prompts (gemm_tc.cu, whose 128-row tiles leave most SMs idle here).
//
// Such a product is a stream of weights with little arithmetic, so the work is laid out for
// the stream: the roles of the operands are swapped.  A block takes 128 rows of W (output
// columns) as the 128-lane operand of tcgen05.mma and the M rows of A, rounded up to a multiple
// of 16, as the N operand; a cluster of up to eight blocks shares one such tile, each block
// walking a part of K through a ring of TMA copies.  What bounds it is the copies in flight and the
// fixed parts (launch, first copy, the meeting of the parts), so:
//   - a ring takes at most 112 KB, for two blocks on an SM: a product's first copies run while
//     the one before it finishes (with all of a part's operands held at once, 200 KB, a block waits for a whole
//     SM: 4800 x 1600, 64 rows, 9.6 us against 8.0);
//   - the weights of the first stages are asked for before the wait for the kernels ahead;
//   - every block sends its float32 sums of a row straight from tensor memory into the shared memory of the
//     block that finishes that row, [sender][row][128 columns]; after one cluster barrier each adds what it was
//     sent in the order of the parts, applies bias / activation / residual and stores along rows, or scatters
//     key and value columns into cache pages.  Sums that stayed with their block and were read from there took
//     a second barrier and a round trip a part.
// Waits on mbarriers are bounded (status bit, abort flag); the cluster barriers are reached by every thread
// on every path.
#include "gemm_epilogue.cuh"
#include "tc_common.cuh"

namespace rl {
namespace tc {

constexpr int RWARPS = 10, RTHREADS = 32 * RWARPS;  // a warp that copies, one that issues, eight that read the accumulator
constexpr int RMAX_CLUSTER = 8;        // the portable limit
constexpr int RMAX_STAGES = 6;
constexpr int RMAX_K = 8192;           // beyond, eight blocks' rings are walked for longer than the other kernels take
constexpr int RW_BYTES = BM * BK * 2;  // a 128 x 64 tile of W

// How a product is cut: blocks of a cluster, K blocks of 64 a block, stages of its ring, rows of A a block finishes.
struct RowsCut {
  int nt, cluster, kb_per, stages, own, tmem_cols;
};

// Shared memory of a block: stages of (W 128 x 64, A NT x 64) bfloat16 | what the cluster's blocks send it, float32 [sender]
// [own][128] | the element offsets of its rows' cache pages [own] | barriers (full and empty of the stages, accumulator), the
// tensor-memory address and the abort flag.
__host__ __device__ inline int rows_stage_bytes(int nt) { return RW_BYTES + nt * BK * 2; }
__host__ __device__ inline int rows_fixed_bytes(int cluster, int own) {
  return cluster * own * BM * 4 + own * 8 + (2 * RMAX_STAGES + 1) * 8 + 16 + 1024;
}

// Grid (cluster size, tiles of 128 output columns); a cluster is one row of the grid.
template <typename TOut>
__global__ __launch_bounds__(RTHREADS) void gemm_tc_rows_kernel(
    const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
    const float* __restrict__ bias, TOut* __restrict__ out, long ldo, int M, int N, int K, const RowsCut cut, int act,
    int residual, KvScatter kv, int* __restrict__ status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t smem_base = smem_u32(smem);
  const int NT = cut.nt, own = cut.own;
  const int stage_bytes = rows_stage_bytes(NT);
  float* recv = reinterpret_cast<float*>(smem + cut.stages * stage_bytes);
  long long* row_base = reinterpret_cast<long long*>(recv + cut.cluster * own * BM);
  const uint32_t bar_base = smem_u32(row_base + own);
  auto full_bar = [&](int s) { return bar_base + 8u * s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (RMAX_STAGES + s); };
  const uint32_t acc_bar = bar_base + 8u * (2 * RMAX_STAGES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(reinterpret_cast<uint8_t*>(row_base + own) + (2 * RMAX_STAGES + 1) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int rank = (int)cluster_rank();
  const int n0 = blockIdx.y * BM;
  const int num_kb = (K + BK - 1) / BK;
  const int kb0 = rank * cut.kb_per;
  const int nkb = min(num_kb - kb0, cut.kb_per);  // > 0: no part of K is empty

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int s = 0; s < cut.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"((uint32_t)cut.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // the cluster's blocks have all begun when this one sends them its sums (waited for below, long after)
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

  bool ok = true;
  if (warp == 0) {
    // The whole warp walks, one lane issues.  Weights are written by no kernel of a step: those of the first stages are asked
    // for before the wait for the kernels ahead.
    const int ahead = min(nkb, cut.stages);
    for (int s = 0; s < ahead; ++s)
      if (elect_one()) {
        mbar_expect_tx(full_bar(s), (uint32_t)stage_bytes);
        tma_load_2d(smem_base + s * stage_bytes, &map_w, full_bar(s), (kb0 + s) * BK, n0);
      }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    int s = 0, done = 0;
    uint32_t ph = 0;
    for (; done < nkb; ++done) {
      if (done >= ahead) {
        ok = mbar_wait_warp(empty_bar(s), ph ^ 1u, abort_flag, status);
        if (!ok) break;
      }
      if (elect_one()) {
        const uint32_t dst = smem_base + s * stage_bytes;
        if (done >= ahead) {
          mbar_expect_tx(full_bar(s), (uint32_t)stage_bytes);
          tma_load_2d(dst, &map_w, full_bar(s), (kb0 + done) * BK, n0);
        }
        tma_load_2d(dst + RW_BYTES, &map_a, full_bar(s), (kb0 + done) * BK, 0);
      }
      __syncwarp();
      if (++s == cut.stages) s = 0, ph ^= 1u;
    }
    if (*abort_flag)  // copies still in flight land before the block ends
      for (int k = max(0, done - cut.stages); k < done; ++k) mbar_wait_quiet(full_bar(k % cut.stages), (uint32_t)(k / cut.stages) & 1u);
  } else if (warp == 1) {
    const uint32_t idesc = instr_desc(NT);
    const uint64_t desc0 = smem_desc(smem_base);
    int s = 0;
    uint32_t ph = 0;
    for (int kb = 0; kb < nkb; ++kb) {
      ok = mbar_wait_warp(full_bar(s), ph, abort_flag, status);
      if (!ok) break;
      const uint64_t w_desc = desc0 + (uint64_t)((uint32_t)(s * stage_bytes) >> 4), a_desc = w_desc + (RW_BYTES >> 4);
      if (elect_one()) {
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) mma_f16(tmem_base, w_desc + 2 * k, a_desc + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
        mma_commit(empty_bar(s));
      }
      __syncwarp();
      if (++s == cut.stages) s = 0, ph ^= 1u;
    }
    if (ok && elect_one()) mma_commit(acc_bar);
    __syncwarp();
  } else if (kv.pool != nullptr && n0 + BM > kv.q_width) {
    // where the keys and values of the block's rows go: the element offset of (page, keys, head 0, place in the page, 0), or
    // -1 for a row that is not written (the step's description is written by none of its kernels)
    for (int i = (int)threadIdx.x - 64; i < own; i += RTHREADS - 64) {
      const int m = rank * own + i;
      long long base = -1;
      if (m < M) {
        const int slot = kv.slots[kv.req_of_token[m]];
        const int pos = kv.positions[m];
        if (slot >= 0) {  // slot -1: padding of a fixed-size batch
          if (pos < 0 || pos >= kv.max_pos) {
            atomicOr(kv.status, RL_STATUS_BAD_POSITION);
          } else {
            const int page = kv.block_table[(size_t)slot * kv.bt_stride + pos / kv.page_size];
            if (page < 0)
              atomicOr(kv.status, RL_STATUS_BAD_PAGE);
            else
              base = ((long long)page * 2 * kv.n_kv_heads * kv.page_size + pos % kv.page_size) * kv.head_dim;
          }
        }
      }
      row_base[i] = base;
    }
  }
  __syncwarp();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");

  // The accumulator's lanes are output columns, its columns rows of A: every row goes to the block that finishes it, the
  // eight warps taking a quarter of the lanes and every second group of 16 rows each.
  if (warp >= 2) {
    ok = mbar_wait_warp(acc_bar, 0u, abort_flag, status);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
      const int quarter = warp & 3;
      const uint32_t mine = smem_u32(recv + rank * own * BM + quarter * 32 + lane);
      for (int c = (warp - 2) >> 2; c < NT / 16; c += 2) {
        uint32_t r[16];
        tmem_load16(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(c * 16), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        int owner = (c * 16) / own, in = c * 16 - owner * own;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(peer_addr(mine, (uint32_t)owner) + (uint32_t)(in * BM * 4)), "r"(r[i])
                       : "memory");
          if (++in == own) in = 0, ++owner;
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncwarp();
  cluster_sync();

  // This block's rows, a row a warp at a time, a lane four neighbouring output columns: the parts of K in their order
  if (warp >= 2 && ok) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int n = n0 + 4 * lane;
    const int n_valid = min(4, N - n);
    const bool vec_ok = ((ldo * (long)sizeof(TOut)) % 16 == 0) && (((uintptr_t)out) % 16 == 0) &&
                        (bias == nullptr || ((uintptr_t)bias) % 16 == 0);
    const float* bias4 = bias != nullptr ? bias + n : nullptr;
    // the four columns lie in one head: head sizes and the query width are multiples of 16
    const bool to_cache = kv.pool != nullptr && n >= kv.q_width;
    long long col_off = 0;
    if (to_cache) {
      const int cidx = n - kv.q_width;
      const int which = cidx / kv.kv_width;
      const int rem = cidx - which * kv.kv_width;
      const int head = rem / kv.head_dim;
      col_off = ((long long)(which * kv.n_kv_heads + head) * kv.page_size) * kv.head_dim + (rem - head * kv.head_dim);
    }
    if (n_valid > 0)
      for (int i = warp - 2; i < own; i += RWARPS - 2) {
        const int t = rank * own + i;
        if (t >= M) break;
        float4 acc = *reinterpret_cast<const float4*>(recv + i * BM + 4 * lane);
        for (int p = 1; p < cut.cluster; ++p) {
          const float4 v = *reinterpret_cast<const float4*>(recv + (p * own + i) * BM + 4 * lane);
          acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
        }
        if (to_cache) {
          const long long base = row_base[i];
          if (base >= 0)
            finish4<__nv_bfloat16>((__nv_bfloat16*)kv.pool + base + col_off, acc, bias4, act, 0, true, n_valid);
        } else {
          finish4<TOut>(out + (size_t)t * ldo + n, acc, bias4, act, residual, vec_ok, n_valid);
        }
      }
  }
  __syncwarp();
  if (warp == 1) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)cut.tmem_cols)
                 : "memory");
  }
}

static int rows_sm_count() {
  static int n_sms = 0;
  if (n_sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n_sms, cudaDevAttrMultiProcessorCount, dev);
    if (n_sms <= 0) n_sms = 1;
  }
  return n_sms;
}

// The split of K over the blocks of a cluster, and the ring.  Returns false when the product does not fit this kernel.
static bool rows_cut(int M, int N, int K, RowsCut* out) {
  if (M < 1 || M > 128 || K < 1) return false;
  if (K > RMAX_K) return false;
  RowsCut c;
  c.nt = (M + 15) / 16 * 16;
  c.tmem_cols = c.nt <= 32 ? 32 : (c.nt <= 64 ? 64 : 128);
  const int num_kb = (K + BK - 1) / BK;
  const long tiles = (N + BM - 1) / BM;
  if (tiles > 65535) return false;
  const int n_sms = rows_sm_count();
  long best = -1;
  for (int want = 1; want <= RMAX_CLUSTER; ++want) {
    const int kb_per = (num_kb + want - 1) / want;
    if ((num_kb + kb_per - 1) / kb_per != want) continue;  // no part is empty
    const int own = (c.nt + want - 1) / want;
    const int room = (c.nt <= 64 ? 112 : 220) * 1024 - rows_fixed_bytes(want, own);
    int stages = room / rows_stage_bytes(c.nt);
    stages = stages > RMAX_STAGES ? RMAX_STAGES : stages;
    stages = stages > kb_per ? kb_per : stages;
    if (stages < 1) continue;
    // Nanoseconds, measured over products of 17 to 128 rows with 768 to 6400 columns: a K block more a block costs 450, a block
    // more 12, and what does not stand on the SMs at once (clusters leave some of their places empty) a second round.
    const long blocks = tiles * want, places = (c.nt <= 64 ? 2L : 1L) * n_sms * 5 / 6;
    const long cost = kb_per * 450L + blocks * 12 + want * 50L + (blocks - 1) / places * 4000;
    if (best < 0 || cost < best) {
      best = cost;
      c.cluster = want;
      c.kb_per = kb_per;
      c.stages = stages;
      c.own = own;
      *out = c;
    }
  }
  return best >= 0;
}

template <typename TOut>
static int launch_rows(const void* A, long lda, const void* W, const float* bias, void* out, long ldo, int M, int N,
                       int K, int act, int residual, const KvScatter& kv, int* status, cudaStream_t stream) {
  RowsCut cut;
  if (!rows_cut(M, N, K, &cut)) return -7;
  CUtensorMap mw, ma;
  int rc = tensor_map(W, N, K, K, BM, &mw);
  if (rc != 0) return rc;
  rc = tensor_map(A, M, K, lda, cut.nt, &ma);
  if (rc != 0) return rc;
  static bool attr_set = false;
  if (!attr_set) {
    note_launch(cudaFuncSetAttribute(gemm_tc_rows_kernel<TOut>, cudaFuncAttributeMaxDynamicSharedMemorySize, 224 * 1024));
    note_launch(cudaFuncSetAttribute(gemm_tc_rows_kernel<TOut>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
    attr_set = true;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cut.cluster, (N + BM - 1) / BM);
  cfg.blockDim = dim3(RTHREADS);
  cfg.dynamicSmemBytes = cut.stages * rows_stage_bytes(cut.nt) + rows_fixed_bytes(cut.cluster, cut.own);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cut.cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  note_launch(launch_kernel(cfg, gemm_tc_rows_kernel<TOut>, mw, ma, bias, (TOut*)out, ldo, M, N, K, cut, act, residual, kv, status));
  return take_launch_error();
}

}  // namespace tc
}  // namespace rl

// Whether rl_gemm_tc_rows takes a product of these sizes (1: yes).
RL_EXPORT int rl_gemm_tc_rows_fits(int M, int N, int K) {
  rl::tc::RowsCut cut;
  return rl::tc::rows_cut(M, N, K, &cut) ? 1 : 0;
}

// bfloat16 A [M <= 128, K] (row stride lda) and W [N, K]; out bfloat16 or float32 [M, N].
// residual != 0: out (float32) += result.  kv_pool != nullptr: output columns from kv_q_width
// on are written into cache pages as keys and values, not to out.  Returns -7 when the sizes
// do not fit (more than 128 rows, or K above 8192).
RL_EXPORT int rl_gemm_tc_rows(int out_dtype, const void* A, long lda, const void* W, const float* bias, void* out,
                              long ldo, int M, int N, int K, int act, int residual, void* kv_pool,
                              const int* kv_block_table, int kv_bt_stride, const int* kv_positions,
                              const int* kv_req_of_token, const int* kv_slots, int kv_q_width, int kv_width,
                              int kv_head_dim, int kv_page_size, int kv_heads, int kv_max_pos, int* status,
                              cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K % 8 != 0 || lda % 8 != 0 || ((uintptr_t)A % 16) != 0 || ((uintptr_t)W % 16) != 0) return -2;
  if (residual && out_dtype != RL_F32) return -3;
  if (out_dtype != RL_F32 && out_dtype != RL_BF16) return -4;
  rl::KvScatter kv{kv_pool, kv_block_table, kv_bt_stride, kv_positions, kv_req_of_token, kv_slots,
                   kv_q_width, kv_width, kv_head_dim, kv_page_size, kv_heads, kv_max_pos, status};
  const int rc = out_dtype == RL_F32
                     ? rl::tc::launch_rows<float>(A, lda, W, bias, out, ldo, M, N, K, act, residual, kv, status, stream)
                     : rl::tc::launch_rows<__nv_bfloat16>(A, lda, W, bias, out, ldo, M, N, K, act, residual, kv,
                                                          status, stream);
  if (rc != 0) return rc;
  RL_CHECK_LAUNCH();
  return 0;
}
