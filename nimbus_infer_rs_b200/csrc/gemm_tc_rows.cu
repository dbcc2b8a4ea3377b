// Matrix product for 17 to 128 rows (a decode step of a larger batch, a short prompt) on the
// 5th-generation tensor cores: out[M,N] = act(X[M,K] * W[N,K]^T + bias) (+ residual), bf16
// operands, fp32 accumulation in tensor memory.
//
// What bounds such a product is not the tensor cores but the thread that feeds them: one
// `tcgen05.mma` costs its issuing thread about 80 clocks whatever its width up to 128 columns
// (measured on a B200: 81 clocks an instruction at N = 32, 64 and 128, 142 at N = 256).  So the
// kernel makes every instruction cover as many weights as it can and gives every CTA few of
// them:
//   * the operands are swapped: the weights are the 128-row operand (A), the step's rows the
//     narrow one (B, N = rows rounded up to 16), so an instruction covers 128 weight rows
//     whatever the number of rows of X -- the accumulator is the product's transpose, 128
//     weight rows (tensor-memory lanes) x rows of X (columns);
//   * K is cut among the CTAs of a thread-block cluster (1 to 8), chosen so that the launch
//     fills the GPU once: each CTA walks over its run of 64-column blocks of K into its own
//     accumulator;
//   * the sums meet through distributed shared memory: every CTA turns its accumulator over into
//     its own shared memory (over the ring, which is free by then) as rows of X x 128 columns; behind a
//     cluster barrier each CTA takes its share of the rows from all of them, 512 consecutive bytes a
//     warp, adds in rank order (the result does not depend on timing), applies bias,
//     activation and residual and stores 16 bytes a thread.  (Sent out instead with `st.async`, 16
//     bytes a store, the exchange went at 8 bytes a clock and SM: 64x2304x1600 15.2 us for 7.2 now,
//     64x768x3072 8.5 for 6.2, 128x1600x6400 18.3 for 11.4)
// Warp 0 issues the TMA loads (128 x 64 boxes of W, rows x 64 boxes of X, 128-byte
// swizzled) into a ring of stages of 200 KB at most (a block of cold weights is 1.5 us away: 128x1600x6400
// 13.4 us with 104 KB); the weights of the first stages are asked for before the wait on the kernel in front (they are
// constants).  Warp 1 owns the tensor memory and issues the MMAs.  Warps 2 to 9 are the epilogue, two per
// quarter of the lanes.
//
// Every wait on an mbarrier is bounded by a clock budget; a wait that runs out raises the
// kernel's error word, all roles leave their loops, every thread still passes the cluster's
// barriers (a hardware barrier has no limit of its own, so nobody may skip it), the CTA frees
// its tensor memory and returns.
//
// Requirements: K % 8 == 0 (16-byte row pitch for TMA), 16-byte aligned bases, N at most
// 128 x the number of SMs.  Reference analogue: Mat::gemm_into (src/model.rs:94-133).
#include "tc05_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BW = 128;              // weight rows per tile = rows of the MMA
constexpr int BK = 64;               // 64 bf16 = 128 bytes = one swizzle atom row
constexpr int UMMA_K = 16;
constexpr int MAX_ROWS = 128;
constexpr int MAX_STAGES = 8;
constexpr int MAX_SPLIT = 8;         // portable cluster size
constexpr int W_BYTES = BW * BK * 2;                 // 16 KB
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 64 + EPI_WARPS * 32;
constexpr int SMEM_BUDGET = 200 * 1024;
constexpr int AHEAD = 2;             // pieces of the residual a thread asks for ahead

struct RowsShape {
  int nb;            // rows of X rounded up to 16: the MMA's N
  int split;         // CTAs of a cluster = runs of K
  int kb_per;        // K blocks per CTA
  int stages;        // stages of the ring
  int stage_bytes;   // W box + X box
  int x_bytes;       // X box
  int chunk;         // rows of X a CTA finishes (a multiple of 4)
  int body;          // bytes of the ring, and of the sums that take its place
  int tmem_cols;     // power of two >= nb, >= 32
  int smem;          // dynamic shared memory
};

__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}

template <typename TOut>
__global__ void __launch_bounds__(THREADS)
gemm_tc_rows_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const float* __restrict__ bias, const float* residual, TOut* out, int M, int N,
                    int K, int act, RowsShape sh, bool vec, int* err_word) {
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;          // swizzle atoms want 1024-byte alignment
  unsigned char* gen = smem_dyn + (base - raw);
  // [ring of stages, then sums: [row of X][128 weight rows]] [barriers] [tmem slot, abort]
  const uint32_t bars = base + (uint32_t)sh.body;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
  const uint32_t acc_full = bars + 8u * (2 * MAX_STAGES);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen + sh.body + (2 * MAX_STAGES + 2) * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  const int n0 = (int)(blockIdx.x / sh.split) * BW;
  const int num_kb = (K + BK - 1) / BK;
  const int kb_lo = (int)rank * sh.kb_per, kb_hi = min(num_kb, kb_lo + sh.kb_per);
  const int n_kb = max(0, kb_hi - kb_lo);

  if (tid == 0) {
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
    for (int s = 0; s < sh.stages; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)sh.tmem_cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc05_fence_before();
  __syncthreads();
  tc05_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  // The weights of the first stages are constants: they are asked for while the kernel in
  // front is still running.  Nothing that concerns the cluster happens before the wait.
  int pre_kb = 0;
  if (tid == 0) {
    pre_kb = min(n_kb, sh.stages);
    for (int i = 0; i < pre_kb; ++i) {
      mbar_expect_tx(full_bar(i), (uint32_t)sh.stage_bytes);
      tma_load_2d(base + i * sh.stage_bytes, &map_w, (kb_lo + i) * BK, n0, full_bar(i));
    }
  }
  nb_grid_dependency_wait();
  // the rows this CTA finishes; a thread of the epilogue takes four columns, the same in every row
  const int m_lo = (int)rank * sh.chunk, m_hi = min(M, m_lo + sh.chunk);
  const int row_first = m_lo + (warp - 2), n = n0 + lane * 4;
  float4 ahead[AHEAD];
  float b4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (warp >= 2) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (bias != nullptr && n + j < N) b4[j] = __ldg(bias + n + j);
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int m = row_first + i * EPI_WARPS;
      ahead[i] = (vec && residual != nullptr && m < m_hi && n < N)
                     ? *reinterpret_cast<const float4*>(residual + (size_t)m * N + n)
                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }

  if (warp == 0) {
    // A TMA tile load costs its issuing thread about 190 clocks whatever the size of its box:
    // up to four lanes, each with every n-th block of K, keep the TMA unit busy.  Their number
    // divides the number of stages, so a lane owns its stages and fills one again only after
    // its own earlier wait for it: it can never be two rounds of the ring ahead of the MMAs
    // (where the parity of an older phase of the stage's barrier would pass for the awaited one).
    pre_kb = __shfl_sync(0xffffffffu, pre_kb, 0);
    const int producers = n_kb <= sh.stages ? 4      // no stage is filled twice
                          : sh.stages % 4 == 0 ? 4 : (sh.stages % 3 == 0 ? 3 : (sh.stages % 2 == 0 ? 2 : 1));
    if (lane < producers) {   // --------------------------------------------- TMA producers
      for (int i = lane; i < n_kb; i += producers) {
        const int s = i % sh.stages;
        const uint32_t dst = base + s * sh.stage_bytes;
        if (i < pre_kb) {   // armed, and its weights on their way: the rows follow
          tma_load_2d(dst + W_BYTES, &map_x, (kb_lo + i) * BK, 0, full_bar(s));
          continue;
        }
        if (!mbar_wait(empty_bar(s), ((i / sh.stages) & 1u) ^ 1u, abort_flag)) break;
        mbar_expect_tx(full_bar(s), (uint32_t)sh.stage_bytes);
        tma_load_2d(dst + W_BYTES, &map_x, (kb_lo + i) * BK, 0, full_bar(s));
        tma_load_2d(dst, &map_w, (kb_lo + i) * BK, n0, full_bar(s));
      }
      nb_launch_dependents();   // every load is on its way
    }
  } else if (warp == 1) {
    if (lane == 0) {   // ------------------------------------------------------ MMA issuer
      const uint32_t idesc = instr_desc_bf16(BW, sh.nb);
      bool ok = true;
      for (int i = 0; i < n_kb && ok; ++i) {
        const int s = i % sh.stages;
        ok = mbar_wait(full_bar(s), (i / sh.stages) & 1u, abort_flag);
        if (!ok) break;
        tc05_fence_after();
        const uint32_t w_addr = base + s * sh.stage_bytes;
        const uint64_t da = smem_desc_sw128(w_addr);
        const uint64_t db = smem_desc_sw128(w_addr + W_BYTES);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)   // 16 elements of K = 32 bytes = 2 address units
          tc05_mma_bf16(tmem_base, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                        (i > 0 || k > 0) ? 1u : 0u);
        if (i + sh.stages < n_kb) tc05_commit(empty_bar(s));   // only a stage that is used again
      }
      if (ok) {
        if (n_kb > 0) tc05_commit(acc_full);
        else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_full) : "memory");
      }
    }
  }

  // ---- epilogue warps: this CTA's sums are complete (and the ring free)
  float* sums = reinterpret_cast<float*>(gen);
  if (warp >= 2 && __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full, 0u, abort_flag), 0) != 0) {
    tc05_fence_after();
    const int quarter = warp & 3;                 // the 32 tensor-memory lanes this warp may read
    float* column = sums + quarter * 32 + lane;   // its weight row's sums, one a row of X
    for (int c0 = (warp - 2) / 4 * 32; c0 < sh.nb; c0 += 64) {
      uint32_t v[32];
      tc05_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
      tc05_wait_ld();
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (c0 + j < sh.nb) column[(c0 + j) * BW] = __uint_as_float(v[j]);
    }
    tc05_fence_before();
  }
  __syncwarp();
  if (sh.split > 1)
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  else
    __syncthreads();
  if (warp >= 2 && *abort_flag == 0) {
    int i = 0;
#pragma unroll 2
    for (int m = row_first; m < m_hi; m += EPI_WARPS, ++i) {
      const uint32_t at = base + (uint32_t)((m * BW + lane * 4) * 4);
      float y[4] = {0.0f, 0.0f, 0.0f, 0.0f}, r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      float4 part[MAX_SPLIT];
#pragma unroll
      for (int q = 0; q < MAX_SPLIT; ++q)           // all asked for before the first is used
        if (q < sh.split) part[q] = ld_cluster4(cluster_addr(at, (uint32_t)q));
#pragma unroll
      for (int q = 0; q < MAX_SPLIT; ++q) {
        if (q >= sh.split) break;
        y[0] += part[q].x; y[1] += part[q].y; y[2] += part[q].z; y[3] += part[q].w;
      }
      if (n >= N) continue;
      const size_t o = (size_t)m * N + n;
      if (residual != nullptr) {
        if (vec) {
          const float4 q = i == 0 ? ahead[0] : i == 1 ? ahead[1] : *reinterpret_cast<const float4*>(residual + o);
          r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N) r[j] = residual[o + j];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] += b4[j];
      nb_apply_act_fast_all(y, act);
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] += r[j];
      if (vec) {
        if constexpr (sizeof(TOut) == 4) {
          *reinterpret_cast<float4*>(out + o) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
          uint2 u;
          __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
          h[0] = __floats2bfloat162_rn(y[0], y[1]);
          h[1] = __floats2bfloat162_rn(y[2], y[3]);
          *reinterpret_cast<uint2*>(out + o) = u;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < N) out[o + j] = nb_from_f32<TOut>(y[j]);
      }
    }
  }
  __syncwarp();
  if (sh.split > 1)       // nobody leaves while another reads its shared memory
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  tc05_fence_before();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) {
      nb_report_timeout(err_word);
      // let TMA copies that are still in flight land before the shared memory goes away
      const long long t0 = clock64();
      while (clock64() - t0 < 4000000LL) {
      }
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base),
                 "r"((uint32_t)sh.tmem_cols)
                 : "memory");
  }
}

int* error_word() {
  int* w = nb_error_words();
  return w ? w + NB_ERRW_GEMM_TC_ROWS : nullptr;
}

int g_force_split = 0;   // tuning and tests: 0 = choose

// How the product is laid out, or false if this kernel does not take it.  The cluster size is
// the one with the shortest walk per CTA (the larger of what its MMAs cost the issuing thread
// and what its loads cost the SM's 64 bytes a clock) plus what a cluster costs, among those
// that put the whole launch on the GPU at once.
bool plan_rows(int M, int N, int K, RowsShape* out) {
  if (M < 1 || M > MAX_ROWS || N < 1 || K < 8 || K % 8 != 0) return false;
  const int sms = nb_device_sms();
  const int tiles_n = (N + BW - 1) / BW;
  if (tiles_n > sms) return false;
  RowsShape s;
  s.nb = (M + 15) / 16 * 16;
  s.x_bytes = s.nb * BK * 2;
  s.stage_bytes = W_BYTES + s.x_bytes;
  s.tmem_cols = s.nb <= 32 ? 32 : (s.nb <= 64 ? 64 : 128);
  const int num_kb = (K + BK - 1) / BK;
  long long best_cost = -1;
  int best = 1;
  for (int split = 1; split <= MAX_SPLIT; ++split) {
    if (g_force_split && split != g_force_split) continue;
    if (tiles_n * split > sms && split > 1) break;
    const int kb_per = (num_kb + split - 1) / split;
    if (split > 1 && (split - 1) * kb_per >= num_kb) continue;   // a CTA without a K block
    const long long mma = (long long)kb_per * (BK / UMMA_K) * 85;
    const long long load = (long long)kb_per * s.stage_bytes / 55;
    const long long cost = (mma > load ? mma : load) + (split > 1 ? 600 : 0) + 40LL * split;
    if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = split; }
  }
  if (best_cost < 0) return false;
  s.split = best;
  s.kb_per = (num_kb + best - 1) / best;
  s.chunk = ((s.nb + best - 1) / best + 3) / 4 * 4;
  int stages = s.kb_per < MAX_STAGES ? s.kb_per : MAX_STAGES;
  while (stages > 1 && stages * s.stage_bytes > SMEM_BUDGET) --stages;
  if (stages < s.kb_per && (stages == 5 || stages == 7)) --stages;     // four or three lanes bring them in
  s.stages = stages;
  const int sums = s.nb * BW * 4;
  s.body = stages * s.stage_bytes > sums ? stages * s.stage_bytes : sums;
  s.smem = s.body + (2 * MAX_STAGES + 2) * 8 + 16 + 1024;
  if (s.smem > 227 * 1024) return false;
  *out = s;
  return true;
}

template <typename TOut>
int launch_rows(const void* X, const void* W, const float* bias, const float* residual, void* out,
                int M, int N, int K, int act, const RowsShape& sh, cudaStream_t stream) {
  CUtensorMap mx, mw;
  int rc = make_map(&mx, X, M, K, sh.nb, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  rc = make_map(&mw, W, N, K, BW, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  auto kern = gemm_tc_rows_kernel<TOut>;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    configured = true;
  }
  const int tiles_n = (N + BW - 1) / BW;
  const bool vec = N % 4 == 0 && (uintptr_t)out % (4 * sizeof(TOut)) == 0 && (uintptr_t)residual % 16 == 0;
  NB_CUDA(nb_launch_clusters(kern, dim3(tiles_n * sh.split), dim3(THREADS), (size_t)sh.smem, stream,
                             sh.split, mx, mw, bias, residual, (TOut*)out, M, N, K, act, sh, vec,
                             error_word()));
  return 0;
}

}  // namespace

// 1 if this kernel takes the product.
NB_EXPORT int nb_gemm_tc_rows_supported(int M, int N, int K) {
  RowsShape sh;
  return plan_rows(M, N, K, &sh) ? 1 : 0;
}

// 1 where this kernel is taken before the tiled one: a long K (24 blocks and more) over few columns,
// where the tiled kernel has few CTAs and each a long walk.  The line is from measurements with an exchange that
// this kernel no longer has.  Chains of products over cold weights, 32-bit results added in place (bf16 with
// GELU), us, here and tiled: 64x2304x1600 7.3 and 9.6 (7.3 and 8.6), 96x4096x3072 11.0 and 17.0 (11.0 and 15.0),
// 128x4096x6400 17.0 and 32.4; over the 144 shapes between 2,304 and 4,736 columns that it gives this kernel 0.83
// (0.95) of the tiled one's time.  But it takes some that the tiled kernel is faster at, near its end in columns
// and at some cuts of K (64x4736x1600 13.7 and 9.9, 96x2304x1600 12.7 and 9.9, 64x3072x2048 13.2 and
// 11.9), and leaves some beyond it (64x4800x3072 12.4 and 16.9, 128x4800x6400 21.2 and 33.1); up to 64
// rows gemm_mid.cu is as fast as this kernel or faster at most of them (64x3072x3072 9.9 and 14.8).
NB_EXPORT int nb_gemm_tc_rows_preferred(int M, int N, int K) {
  RowsShape sh;
  if (!plan_rows(M, N, K, &sh)) return 0;
  const int num_kb = (K + BK - 1) / BK;
  return num_kb >= 24 && N <= 74 * 64 && (M <= 96 || num_kb >= 48);
}

// The layout chosen for a shape (tests and reports): nb, split, kb_per, stages, chunk, smem.
NB_EXPORT int nb_gemm_tc_rows_plan(int M, int N, int K, int* out6) {
  RowsShape sh;
  if (!plan_rows(M, N, K, &sh)) return 0;
  out6[0] = sh.nb; out6[1] = sh.split; out6[2] = sh.kb_per; out6[3] = sh.stages; out6[4] = sh.chunk;
  out6[5] = sh.smem;
  return 1;
}

// Tuning and tests: the cluster size to use (0 = choose).  Returns the earlier setting.
NB_EXPORT int nb_gemm_tc_rows_force_split(int split) {
  const int was = g_force_split;
  g_force_split = split < 0 ? 0 : (split > MAX_SPLIT ? MAX_SPLIT : split);
  return was;
}

NB_EXPORT int nb_gemm_tc_rows_set_wait_budget(long long cycles) { return set_wait_budget(cycles); }

NB_EXPORT int nb_gemm_tc_rows(const void* X, const void* W, const float* bias, const float* residual,
                              void* out, int out_dtype, int M, int N, int K, int act,
                              cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  RowsShape sh;
  NB_REQUIRE(plan_rows(M, N, K, &sh), NB_ERR_UNSUPPORTED,
             "gemm_tc_rows: takes 1 to %d rows, K a multiple of 8 and at most %d columns (M=%d N=%d K=%d)",
             MAX_ROWS, BW * nb_device_sms(), M, N, K);
  NB_REQUIRE((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0, NB_ERR_UNSUPPORTED,
             "gemm_tc_rows: operands must be 16-byte aligned");
  int rc;
  if (out_dtype == NB_F32)
    rc = launch_rows<float>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  else if (out_dtype == NB_BF16)
    rc = launch_rows<bf16>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  else
    NB_REQUIRE(false, NB_ERR_BAD_ARG, "gemm_tc_rows: unknown output dtype %d", out_dtype);
  if (rc) return rc;
  NB_CHECK_LAUNCH("gemm_tc_rows");
  return 0;
}
