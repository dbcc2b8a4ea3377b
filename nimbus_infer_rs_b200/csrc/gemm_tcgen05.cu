// Matrix product on the 5th-generation tensor cores (sm_100a): out[M,N] = act(X[M,K] *
// W[N,K]^T + bias) (+ residual), bf16 operands, fp32 accumulation in tensor memory.
//
// A CTA computes 128 x BN tiles (BN = 64, 96, 128, 192 or 256, picked so that the tiles fill
// the SMs in as few waves as possible), one after another.  Warp 0 is the producer: one thread issues TMA loads of
// 128 x 64 (X) and BN x 64 (W) bf16 boxes, 128-byte swizzled, into a ring of shared-memory
// stages, each guarded by a full/empty mbarrier pair.  Warp 1 owns the tensor memory
// allocation and one of its threads issues `tcgen05.mma` (M=128, N=BN, K=16; four per stage)
// with shared-memory matrix descriptors; `tcgen05.commit` hands a stage back to the producer
// and, after the last K block of a tile, signals that tile's accumulator (there are two, used
// in turn).  The last warp brings the rows of W where the tiles are large (see `split_xw`).
// The other 4 to 16 warps are the epilogue: each reads its share of the columns of
// its 32-lane quarter of the accumulator with `tcgen05.ld`, hands the accumulator back, applies bias / GELU / residual in fp32 and
// stores its rows while the MMAs of the next tile already run.  Edges need no special code on the load side: TMA
// zero-fills rows beyond M or N and columns beyond K.
//
// Every wait on an mbarrier is bounded by a clock budget; a wait that runs out raises an
// error flag (nb_gemm_tcgen05_error), all roles leave their loops, the CTA lets its copies in
// flight land, frees its tensor memory and returns.
//
// Requirements: K % 8 == 0 (16-byte row pitch for TMA), 16-byte aligned bases.
// Reference analogue: Mat::gemm_into (src/model.rs:94-133).
#include "tc05_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

// Tuning (nb_gemm_tcgen05_tune): whether a CTA with one tile and a long K has two MMA-issuing
// threads, and whether the producer is more than one lane.  What a launch passes to the
// kernel: bit 0: two issuing threads; bits 1-2: the producer is 0 one lane, 1 a warp for X and
// a warp for W (large tiles), 2 lanes that share out the ring's stages (a single row tile).
bool g_dual = true, g_lanes = true;

constexpr int BM = 128;
constexpr int BK = 64;               // 64 bf16 = 128 bytes = one swizzle atom row
constexpr int UMMA_K = 16;
// Epilogue warps per CTA: a warp may read only the 32 tensor-memory lanes of its quarter
// (warp index mod 4), so the warps of a quarter share the tile's columns among them.
// With the direct-store epilogue (EPI 0) there are 16 warps for wide tiles, 8 otherwise; with
// the shared-memory / TMA-store epilogue (EPI 1) every warp owns 64 columns of its quarter.
__host__ __device__ constexpr int epi_warps(int bn, int epi) {
  return epi ? 4 * ((bn + 63) / 64) : (bn >= 128 ? 16 : 8);
}
// Tensor-memory columns between the two accumulators of a CTA: allocations are powers of two.
__host__ __device__ constexpr int acc_stride(int bn) {
  return bn <= 64 ? 64 : (bn <= 128 ? 128 : 256);
}
__host__ __device__ constexpr int cta_threads(int bn, int epi) { return 96 + 32 * epi_warps(bn, epi); }

// One CTA per SM walks over tiles; two accumulators in tensor memory let the epilogue of one
// tile overlap the main loop of the next.  EPI 1 adds a staging area for the epilogue: 4 KB
// (32 rows x 128 bytes, 128-byte swizzled) per epilogue warp for bf16 output, twice that for
// fp32 output up to 128 columns (two 32-column boxes per warp, which also receive the residual by
// TMA).  Wider fp32 tiles have one box a warp, through which its two chunks of columns go one after the
// other: what that adds to the epilogue (a store to be read, a second residual to be brought) runs beside
// the next tile's products, and the 64 KB it saves are two stages of the ring.
// PAIR 1: two CTAs of a cluster share 256 x BN tiles (`cta_group::2`): each brings its 128
// rows of X and half of the tile's rows of W, so a stage holds BN / 2 rows of W.
template <int BN, int EPI, int ESIZE, int PAIR>
struct SmemLayout {
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int EPI_WARPS = epi_warps(BN, EPI);
  // fp32 tiles wider than 128 columns: one 32-column box a warp, used twice a tile
  static constexpr int BOXES = ESIZE == 4 && BN <= 128 ? 2 : 1;
  static constexpr int STG_PER_WARP = EPI ? BOXES * 4096 : 0;
  static constexpr int STG_BYTES = EPI_WARPS * STG_PER_WARP;
  static constexpr int BUDGET = 222 * 1024;   // of the 227 KB a CTA may have
  static constexpr int STAGES_RAW = (BUDGET - STG_BYTES) / STAGE_BYTES;
  // 2, 3, 4, 6 or 8 stages: the producer lanes share the stages out among them (see the kernel)
  static constexpr int STAGES = STAGES_RAW > 8 ? 8 : (STAGES_RAW == 7 ? 6 : (STAGES_RAW == 5 ? 4 : STAGES_RAW));
  static constexpr int PRODUCERS = PAIR ? 1 : (STAGES % 4 == 0 ? 4 : (STAGES % 3 == 0 ? 3 : (STAGES % 2 == 0 ? 2 : 1)));
  static constexpr int TILES_BYTES = STAGES * STAGE_BYTES;
  // after tiles and staging: full[STAGES], empty[STAGES], accumulator full[2] / empty[2], two
  // residual barriers per epilogue warp, then the tensor-memory base address and the abort flag
  static constexpr int N_BARRIERS = 2 * STAGES + 4 + 2 * EPI_WARPS;
  static constexpr int TOTAL = TILES_BYTES + STG_BYTES + N_BARRIERS * 8 + 16 + 1024 /* alignment slack */;
};

template <int BN, int EPI, typename TOut, int PAIR>
__global__ void __launch_bounds__(cta_threads(BN, EPI), 1)
gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ CUtensorMap map_out, const float* __restrict__ bias,
                    const float* residual, TOut* out, int M, int N, int K, int act, int tiles_n,
                    int num_tiles, int a_box_bytes, int* err_word, int tune) {
  using L = SmemLayout<BN, EPI, (int)sizeof(TOut), PAIR>;
  constexpr int EW = L::EPI_WARPS;
  constexpr int ACC = acc_stride(BN);
  static_assert(!PAIR || (EPI == 1 && BN % 32 == 0), "paired CTAs: TMA epilogue only");
  static_assert(BN % 32 == 0 && BN >= 32 && BN <= 256, "tile width");
  static_assert(EPI == 1 || BN == 64 || BN == 128 || BN == 256, "direct-store epilogue: 64/128/256");
  static_assert(BN % 64 == 0 || (EPI == 1 && sizeof(TOut) == 4), "odd widths: fp32 TMA epilogue only");
  extern __shared__ unsigned char smem_dyn[];
  // 1024-byte alignment (swizzle atoms), computed on the shared-window address
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char* gen = smem_dyn + (base - raw);
  const uint32_t stg_base = base + L::TILES_BYTES;          // epilogue staging (EPI 1)
  const uint32_t bars = stg_base + L::STG_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (L::STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (2 * L::STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (2 * L::STAGES + 2 + b); };
  auto res_bar = [&](int w, int u) { return bars + 8u * (2 * L::STAGES + 4 + 2 * w + u); };
  uint32_t* tmem_slot =
      reinterpret_cast<uint32_t*>(gen + L::TILES_BYTES + L::STG_BYTES + L::N_BARRIERS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int num_kb = (K + BK - 1) / BK;
  // Paired CTAs: rank 0 is the leader.  It alone issues the MMAs (which read both CTAs'
  // shared memory and write both CTAs' tensor memory); the TMA loads of both CTAs count on the
  // leader's full barriers; commits go to the barriers of both; the epilogue warps of both tell
  // the leader's accumulator-empty barriers.
  uint32_t rank = 0;
  if constexpr (PAIR) asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(rank));
  const int walker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;    // who walks over tiles
  const int n_walkers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int m_off = PAIR ? (int)rank * BM : 0;                   // this CTA's rows in a tile
  constexpr int TILE_M = PAIR ? 2 * BM : BM;

  if (tid == 0) {
    prefetch_tensormap(&map_w);
    prefetch_tensormap(&map_x);
    if constexpr (EPI == 1) prefetch_tensormap(&map_out);
    for (int s = 0; s < L::STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), PAIR ? 2 * EW : EW);   // one arrival per epilogue warp (of both CTAs)
    }
    for (int w = 0; w < EW; ++w) {
      mbar_init(res_bar(w, 0), 1);
      mbar_init(res_bar(w, 1), 1);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if constexpr (PAIR) {   // the peer's barriers exist before anything of ours can reach them
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  if (warp == 1) {   // the whole warp allocates two accumulators, ACC columns apart
    if constexpr (PAIR) {   // warp 1 of both CTAs, the same columns in both
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                       smem_u32(tmem_slot)),
                   "r"((uint32_t)(2 * ACC))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                       smem_u32(tmem_slot)),
                   "r"((uint32_t)(2 * ACC))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
  }
  tc05_fence_before();
  __syncthreads();
  tc05_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Barriers and tensor memory are set up; what the kernel before this one wrote (the rows of
  // X, the residual) is touched from here on.  Under a programmatic launch the set-up above
  // ran while that kernel was finishing -- and so do the loads of the first tile's weights
  // (constants): a product of a decode step is a few microseconds long, and the trip to HBM
  // for its first weights would be a good part of that.
  int pre_kb = 0;   // K blocks whose weights are already on their way (the producer's)
  if (tid == 0 && walker < num_tiles) {
    pre_kb = num_kb < L::STAGES ? num_kb : L::STAGES;
    const int n0 = (walker % tiles_n) * BN + (PAIR ? (int)rank * (BN / 2) : 0);
    for (int kb = 0; kb < pre_kb; ++kb) {
      const uint32_t w_dst = base + kb * L::STAGE_BYTES + L::A_BYTES;
      if constexpr (PAIR) {
        if (rank == 0) mbar_expect_tx(full_bar(kb), 2u * ((uint32_t)a_box_bytes + L::B_BYTES));
        tma_load_2d_pair(w_dst, &map_w, kb * BK, n0, cluster_addr(full_bar(kb), 0));
      } else {
        mbar_expect_tx(full_bar(kb), (uint32_t)a_box_bytes + L::B_BYTES);
        tma_load_2d(w_dst, &map_w, kb * BK, n0, full_bar(kb));
      }
    }
  }
  nb_grid_dependency_wait();
  if (warp == 0) pre_kb = __shfl_sync(0xffffffffu, pre_kb, 0);   // the producer lanes all need it

  // Two issuing threads.  A `tcgen05.mma` costs the thread that issues it about 80 clocks
  // whatever its width, so a CTA with one tile and a long K (a decode step, a short prompt) is
  // bound by that thread while the tensor cores idle; two threads with an accumulator each
  // get rid of an instruction every 50 clocks between them.  The first takes the even blocks
  // of K into the first accumulator, lane 0 of the first epilogue warp (idle until then) the
  // odd ones into the second, and the epilogue adds the two.
  const bool dual = !PAIR && (tune & 1) && num_tiles <= n_walkers && num_kb >= 8;
  auto dual_walk = [&](int first) {
    constexpr uint32_t idesc = instr_desc_bf16(TILE_M, BN);
    const uint32_t d_tmem = tmem_base + (uint32_t)first * ACC;
    bool ok = walker < num_tiles;
    for (int kb = first; kb < num_kb && ok; kb += 2) {
      const int s = kb % L::STAGES;
      ok = mbar_wait(full_bar(s), (uint32_t)(kb / L::STAGES) & 1u, abort_flag);
      if (!ok) break;
      tc05_fence_after();
      const uint32_t a_addr = base + s * L::STAGE_BYTES;
      const uint64_t da = smem_desc_sw128(a_addr);
      const uint64_t db = smem_desc_sw128(a_addr + L::A_BYTES);
#pragma unroll
      for (int k = 0; k < BK / UMMA_K; ++k)
        tc05_mma_bf16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                      (kb > first || k > 0) ? 1u : 0u);
      tc05_commit(empty_bar(s));
    }
    if (ok) tc05_commit(acc_full(first));
  };

  // The CTA walks over output tiles blockIdx.x, blockIdx.x + gridDim.x, ...; the shared-memory
  // ring runs on across tiles, and while the epilogue drains one accumulator the MMAs of the
  // next tile fill the other.
  //
  // A TMA tile load costs its issuing thread about 190 clocks whatever the size of the box
  // (measured: 16 to 256 rows of 128 bytes), so one thread brings in at most 85 bytes a clock
  // with the two boxes of a wide tile and 40 with those of a 64-row product; four lanes of the
  // producer's warp, each with every fourth block of K, reach what the TMA unit takes (about
  // 100 bytes a clock).
  // The number of lanes divides the number of stages, so a lane owns its stages: it fills a
  // stage again only after its own earlier wait for that stage, and can never be two rounds
  // of the ring ahead of the MMAs that free it (where the parity of an older phase of the
  // stage's barrier would pass for the one it waits for), in whatever order two issuing
  // threads consume the stages.
  const int PRODUCERS = (tune >> 1) == 2 ? L::PRODUCERS : 1;
  // Large tiles: warp 0 brings
  // the rows of X, the last warp the rows of W, both block after block in order, so the ring
  // fills in the order the MMAs read it at twice one thread's issue rate.  (As two lanes of one
  // warp they still took turns: 997 x 768 x 3072 16.6 us, as two warps 14.5; 997 x 1024 x 4096
  // 20.8 and 17.8.)  The warp of X arms
  // the stage's barrier with the bytes of both boxes; bytes of W that land before that only
  // take the count below zero for a while (the phase cannot end before the arming arrives).
  const bool split_xw = (tune >> 1) == 1;
  if (warp == 2 + EW && !split_xw) {
    // nothing to bring in
  } else if (split_xw && (warp == 0 || warp == 2 + EW)) {
    const bool rows_of_x = warp == 0;
    if (lane == 0) {
      pre_kb = walker < num_tiles ? (num_kb < L::STAGES ? num_kb : L::STAGES) : 0;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = walker; tile < num_tiles && ok; tile += n_walkers) {
        const int m0 = (tile / tiles_n) * TILE_M + m_off;
        const int n0 = (tile % tiles_n) * BN + (PAIR ? (int)rank * (BN / 2) : 0);
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % L::STAGES;
          const uint32_t phase = (it / L::STAGES) & 1u;
          const bool early = tile == walker && kb < pre_kb;   // armed, W on its way since before the wait
          if (!early) ok = mbar_wait(empty_bar(s), phase ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t a_dst = base + s * L::STAGE_BYTES;
          if constexpr (PAIR) {
            // both CTAs' bytes are counted on the leader's barrier, which the leader arms
            const uint32_t lead_bar = cluster_addr(full_bar(s), 0);
            if (rows_of_x) {
              if (rank == 0 && !early) mbar_expect_tx(full_bar(s), 2u * ((uint32_t)a_box_bytes + L::B_BYTES));
              tma_load_2d_pair(a_dst, &map_x, kb * BK, m0, lead_bar);
            } else if (!early) {
              tma_load_2d_pair(a_dst + L::A_BYTES, &map_w, kb * BK, n0, lead_bar);
            }
            continue;
          }
          if (rows_of_x) {
            if (!early) mbar_expect_tx(full_bar(s), (uint32_t)a_box_bytes + L::B_BYTES);
            tma_load_2d(a_dst, &map_x, kb * BK, m0, full_bar(s));
          } else if (!early) {
            tma_load_2d(a_dst + L::A_BYTES, &map_w, kb * BK, n0, full_bar(s));
          }
        }
      }
      nb_launch_dependents();
    }
  } else if (warp == 0) {
    if (lane < PRODUCERS) {   // --------------------------------------------- TMA producers
      uint32_t it_tile = 0;
      bool ok = true;
      for (int tile = walker; tile < num_tiles && ok; tile += n_walkers, it_tile += (uint32_t)num_kb) {
        const int m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
        // a lane takes every PRODUCERS-th block of the CTA's whole walk (across its tiles)
        const int kb_first = (int)(((uint32_t)lane + PRODUCERS - it_tile % PRODUCERS) % PRODUCERS);
        for (int kb = kb_first; kb < num_kb; kb += PRODUCERS) {
          const uint32_t it = it_tile + (uint32_t)kb;
          const int s = it % L::STAGES;
          const uint32_t phase = (it / L::STAGES) & 1u;
          if (!(tile == walker && kb < pre_kb)) ok = mbar_wait(empty_bar(s), phase ^ 1u, abort_flag);
          if (!ok) break;
          const uint32_t a_dst = base + s * L::STAGE_BYTES;
          if (tile == walker && kb < pre_kb) {
            // the stage was armed and its weights asked for before the wait: the rows follow
            tma_load_2d(a_dst, &map_x, kb * BK, m0, full_bar(s));
          } else {
            // the X box has fewer than 128 rows when the whole product has (see the launcher)
            mbar_expect_tx(full_bar(s), (uint32_t)a_box_bytes + L::B_BYTES);
            tma_load_2d(a_dst, &map_x, kb * BK, m0, full_bar(s));
            tma_load_2d(a_dst + L::A_BYTES, &map_w, kb * BK, n0, full_bar(s));
          }
        }
      }
      // every load of this CTA is on its way: the next kernel may be set up while the last
      // products and the epilogue run
      nb_launch_dependents();
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0 && dual) {
      dual_walk(0);
    } else if (lane == 0 && rank == 0) {   // ----------------------------------- MMA issuer
      constexpr uint32_t idesc = instr_desc_bf16(TILE_M, BN);
      uint32_t it = 0, t = 0;
      bool ok = true;
      for (int tile = walker; tile < num_tiles && ok; tile += n_walkers, ++t) {
        const uint32_t ab = t & 1u, aphase = (t >> 1) & 1u;
        ok = mbar_wait(acc_empty(ab), aphase ^ 1u, abort_flag);   // the epilogue has drained it
        if (!ok) break;
        tc05_fence_after();
        const uint32_t d_tmem = tmem_base + ab * ACC;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % L::STAGES;
          const uint32_t phase = (it / L::STAGES) & 1u;
          ok = mbar_wait(full_bar(s), phase, abort_flag);
          if (!ok) break;
          tc05_fence_after();
          const uint32_t a_addr = base + s * L::STAGE_BYTES;
          const uint64_t da = smem_desc_sw128(a_addr);
          const uint64_t db = smem_desc_sw128(a_addr + L::A_BYTES);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // advancing K by 16 elements inside the swizzle atom = 32 bytes = 2 address units
            if constexpr (PAIR)
              tc05_mma_bf16_pair(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                                 (kb > 0 || k > 0) ? 1u : 0u);
            else
              tc05_mma_bf16(d_tmem, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                            (kb > 0 || k > 0) ? 1u : 0u);
          }
          // the stage is free (in both CTAs) once these MMAs have read it
          if constexpr (PAIR) tc05_commit_pair(empty_bar(s)); else tc05_commit(empty_bar(s));
        }
        // complete once all MMAs issued so far are done
        if (ok) { if constexpr (PAIR) tc05_commit_pair(acc_full(ab)); else tc05_commit(acc_full(ab)); }
      }
    }
  } else if constexpr (EPI == 1) {   // ---------- epilogue through shared memory and TMA stores
    // Warp e of the epilogue owns the 32 tensor-memory lanes of its quarter and one 64-column
    // unit of the tile (the last unit of a 96-wide tile has 32).  bf16 output: the unit is one
    // 32 x 64 box; fp32 output: 32 x 32 boxes, each in a buffer of its own, into which the
    // residual (the output tensor itself, updated in place) is brought by TMA while the
    // accumulator is still being computed.  Rows and columns beyond M and N are clipped by the
    // TMA unit.
    constexpr bool F32 = sizeof(TOut) == 4;
    const int e = warp - 2;
    const int quarter = warp & 3;
    const int unit = e >> 2;                     // 64 columns each
    const int nch = (unit * 64 + 64 <= BN) ? 2 : 1;   // 32-column chunks of this warp's unit
    const uint32_t stg = stg_base + (uint32_t)e * L::STG_PER_WARP;
    const uint32_t my_row = stg + (uint32_t)lane * 128u;
    const uint32_t swz = (uint32_t)(lane & 7);
    uint32_t t = 0;
    const uint32_t lead_empty0 = PAIR ? cluster_addr(acc_empty(0), 0) : 0u;
    if (dual) {   // the second issuing thread, before its warp turns to the epilogue
      if (e == 0 && lane == 0) dual_walk(1);
      __syncwarp();
    }
    for (int tile = walker; tile < num_tiles; tile += n_walkers, ++t) {
      const int m0 = (tile / tiles_n) * TILE_M + m_off, n0 = (tile % tiles_n) * BN;
      const int row0 = m0 + quarter * 32, col0 = n0 + unit * 64;
      const uint32_t ab = t & 1u, aphase = (t >> 1) & 1u;
      if (lane == 0) {
        bulk_wait_read_all();   // the stores of the previous tile have read this warp's buffers
        if (F32 && residual != nullptr) {
          for (int u = 0; u < nch && u < L::BOXES; ++u) {
            mbar_expect_tx(res_bar(e, u), 4096u);
            tma_load_2d(stg + u * 4096u, &map_out, col0 + u * 32, row0, res_bar(e, u));
          }
        }
      }
      __syncwarp();
      // the bias of this warp's columns (a constant) is fetched while the products still run:
      // behind the accumulator it would be a trip to memory at the very end of the kernel
      float bias_pre[2] = {0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (bias && c < nch && col0 + c * 32 + lane < N) bias_pre[c] = __ldg(bias + col0 + c * 32 + lane);
      bool ready =
          __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full(ab), aphase, abort_flag), 0) != 0;
      if (ready && dual)
        ready = __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full(1), 0u, abort_flag), 0) != 0;
      if (!ready) break;
      tc05_fence_after();
#pragma unroll 1
      for (int c = 0; c < nch; ++c) {
        uint32_t v[32];
        tc05_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + ab * ACC +
                               (uint32_t)(unit * 64 + c * 32), v);
        if (dual) {   // the odd blocks of K
          uint32_t w[32];
          tc05_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + ACC +
                                 (uint32_t)(unit * 64 + c * 32), w);
          tc05_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        }
        tc05_wait_ld();
        if (c == nch - 1) {   // this warp has read its share of the accumulator: hand it back
          tc05_fence_before();
          __syncwarp();
          if (lane == 0) {
            if constexpr (PAIR)
              asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(
                               lead_empty0 + 8u * ab)
                           : "memory");
            else
              asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_empty(ab)) : "memory");
          }
        }
        const int nb = col0 + c * 32;
        const float bias_l = c == 0 ? bias_pre[0] : bias_pre[1];
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          f[j] = __uint_as_float(v[j]) + __shfl_sync(0xffffffffu, bias_l, j);
        }
        nb_apply_act_fast_all(f, act);
        if constexpr (F32) {
          const uint32_t box = L::BOXES == 2 ? c * 4096u : 0u;
          const uint32_t buf = my_row + box;
          if (L::BOXES == 1 && c > 0) {      // the box is free once the first chunk's store has read it
            if (lane == 0) {
              bulk_wait_read_all();
              if (residual != nullptr) {
                mbar_expect_tx(res_bar(e, c), 4096u);
                tma_load_2d(stg, &map_out, nb, row0, res_bar(e, c));
              }
            }
            __syncwarp();
          }
          if (residual != nullptr) {
            const bool got = __shfl_sync(0xffffffffu,
                                         (int)mbar_wait(res_bar(e, c), t & 1u, abort_flag), 0) != 0;
            if (got) {
#pragma unroll
              for (int q4 = 0; q4 < 8; ++q4) {
                float4 r4;
                asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                             : "=f"(r4.x), "=f"(r4.y), "=f"(r4.z), "=f"(r4.w)
                             : "r"(buf + (((uint32_t)q4 ^ swz) << 4)));
                f[4 * q4] += r4.x; f[4 * q4 + 1] += r4.y; f[4 * q4 + 2] += r4.z; f[4 * q4 + 3] += r4.w;
              }
            }
          }
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};\n" ::"r"(buf + (((uint32_t)q4 ^ swz) << 4)),
                         "f"(f[4 * q4]), "f"(f[4 * q4 + 1]), "f"(f[4 * q4 + 2]), "f"(f[4 * q4 + 3])
                         : "memory");
          fence_async_smem();
          __syncwarp();
          if (lane == 0 && nb < N && row0 < M) {
            tma_store_2d(&map_out, stg + box, nb, row0);
            bulk_commit();
          }
        } else {
          // 32 columns = four 16-byte pieces of the row's 128 bytes; the second chunk follows
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t p0, p1, p2, p3;
            {
              __nv_bfloat162 h0 = __floats2bfloat162_rn(f[8 * q4], f[8 * q4 + 1]);
              __nv_bfloat162 h1 = __floats2bfloat162_rn(f[8 * q4 + 2], f[8 * q4 + 3]);
              __nv_bfloat162 h2 = __floats2bfloat162_rn(f[8 * q4 + 4], f[8 * q4 + 5]);
              __nv_bfloat162 h3 = __floats2bfloat162_rn(f[8 * q4 + 6], f[8 * q4 + 7]);
              p0 = *reinterpret_cast<uint32_t*>(&h0); p1 = *reinterpret_cast<uint32_t*>(&h1);
              p2 = *reinterpret_cast<uint32_t*>(&h2); p3 = *reinterpret_cast<uint32_t*>(&h3);
            }
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};\n" ::"r"(
                             my_row + ((((uint32_t)(c * 4 + q4)) ^ swz) << 4)),
                         "r"(p0), "r"(p1), "r"(p2), "r"(p3)
                         : "memory");
          }
          if (c == 1) {
            fence_async_smem();
            __syncwarp();
            if (lane == 0 && col0 < N && row0 < M) {
              tma_store_2d(&map_out, stg, col0, row0);
              bulk_commit();
            }
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();   // stores must have left shared memory before it goes away
  } else {             // ------------------------------------------------------ epilogue, direct stores
    const int quarter = warp & 3;   // the 32 tensor-memory lanes this warp may read
    const int half = (warp - 2) >> 2;   // which share of the tile's columns it takes
    constexpr int CHUNKS = BN / 32 / (EW / 4);   // 32-column chunks per warp
    uint32_t t = 0;
    if (dual) {   // the second issuing thread, before its warp turns to the epilogue
      if (warp == 2 && lane == 0) dual_walk(1);
      __syncwarp();
    }
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++t) {
      const int m0 = (tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
      const uint32_t ab = t & 1u, aphase = (t >> 1) & 1u;
      // the bias of this warp's columns, fetched while the products still run
      float bias_pre[CHUNKS];
#pragma unroll
      for (int c = 0; c < CHUNKS; ++c) {
        const int nbc = n0 + (half * CHUNKS + c) * 32;
        bias_pre[c] = (bias && nbc + lane < N) ? __ldg(bias + nbc + lane) : 0.0f;
      }
      // lane 0 decides for the warp: the tensor-memory loads below need all 32 lanes
      bool ready =
          __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full(ab), aphase, abort_flag), 0) != 0;
      if (ready && dual)
        ready = __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full(1), 0u, abort_flag), 0) != 0;
      if (!ready) break;
      tc05_fence_after();
#pragma unroll 1
      for (int c = half * CHUNKS; c < (half + 1) * CHUNKS; ++c) {
        uint32_t v[32];
        tc05_ld_32x32b_x32(
            tmem_base + ((uint32_t)(quarter * 32) << 16) + ab * ACC + (uint32_t)(c * 32), v);
        if (dual) {   // the odd blocks of K
          uint32_t w[32];
          tc05_ld_32x32b_x32(tmem_base + ((uint32_t)(quarter * 32) << 16) + ACC + (uint32_t)(c * 32), w);
          tc05_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        }
        tc05_wait_ld();
        if (c == (half + 1) * CHUNKS - 1) {   // this warp has read its share: hand it back
          tc05_fence_before();
          __syncwarp();
          if (lane == 0)
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_empty(ab)) : "memory");
        }
        const int nb = n0 + c * 32;
        // bias of the chunk's 32 columns: one value per lane
        float bias_l = bias_pre[0];
#pragma unroll
        for (int q = 1; q < CHUNKS; ++q)
          if (c - half * CHUNKS == q) bias_l = bias_pre[q];
        // The accumulator comes with a lane per row and a register per column; stored that way
        // a warp's instruction would touch 32 rows, four bytes each.  The 32 x 32 block is
        // transposed across the warp (five rounds of exchanges between lanes 16, 8, 4, 2, 1
        // apart), after which lane l holds column l and register i row i: an instruction then
        // writes 32 consecutive columns of one row, whatever the width of the output (the
        // logits' 50,257 columns are no multiple of anything).
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
#pragma unroll
        for (int s2 = 16; s2 >= 1; s2 >>= 1) {
          const bool upper = (lane & s2) != 0;
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (j & s2) continue;
            const float send = upper ? f[j] : f[j + s2];
            const float got = __shfl_xor_sync(0xffffffffu, send, s2);
            if (upper) f[j] = got; else f[j + s2] = got;
          }
        }
        const int col = nb + lane;
        const int row0 = m0 + quarter * 32;
        if (col < N) {
#pragma unroll
          for (int i = 0; i < 32; ++i) f[i] += bias_l;
          nb_apply_act_fast_all(f, act);
          float rs[32];   // `residual` may be `out` itself: all of it before the first store
#pragma unroll
          for (int i = 0; i < 32; ++i)
            rs[i] = (residual && row0 + i < M) ? residual[(size_t)(row0 + i) * N + col] : 0.0f;
#pragma unroll
          for (int i = 0; i < 32; ++i) {
            if (row0 + i >= M) break;
            const float y = f[i] + rs[i];
            if constexpr (sizeof(TOut) == 4) reinterpret_cast<float*>(out)[(size_t)(row0 + i) * N + col] = y;
            else reinterpret_cast<bf16*>(out)[(size_t)(row0 + i) * N + col] = __float2bfloat16_rn(y);
          }
        }
      }
    }
  
  }

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
  if constexpr (PAIR) {   // neither CTA leaves while the other may still reach into it
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  if (warp == 1) {
    tc05_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base),
                   "r"((uint32_t)(2 * ACC))
                   : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem_base),
                   "r"((uint32_t)(2 * ACC))
                   : "memory");
  }
}

// The word of pinned host memory in which these kernels report a wait that ran out.
int* error_word() {
  int* w = nb_error_words();
  return w ? w + NB_ERRW_GEMM_TCGEN05 : nullptr;
}

// A wait that nothing ends: one thread waits, with the same bounded wait as the kernels above,
// on a barrier that never gets its arrival, and reports the time-out the way they do.  It is
// how a test sees the limit work without any kernel being made to stall.
__global__ void wait_probe_kernel(int* err_word, int* status) {
  __shared__ __align__(8) unsigned long long bar_mem;
  __shared__ int abort_mem;
  const uint32_t bar = smem_u32(&bar_mem);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    abort_mem = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    const bool ok = mbar_wait(bar, 0u, &abort_mem);
    if (!ok) nb_report_timeout(err_word);
    *status = ok ? 1 : 2;
  }
}

// ---------------------------------------------------------------------------------- host
template <int BN, int EPI, typename TOut, int PAIR = 0>
int launch(const void* X, const void* W, const float* bias, const float* residual, void* out, int M,
           int N, int K, int act, cudaStream_t stream) {
  using L = SmemLayout<BN, EPI, (int)sizeof(TOut), PAIR>;
  static_assert(L::STAGES >= 2, "tile shape leaves no room for a pipeline");
  CUtensorMap mx, mw, mo;
  // A product of fewer than 128 rows brings only its rows (in eighths of a tile) into the X
  // part of a stage: the other rows of the MMA's 128 are whatever shared memory holds, and so
  // are their results, which no epilogue stores (rows >= M).  Fewer bytes per K block matter:
  // a single row tile is a stream bound by what one SM can load.
  const int a_rows = M >= BM ? BM : ((M + 15) / 16) * 16;
  int rc = make_map(&mx, X, M, K, a_rows, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  rc = make_map(&mw, W, N, K, PAIR ? BN / 2 : BN, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  if (EPI) {
    rc = sizeof(TOut) == 4
             ? make_map(&mo, out, M, N, 32, 32, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4)
             : make_map(&mo, out, M, N, 32, 64, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
    if (rc) return rc;
  } else {
    mo = mx;   // unused
  }
  auto kern = gemm_tcgen05_kernel<BN, EPI, TOut, PAIR>;
  const int smem = L::TOTAL;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    configured = true;
  }
  constexpr int TILE_M = PAIR ? 2 * BM : BM;
  const int tiles_n = (N + BN - 1) / BN;
  const long long num_tiles = (long long)tiles_n * ((M + TILE_M - 1) / TILE_M);
  NB_REQUIRE(num_tiles < (1ll << 31), NB_ERR_UNSUPPORTED, "gemm_tcgen05: too many tiles");
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    NB_CUDA(cudaGetDevice(&dev));
    NB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  if constexpr (PAIR) {
    // clusters of two CTAs, one cluster per pair of SMs
    const int pairs = (int)(num_tiles < sms / 2 ? num_tiles : sms / 2);
    NB_CUDA(nb_launch_clusters(kern, dim3(2 * pairs), dim3(cta_threads(BN, EPI)), (size_t)smem, stream, 2, mx, mw,
                               mo, bias, residual, (TOut*)out, M, N, K, act, tiles_n, (int)num_tiles,
                               a_rows * BK * 2, error_word(), 1 << 1));
    return 0;
  }
  const int grid = (int)(num_tiles < sms ? num_tiles : sms);   // one CTA per SM walks the tiles
  // Several producer lanes only for a single row tile (a decode step, a short prompt): its
  // boxes are small and the producer's issue rate bounds the kernel.  With large tiles the
  // MMAs bound it, and lanes that fill the ring out of order only delay the stage the MMAs
  // wait for (a 2,048-token prefill: 1.16 -> 1.28 ms with four lanes); there one warp brings X
  // and one W, both in order (the kernel's `split_xw`).
  const int tune = (g_dual ? 1 : 0) | ((g_lanes ? (M <= BM ? 2 : 1) : 0) << 1);
  NB_CUDA(nb_launch(kern, dim3(grid), dim3(cta_threads(BN, EPI)), (size_t)smem, stream, mx, mw, mo, bias,
                    residual, (TOut*)out, M, N, K, act, tiles_n, (int)num_tiles, a_rows * BK * 2,
                    error_word(), tune));
  return 0;
}

// Tile width.  A single row tile (at most 128 rows) is a weight stream: many narrow tiles
// with a deep ring; of more tiles than SMs (the output head) 128 wide, since an MMA costs its
// issuing thread the same up to 128 columns.
int pick_stream_width(int N) { return (N + 63) / 64 > nb_device_sms() ? 128 : 64; }

// Wider tiles re-read less of X and W from L2, and pairs of CTAs bring half of the weight tile each
// (what bounds a large product is the 64 bytes per clock an SM can take in: 48 KB a block of K
// for a 128 x 256 tile, 32 KB in a pair); but what counts for products of a few hundred tiles is how many
// waves the SMs, or pairs of them, need and how long a wave is.  So every shape has a line
// of its own, us = start + waves x (wave + blocks of K x block), fitted to 13 products of 15 heights from
// 160 to 12,000 rows each, with cold weights and fp32 results added in place or bf16 with GELU: off by 4
// to 7 % on average, and the shape chosen by them 0.1 % slower than the fastest one.  Measured (us; what
// was taken before, with pairs up to 128 columns for fp32 from three waves on, without their early
// start): 4128x1024x4096 34.5 (46.7), 6765x768x3072 38.4 (49.6), 7232x1600x6400 130 (200), 7232x1600x1600 43.8
// (55.7), 2048x1600x6400 39.6 (63.4), 12000x2048x2048 95.7 (127), 6765x2304x768 29.0 (31.1), 4128x3072x768 23.6
// (26.4).
struct TileCost { int bn, pair; float start, wave, block; };
constexpr TileCost COST_F32[] = {{64, 0, 2.07f, 1.30f, 0.253f}, {96, 0, 2.61f, 1.40f, 0.289f}, {128, 0, 2.37f, 1.85f, 0.298f},
                                 {96, 1, 4.73f, 0.57f, 0.285f}, {128, 1, 4.97f, 1.12f, 0.285f}, {192, 1, 4.74f, 2.59f, 0.293f},
                                 {256, 1, 2.33f, 4.56f, 0.367f}};
constexpr TileCost COST_B16[] = {{64, 0, 3.39f, 0.38f, 0.294f}, {128, 0, 3.63f, 1.33f, 0.306f}, {192, 0, 3.78f, 1.60f, 0.345f},
                                 {256, 0, 4.56f, 1.22f, 0.477f}, {128, 1, 5.40f, 0.70f, 0.307f}, {192, 1, 5.39f, 1.25f, 0.317f},
                                 {256, 1, 5.72f, 1.15f, 0.395f}};
// Direct stores (rows that TMA cannot store) take single CTAs of 64, 128 and 256 columns, by fewest waves
// x (width + a tile's fixed cost, about 48 columns' worth of time).
constexpr TileCost COST_DIRECT[] = {{256, 0, 0.0f, 304.0f, 0.0f}, {128, 0, 0.0f, 176.0f, 0.0f}, {64, 0, 0.0f, 112.0f, 0.0f}};

int g_use_pairs = 1;   // pairs of CTAs: 0 off, 1 where they are faster, 2 wherever a paired kernel exists
int g_force_bn = 0, g_force_pair = 0;

template <int COUNT>
TileCost pick_tile(const TileCost (&cost)[COUNT], int M, int N, int K, int pairs) {
  const long long sms = nb_device_sms(), blocks = (K + BK - 1) / BK;
  TileCost best = {};
  float best_us = 0.0f;
  for (const TileCost& c : cost) {
    if (c.pair ? pairs == 0 || M <= BM : pairs == 2 && M > BM) continue;
    if (c.bn > N && c.bn > 64 && !(c.pair && c.bn == 96) && !(pairs == 2 && c.bn == 128)) continue;   // wider than the output
    const long long rows = c.pair ? 2 * BM : BM, walkers = c.pair ? sms / 2 : sms;
    const long long tiles = ((M + rows - 1) / rows) * ((N + c.bn - 1) / c.bn);
    const float us = c.start + (float)((tiles + walkers - 1) / walkers) * (c.wave + (float)blocks * c.block);
    if (best.bn == 0 || us < best_us) { best = c; best_us = us; }
  }
  return best;
}

template <int COUNT>
bool has_tile(const TileCost (&cost)[COUNT], int bn, int pair) {
  for (const TileCost& c : cost)
    if (c.bn == bn && c.pair == pair) return true;
  return false;
}

}  // namespace

// 1 if the tensor-core kernel takes this product.
NB_EXPORT int nb_gemm_tcgen05_supported(int x_dtype, int w_dtype, int M, int N, int K) {
  return x_dtype == NB_BF16 && w_dtype == NB_BF16 && K % 8 == 0 && M >= 1 && N >= 1 && K >= 8 &&
         (M + BM - 1) / BM <= 65535;
}

// Comparison runs: two MMA-issuing threads on or off, several producer lanes on or off.
NB_EXPORT int nb_gemm_tcgen05_tune(int dual, int lanes) {
  g_dual = dual != 0;
  g_lanes = lanes != 0;
  return 0;
}

// Tuning and tests: a tile width and whether pairs of CTAs take it (0: choose).  While one is set, products
// that have no kernel of it (of that result type, of up to 128 rows, with direct stores) are refused.
NB_EXPORT int nb_gemm_tcgen05_force(int width, int pair) {
  NB_REQUIRE(width == 0 || has_tile(COST_F32, width, pair) || has_tile(COST_B16, width, pair), NB_ERR_BAD_ARG,
             "gemm_tcgen05: no tile of %d columns%s", width, pair ? " for pairs of CTAs" : "");
  g_force_bn = width;
  g_force_pair = pair;
  return 0;
}

// Pairs of CTAs on 256-row tiles: 0 never, 1 where the cost model prefers them, 2 wherever a
// paired kernel exists.
NB_EXPORT int nb_gemm_tcgen05_use_pairs(int mode) {
  g_use_pairs = mode < 0 ? 0 : (mode > 2 ? 2 : mode);
  return 0;
}

// Waits for the device, then reads (and lowers) the word that a timed-out wait of these kernels
// raises.
NB_EXPORT int nb_gemm_tcgen05_error() {
  if (cudaDeviceSynchronize() != cudaSuccess) return -1;
  volatile int* w = error_word();
  if (w == nullptr) return 0;
  const int v = *w;
  if (v) *w = 0;
  return v;
}

// Clock cycles a wait of these kernels may take before it gives up (default 4e9, about two
// seconds).  Takes effect for kernels launched after the call.
NB_EXPORT int nb_gemm_tcgen05_set_wait_budget(long long cycles) {
  NB_REQUIRE(cycles >= 0, NB_ERR_BAD_ARG, "wait budget must not be negative");
  return set_wait_budget(cycles);
}

// Runs the bounded wait on a barrier that nothing completes: `status` (device int) receives 2
// when the wait gave up after the budget (and the probe's error word is raised), 1 if it came
// back complete.
NB_EXPORT int nb_wait_probe(int* status, cudaStream_t stream) {
  int* w = nb_error_words();
  wait_probe_kernel<<<1, 32, 0, stream>>>(w ? w + NB_ERRW_PROBE : nullptr, status);
  NB_CHECK_LAUNCH("wait_probe");
  return 0;
}

NB_EXPORT int nb_gemm_tcgen05(const void* X, const void* W, const float* bias, const float* residual,
                              void* out, int out_dtype, int M, int N, int K, int act,
                              cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  NB_REQUIRE(nb_gemm_tcgen05_supported(NB_BF16, NB_BF16, M, N, K), NB_ERR_UNSUPPORTED,
             "gemm_tcgen05: needs bf16 operands and a width that is a multiple of 8 (M=%d N=%d K=%d)",
             M, N, K);
  NB_REQUIRE((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)out % 16 == 0 &&
                 (uintptr_t)residual % 16 == 0,
             NB_ERR_UNSUPPORTED, "gemm_tcgen05: operands must be 16-byte aligned");
  // Epilogue through shared memory and TMA stores (full-line writes, residual fetched by TMA)
  // when the output rows are 16-byte multiples and the residual, if any, is the output
  // itself; otherwise every thread stores its own row segment.
  const int esize = out_dtype == NB_F32 ? 4 : 2;
  const bool tma_epi = ((long long)N * esize) % 16 == 0 && (residual == nullptr || residual == out);
  NB_REQUIRE(g_force_bn == 0 || (M > BM && tma_epi && (out_dtype == NB_F32 ? has_tile(COST_F32, g_force_bn, g_force_pair)
                                                                         : has_tile(COST_B16, g_force_bn, g_force_pair))),
             NB_ERR_BAD_ARG, "gemm_tcgen05: this product has no kernel of the %d columns that are set", g_force_bn);
  TileCost tile = {M <= BM ? pick_stream_width(N) : 0, 0};
  if (M > BM) {
    if (!tma_epi) tile = pick_tile(COST_DIRECT, M, N, K, 0);
    else if (g_force_bn) tile = {g_force_bn, g_force_pair};
    else if (out_dtype == NB_F32) tile = pick_tile(COST_F32, M, N, K, g_use_pairs);
    else tile = pick_tile(COST_B16, M, N, K, g_use_pairs);
  }
  const int bn = tile.bn, pair_bn = tile.pair ? tile.bn : 0;
  int rc;
  if (pair_bn) {
    rc = NB_ERR_BAD_ARG;
    if (out_dtype == NB_F32) {
      if (pair_bn == 256) rc = launch<256, 1, float, 1>(X, W, bias, residual, out, M, N, K, act, stream);
      else if (pair_bn == 192) rc = launch<192, 1, float, 1>(X, W, bias, residual, out, M, N, K, act, stream);
      else if (pair_bn == 128) rc = launch<128, 1, float, 1>(X, W, bias, residual, out, M, N, K, act, stream);
      else if (pair_bn == 96) rc = launch<96, 1, float, 1>(X, W, bias, residual, out, M, N, K, act, stream);
    } else if (out_dtype == NB_BF16) {
      if (pair_bn == 256) rc = launch<256, 1, bf16, 1>(X, W, bias, residual, out, M, N, K, act, stream);
      else if (pair_bn == 192) rc = launch<192, 1, bf16, 1>(X, W, bias, residual, out, M, N, K, act, stream);
      else if (pair_bn == 128) rc = launch<128, 1, bf16, 1>(X, W, bias, residual, out, M, N, K, act, stream);
    }
    NB_REQUIRE(rc != NB_ERR_BAD_ARG, NB_ERR_BAD_ARG, "gemm_tcgen05: no paired kernel of width %d", pair_bn);
    if (rc) return rc;
    NB_CHECK_LAUNCH("gemm_tcgen05");
    return 0;
  }
#define NB_TC(BN_, EPI_, T_) rc = launch<BN_, EPI_, T_>(X, W, bias, residual, out, M, N, K, act, stream)
  if (out_dtype == NB_F32) {
    if (tma_epi) {
      if (bn == 128) NB_TC(128, 1, float); else if (bn == 96) NB_TC(96, 1, float); else NB_TC(64, 1, float);
    } else {
      if (bn == 256) NB_TC(256, 0, float); else if (bn == 128) NB_TC(128, 0, float); else NB_TC(64, 0, float);
    }
  } else if (out_dtype == NB_BF16) {
    if (tma_epi) {
      if (bn == 256) NB_TC(256, 1, bf16); else if (bn == 192) NB_TC(192, 1, bf16);
      else if (bn == 128) NB_TC(128, 1, bf16); else NB_TC(64, 1, bf16);
    } else {
      if (bn == 256) NB_TC(256, 0, bf16); else if (bn == 128) NB_TC(128, 0, bf16); else NB_TC(64, 0, bf16);
    }
  } else {
    NB_REQUIRE(false, NB_ERR_BAD_ARG, "gemm_tcgen05: unknown output dtype %d", out_dtype);
  }
#undef NB_TC
  if (rc) return rc;
  NB_CHECK_LAUNCH("gemm_tcgen05");
  return 0;
}
