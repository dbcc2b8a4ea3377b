// Matrix product of fp32 rows with fp32 weights on the tensor cores, out[M,N] = act(X W^T + bias)
// (+ residual), as exact as fp32 multiply-adds: the prompts of the true 32-bit path.
//
// The multiply-adds of the CUDA cores bound such a product at some 40 TFLOP/s (gemm_f32.cu).  Every
// fp32 number is the sum of three bf16 numbers, x = h + m + l (8 bits of the mantissa each), so
//   x w = hh' + (hm' + mh') + (mm' + hl' + lh') + (ml' + lm' + ll')
// and all but the last bracket, which is below 2^-24 of the product, is computed: six products
// of bf16 tiles by tcgen05, whose products are exact.  What is not exact is the tensor cores'
// accumulation: it cuts instead of rounding, and its error grows with the number of
// instructions added up in one place (7.3e-7 of the result after 48, 3.2e-6 after 192).  So
// the large terms hh' are taken out of tensor memory every 8 instructions (128 numbers of K) and
// added up in registers, rounded; the small ones have an accumulator of their own, in which the
// same error counts 2^-8 as much.
//
// A pass of its own (split_kernel, a warp a row) writes the three pieces of the rows of X and of W
// into scratch memory, every time: nothing is kept from one call to the next.  It also marks the
// rows that cannot be split: those with an infinity or NaN in them (infinity minus infinity) and
// those all of whose numbers are so small that the last piece would be subnormal; their results
// are computed by plain multiply-adds in the epilogue.
//
// Error against 64 bits (2-norm, normal rows, weights of 0.02): 1.5e-7 at K = 768 and 2.3e-7 at
// 3072, where multiply-adds in one sequence have 3.5e-7 and 7.0e-7, in eight parts 1.8e-7 and 2.6e-7.
//
// A CTA takes a 128 x 128 tile.  A block of 64 of K takes 2,800 clocks, where its 24 instructions
// cost their issuing thread 1,900 and its 96 KB of loads want 1,750 at the 55 bytes a clock an SM
// takes in; neither handing the pieces back to the loads one by one nor a second issuing thread
// made a prompt faster by more than the timing varies (two prompts of GPT-2 124M 6.21 and 6.16 ms).
// Warp 0 brings the pieces of 64 columns of K by TMA (six 128 x 64
// boxes a block, two blocks in flight), warp 1 issues the MMAs, eight warps take the
// accumulators out and finish the tile through shared memory.  Every wait has a clock budget.
//
// Reference analogue: Mat::gemm_into (src/model.rs:88-133).
#include "tc05_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BN = 128, BK = 64;
constexpr int PIECE = BM * BK * 2;          // bytes of a 128 x 64 box
constexpr int BLOCK_BYTES = 6 * PIECE;      // X's three pieces, W's three pieces
constexpr int STAGES = 2;                   // blocks of K in flight
constexpr int CHUNK = 2;                    // blocks of K between two takings-out
constexpr int EPI = 8;                      // warps of the epilogue
constexpr int THREADS = 64 + 32 * EPI;
constexpr int OLD = BN + 4;                 // floats between rows of the finished tile
constexpr int SMEM = STAGES * BLOCK_BYTES + 1024 + 256;
static_assert(BM * OLD * 4 <= STAGES * BLOCK_BYTES, "the finished tile goes where the ring was");

__device__ __forceinline__ void split3(float x, bool whole, bf16& h, bf16& m, bf16& l) {
  h = whole ? __float2bfloat16_rz(x) : __float2bfloat16_rn(0.0f);
  const float r = whole ? x - __bfloat162float(h) : 0.0f;       // exact
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(r - __bfloat162float(m));             // exact
}

// Rows 0 .. M-1 of X and 0 .. N-1 of W, a warp each, into pieces [3][rows][K]; flags[row] = 1 for
// rows that cannot be split (their pieces are zeros).  K % 4 == 0.
__global__ void __launch_bounds__(256)
split_kernel(const float* X, const float* __restrict__ W, bf16* xp, bf16* wp, int* x_flags, int* w_flags,
             int M, int N, int K) {
  nb_grid_dependency_wait();
  nb_launch_dependents();
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= M + N) return;
  const bool is_w = row >= M;
  const int r = is_w ? row - M : row, rows = is_w ? N : M;
  const float4* src = reinterpret_cast<const float4*>((is_w ? W : X) + (size_t)r * K);
  bf16* dst = (is_w ? wp : xp) + (size_t)r * K;
  float top = 0.0f;
  bool finite = true;
  for (int k = lane; k < K / 4; k += 32) {
    const float4 f = src[k];
    const float v[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      finite = finite && (__float_as_uint(v[e]) & 0x7f800000u) != 0x7f800000u;
      top = fmaxf(top, fabsf(v[e]));
    }
  }
  finite = __all_sync(0xffffffffu, finite);
  top = nb_warp_max(top);
  const bool whole = finite && (top == 0.0f || top >= 1e-27f);      // 2^-90
  if (lane == 0) (is_w ? w_flags : x_flags)[r] = whole ? 0 : 1;
  for (int k = lane; k < K / 4; k += 32) {
    const float4 f = src[k];
    const float v[4] = {f.x, f.y, f.z, f.w};
    bf16 p[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split3(v[e], whole, p[0][e], p[1][e], p[2][e]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint2*>(dst + (size_t)i * rows * K + k * 4) = *reinterpret_cast<const uint2*>(p[i]);
  }
}

template <typename TOut>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const float* X, const float* __restrict__ W, const int* x_flags, const int* w_flags,
                   const float* __restrict__ bias, const float* residual, TOut* out, int M, int N, int K,
                   int act, int tiles_n, int* err_word) {
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;          // swizzle atoms are 1024 bytes
  float* tile_s = reinterpret_cast<float*>(smem_dyn + (base - raw));       // [BM][OLD], over the ring
  const uint32_t bars = base + STAGES * BLOCK_BYTES;
  auto full = [&](int s, int p) { return bars + 8u * (s * 3 + p); };       // one a piece
  auto empty = [&](int s) { return bars + 8u * (3 * STAGES + s); };
  auto acc_full = [&](int b) { return bars + 8u * (4 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (4 * STAGES + 2 + b); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_dyn + (bars - raw) + 8 * (4 * STAGES + 4));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  const int blocks = (K + BK - 1) / BK, chunks = (blocks + CHUNK - 1) / CHUNK;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      for (int p = 0; p < 3; ++p) mbar_init(full(s, p), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(acc_full(b), 1);
      mbar_init(acc_empty(b), EPI);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)),
                 "r"(512u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  tc05_fence_before();
  __syncthreads();
  tc05_fence_after();
  const uint32_t tmem = *tmem_slot;          // columns 0, 128: large terms, in turn; 256: small terms
  nb_grid_dependency_wait();
  nb_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < blocks; ++kb) {
        const int s = kb % STAGES;
        if (!mbar_wait(empty(s), (((uint32_t)(kb / STAGES)) & 1u) ^ 1u, abort_flag)) break;
        const uint32_t st = base + (uint32_t)(s * BLOCK_BYTES);
        for (int p = 0; p < 3; ++p) {        // a box beyond its piece's rows brings rows nobody stores
          mbar_expect_tx(full(s, p), 2u * PIECE);
          tma_load_2d(st + (uint32_t)(p * PIECE), &map_x, kb * BK, p * M + m0, full(s, p));
          tma_load_2d(st + (uint32_t)((3 + p) * PIECE), &map_w, kb * BK, p * N + n0, full(s, p));
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = instr_desc_bf16(BM, BN);
      bool ok = true;
      for (int kb = 0; kb < blocks && ok; ++kb) {
        const int s = kb % STAGES, c = kb / CHUNK, b = c & 1;
        const uint32_t phase = (uint32_t)(kb / STAGES) & 1u;
        const bool first = kb % CHUNK == 0;
        if (first) {
          ok = mbar_wait(acc_empty(b), ((uint32_t)(c >> 1) & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          tc05_fence_after();
        }
        const uint32_t st = base + (uint32_t)(s * BLOCK_BYTES);
        auto product = [&](int px, int pw, uint32_t d, bool fresh) {
          const uint64_t da = smem_desc_sw128(st + (uint32_t)(px * PIECE));
          const uint64_t db = smem_desc_sw128(st + (uint32_t)((3 + pw) * PIECE));
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            tc05_mma_bf16(d, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, (fresh && k == 0) ? 0u : 1u);
        };
        const uint32_t small = tmem + 256u;
        ok = mbar_wait(full(s, 0), phase, abort_flag);
        if (!ok) break;
        tc05_fence_after();
        product(0, 0, tmem + (uint32_t)b * 128u, first);
        ok = mbar_wait(full(s, 1), phase, abort_flag);
        if (!ok) break;
        tc05_fence_after();
        product(0, 1, small, kb == 0);
        product(1, 0, small, false);
        product(1, 1, small, false);
        ok = mbar_wait(full(s, 2), phase, abort_flag);
        if (!ok) break;
        tc05_fence_after();
        product(0, 2, small, false);
        product(2, 0, small, false);
        tc05_commit(empty(s));
        // (the last of these also says that the small terms are complete)
        if (kb % CHUNK == CHUNK - 1 || kb + 1 == blocks) tc05_commit(acc_full(b));
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;       // 32 rows, 64 columns
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 64);
    float f[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) f[j] = 0.0f;
    bool ok = true;
    for (int c = 0; c < chunks && ok; ++c) {
      const int b = c & 1;
      ok = __shfl_sync(0xffffffffu, (int)mbar_wait(acc_full(b), (uint32_t)(c >> 1) & 1u, abort_flag), 0) != 0;
      if (!ok) break;
      tc05_fence_after();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t v[32];
        tc05_ld_32x32b_x32(lanes + (uint32_t)(b * 128 + q * 32), v);
        tc05_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) f[q * 32 + j] += __uint_as_float(v[j]);
      }
      tc05_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_empty(b)) : "memory");
    }
    if (ok) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t v[32];
        tc05_ld_32x32b_x32(lanes + (uint32_t)(256 + q * 32), v);
        tc05_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) f[q * 32 + j] += __uint_as_float(v[j]);
      }
      // all MMAs are done: the ring is free
      float* row = tile_s + (size_t)(quarter * 32 + lane) * OLD + half * 64;
#pragma unroll
      for (int j = 0; j < 64; j += 4)
        *reinterpret_cast<float4*>(row + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
    }
  }
  tc05_fence_before();
  __syncthreads();
  const bool aborted = *abort_flag != 0;
  if (!aborted && warp >= 2) {
    // a warp a row at a time: four columns a lane
    const bool vec = N % 4 == 0 && (uintptr_t)out % (4 * sizeof(TOut)) == 0 && (uintptr_t)residual % 16 == 0;
    const int n = n0 + lane * 4;
    float b4[4];
    bool odd_w = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      b4[j] = (bias != nullptr && n + j < N) ? __ldg(bias + n + j) : 0.0f;
      odd_w = odd_w || (n + j < N && w_flags[n + j] != 0);
    }
#pragma unroll 2
    for (int i = warp - 2; i < BM; i += EPI) {
      const int m = m0 + i;
      if (m >= M) break;
      if (n >= N) continue;
      const float4 t = *reinterpret_cast<const float4*>(tile_s + (size_t)i * OLD + lane * 4);
      float y[4] = {t.x, t.y, t.z, t.w}, r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      const size_t o = (size_t)m * N + n;
      if (residual != nullptr) {
        if (vec) {
          const float4 q = *reinterpret_cast<const float4*>(residual + o);
          r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N) r[j] = residual[o + j];
        }
      }
      if (odd_w || x_flags[m] != 0) {          // rows that could not be split
        const bool odd_x = x_flags[m] != 0;
#pragma unroll 1
        for (int j = 0; j < 4 && n + j < N; ++j) {
          if (!odd_x && w_flags[n + j] == 0) continue;
          float a = 0.0f;
          for (int k = 0; k < K; ++k) a = fmaf(X[(size_t)m * K + k], W[(size_t)(n + j) * K + k], a);
          if (j == 0) y[0] = a; else if (j == 1) y[1] = a; else if (j == 2) y[2] = a; else y[3] = a;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] += b4[j];
      if (act != NB_ACT_NONE) {
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
          const float z = j == 0 ? y[0] : j == 1 ? y[1] : j == 2 ? y[2] : y[3];
          const float g = nb_apply_act(z, act);
          if (j == 0) y[0] = g; else if (j == 1) y[1] = g; else if (j == 2) y[2] = g; else y[3] = g;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) y[j] += r[j];
      if (vec) {
        if constexpr (sizeof(TOut) == 4) {
          *reinterpret_cast<float4*>(out + o) = make_float4(y[0], y[1], y[2], y[3]);
        } else {
          uint2 u;
          __nv_bfloat162* hh = reinterpret_cast<__nv_bfloat162*>(&u);
          hh[0] = __floats2bfloat162_rn(y[0], y[1]);
          hh[1] = __floats2bfloat162_rn(y[2], y[3]);
          *reinterpret_cast<uint2*>(out + o) = u;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < N) out[o + j] = nb_from_f32<TOut>(y[j]);
      }
    }
  }
  if (aborted) {
    if (tid == 0) {
      nb_report_timeout(err_word);
      // let copies that are still in flight land before the shared memory goes away
      const long long t0 = clock64();
      while (clock64() - t0 < 4000000LL) {}
    }
    __syncthreads();
  }
  if (warp == 1) {
    tc05_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
  }
}

long long align256(long long n) { return (n + 255) & ~255LL; }

template <typename TOut>
int launch(const float* X, const float* W, const float* bias, const float* residual, void* out, int M,
           int N, int K, int act, unsigned char* scratch, cudaStream_t stream) {
  bf16* xp = (bf16*)scratch;
  bf16* wp = (bf16*)(scratch + align256(6LL * M * K));
  int* x_flags = (int*)(scratch + align256(6LL * M * K) + align256(6LL * N * K));
  int* w_flags = x_flags + M;
  CUtensorMap mx, mw;
  int rc = make_map(&mx, xp, 3LL * M, K, BM, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  rc = make_map(&mw, wp, 3LL * N, K, BN, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  auto kern = gemm_f32_tc_kernel<TOut>;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    configured = true;
  }
  NB_CUDA(nb_launch(split_kernel, dim3((unsigned)((M + N + 7) / 8)), dim3(256), 0, stream, X, W, xp, wp, x_flags,
                    w_flags, M, N, K));
  const int tiles_n = (N + BN - 1) / BN;
  int* w = nb_error_words();
  NB_CUDA(nb_launch(kern, dim3((unsigned)(tiles_n * ((M + BM - 1) / BM))), dim3(THREADS), (size_t)SMEM, stream,
                    mx, mw, X, W, x_flags, w_flags, bias, residual, (TOut*)out, M, N, K, act, tiles_n,
                    w ? w + NB_ERRW_GEMM_F32_TC : nullptr));
  return 0;
}

}  // namespace

// 1 if this kernel takes the product.
NB_EXPORT int nb_gemm_f32_tc_supported(int M, int N, int K) {
  return M >= 1 && N >= 1 && K >= 8 && K % 8 == 0 && (long long)M + N < (1 << 28) ? 1 : 0;
}

// 1 where it is faster than the multiply-adds of gemm_f32.cu, by what the two take (us): this one
// 1.7 a block of K and wave of tiles, the pieces' bytes at 4 TB/s, and 4; the other 10 and the
// product at 30 TFLOP/s.  Measured, this kernel and the other: 2024x2304x768 58 and 177,
// 2024x3072x768 86 and 258, 2024x768x3072 99 and 323, 1000x768x768 27 and 49, 333x2304x768 29 and 49,
// 333x768x768 26 and 26, 333x768x3072 74 and 70, 200x3072x768 30 and 48, 128x2304x768 28 and 27,
// 128x768x3072 73 and 30.
NB_EXPORT int nb_gemm_f32_tc_preferred(int M, int N, int K) {
  if (!nb_gemm_f32_tc_supported(M, N, K) || M < 65) return 0;
  const double tiles = (double)((M + BM - 1) / BM) * ((N + BN - 1) / BN), blocks = (K + BK - 1) / BK;
  const double waves = (double)(long long)((tiles + 147.0) / 148.0);
  const double here = waves * blocks * 1.7 + ((double)M + N) * K * 10.0 / 4e6 + 4.0;
  return here < 10.0 + 2.0 * M * N * K / 30e6 ? 1 : 0;
}

// Bytes of scratch memory of nb_gemm_f32_tc (256-byte aligned).
NB_EXPORT long long nb_gemm_f32_tc_scratch(int M, int N, int K) {
  return align256(6LL * M * K) + align256(6LL * N * K) + 4LL * (M + N);
}

NB_EXPORT int nb_gemm_f32_tc_set_wait_budget(long long cycles) { return set_wait_budget(cycles); }

// X, W fp32.  `residual` may be `out` (fp32): every element is read and written by the same thread.
NB_EXPORT int nb_gemm_f32_tc(const void* X, const void* W, const float* bias, const float* residual, void* out,
                             int out_dtype, int M, int N, int K, int act, void* scratch, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  NB_REQUIRE(nb_gemm_f32_tc_supported(M, N, K), NB_ERR_UNSUPPORTED,
             "gemm_f32_tc: needs a width that is a multiple of 8 (M=%d N=%d K=%d)", M, N, K);
  NB_REQUIRE((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0 && (uintptr_t)scratch % 256 == 0, NB_ERR_UNSUPPORTED,
             "gemm_f32_tc: operands must be 16-byte aligned, scratch 256");
  int rc;
  if (out_dtype == NB_F32)
    rc = launch<float>((const float*)X, (const float*)W, bias, residual, out, M, N, K, act, (unsigned char*)scratch, stream);
  else if (out_dtype == NB_BF16)
    rc = launch<bf16>((const float*)X, (const float*)W, bias, residual, out, M, N, K, act, (unsigned char*)scratch, stream);
  else
    NB_REQUIRE(false, NB_ERR_BAD_ARG, "gemm_f32_tc: unknown output type %d", out_dtype);
  if (rc) return rc;
  NB_CHECK_LAUNCH("gemm_f32_tc");
  return 0;
}
