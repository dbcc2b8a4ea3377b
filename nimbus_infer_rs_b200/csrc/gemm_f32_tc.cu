// Matrix product of fp32 rows with fp32 weights on the tensor cores, out[M,N] = act(X W^T + bias)
// (+ residual), no further from 64 bits than fp32 multiply-adds (figures, and the exception, below): the
// prompts of the true 32-bit path.
//
// The multiply-adds of the CUDA cores bound such a product at some 40 TFLOP/s (gemm_f32.cu).  Every
// fp32 number is the sum of three bf16 numbers (the split of Henry, Tang and Heinecke, "Leveraging the
// bfloat16 artificial intelligence datatype for higher-precision computations", 2019), x = h + m + l,
// each the nearest to what the ones before leave (so |m| <= 2^-8 and |l| <= 2^-17 of the power of two
// below |x|), and
//   x w = hh' + (hm' + mh' + mm' + hl' + lh' + ml' + lm') + ll'
// All but the last term, which is at most 2^-34 of the product, is computed: eight products of bf16
// tiles by tcgen05, whose products are exact.  What is not exact is the tensor cores' accumulation: an
// instruction (16 of K) cuts its sum instead of rounding it, so that errors of one sign pile up in an
// accumulator that is left alone (over 6,400 numbers of one sign 8.0e-7 of the result, where
// multiply-adds have 0.9e-7).  So the large terms hh' are taken out of tensor memory every 32 of K, and
// the small ones, in which the same error counts 2^-8 as much or less, every 512; both are
// added up in registers, rounded, in runs of about sqrt(K / 64) blocks whose sums are added up in turn
// (one chain of K / 32 additions would round as often as the multiply-adds do).
//
// A pass of its own (split_kernel, a warp a row, four beyond 1,024 of K) writes the three pieces of the rows of X and of W
// into scratch memory, every time: nothing is kept from one call to the next.  Rows all of whose numbers
// are below 2^-30 are split times a power of two that brings the largest into [1, 2), and the result is
// multiplied back: their small terms would be subnormal, where every cut is of 2^-149 (both operands of
// 1e-19: 2.2e-7 of the result for 1.8e-7 of the multiply-adds at K = 768).  The pass also marks the
// rows that cannot be split: those with an infinity or NaN in them (infinity minus infinity) and those
// with a number above 2^50 (hh' of two such may be infinite where x w is not, and a sum of
// pieces NaN where that of the products is infinite); their results are computed by plain
// multiply-adds in the epilogue.
//
// Error against 64 bits (2-norm over 330 x 3264 results) at K = 128, 768 and 6,400, and in brackets that of
// the multiply-adds of gemm_f32.cu, which leave K whole over so many tiles, in units of 1e-8: normal rows
// 6.2, 8.1, 11.7 (20, 35, 101); numbers of one sign 5.8, 6.1, 6.7 (16, 21, 59); one term a row 10^4 times
// the others 8.9, 10.3, 13.1 (21, 35, 106); one channel 300 times the others 9.8, 11.6, 13.0 (24, 41, 116);
// one term a row 2.5 (2.5).  It is larger for four terms a row over a long K, 2.7, 4.0, 4.6 (4.0, 4.2, 4.2):
// seven roundings against four; and, over a short one, where the terms of both operands are spread
// over 2^80, 6.0, 7.7, 10.9 (5.1, 8.6, 22.7): a cut of up to one unit in the last place against half a one.
// (Cut in parts, over so few tiles that they are the faster ones, multiply-adds come nearer: numbers
// of one sign at K = 128 in two parts 5.4.)
//
// A CTA takes a tile of 128 rows and 128 columns, or 96 where that takes no more waves of tiles.  What
// bounds a block of 64 of K is the shared memory that its instructions read their operands from and its
// loads write to, and the instructions' number: W's neighbouring pieces lie behind one another and are
// taken as one operand of twice the width, hm' beside hl', mh' beside mm', lh' beside lm', into two halves
// of the small terms' accumulator, which are added up when they are taken out: 20 instructions a block
// that read 208 KB, where one at a time took 32 and 256 KB (us, split_kernel included, now and then:
// 2024x2304x768 57 and 63, 2024x3072x768 82 and 88; with 96 columns 2024x768x768 28 and 35, 2024x768x3072 85 and
// 115).  (With six products, ml' and lm' left out, and the large terms taken out every 128 of K, one piece
// at a time: 2024x2304x768 55, 2024x768x3072 94.  Large terms taken out every 16 of K by eight warps:
// 2024x768x3072 151.)
// Warp 0 brings the pieces of 64 columns of K by TMA (six 128 x 64
// boxes a block, two blocks in flight), warp 1 issues the MMAs, sixteen or twelve warps take the
// accumulators (two for the large terms, one in two halves for the small) out and finish the tile through shared
// memory.  Every wait has a clock budget.
//
// Reference analogue: Mat::gemm_into (src/model.rs:88-133).
#include <cmath>

#include "gemm_f32.cuh"
#include "tc05_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BK = 64;
constexpr int STAGES = 2;                   // blocks of K in flight
constexpr int SMALL = 8;                    // blocks of K whose small terms are added up in one place

template <int BN>                           // columns of a tile
struct Tile {
  static constexpr int XPIECE = BM * BK * 2, WPIECE = BN * BK * 2;        // bytes of the boxes
  static constexpr int BLOCK_BYTES = 3 * (XPIECE + WPIECE);               // X's three pieces, W's three pieces
  static constexpr int EPI = 4 * (BN / 32);                               // warps of the epilogue
  static constexpr int THREADS = 64 + 32 * EPI;
  static constexpr int OLD = BN + 4;                                      // floats between rows of the finished tile
  static constexpr int SMEM = STAGES * BLOCK_BYTES + 1024 + 256;
  static_assert(BN % 32 == 0 && BN <= 128, "large and small accumulators fill the tensor memory");
  static_assert(BM * OLD * 4 <= STAGES * BLOCK_BYTES, "the finished tile goes where the ring was");
};

__device__ __forceinline__ void split3(float x, bf16& h, bf16& m, bf16& l) {
  h = __float2bfloat16_rn(x);
  const float r = x - __bfloat162float(h);                      // exact
  m = __float2bfloat16_rn(r);
  l = __float2bfloat16_rn(r - __bfloat162float(m));             // exact
}

// Sixteen columns of this warp's 32 rows of tensor memory.
__device__ __forceinline__ void tc05_ld_32x32b_x16(uint32_t taddr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15])
      : "r"(taddr)
      : "memory");
}

// Rows 0 .. M-1 of X and 0 .. N-1 of W, WPR warps each, into pieces [3][rows][K]; scale[row] is what
// a result of the row is to be multiplied by, 0 for rows that cannot be split (their pieces are zeros).
// K % 4 == 0.  Bound by its bytes and by how many of them are on their way: a row of up to HELD
// pieces of four numbers a thread is read once, all of it asked for together, and kept.
constexpr int HELD = 8;
template <int WPR>
__global__ void __launch_bounds__(256)
split_kernel(const float* X, const float* __restrict__ W, bf16* xp, bf16* wp, float* x_scale,
             float* w_scale, int M, int N, int K) {
  constexpr int TPR = 32 * WPR, ROWS = 8 / WPR;
  __shared__ float s_top[8];
  nb_grid_dependency_wait();
  nb_launch_dependents();
  const int warp = threadIdx.x >> 5, row = blockIdx.x * ROWS + warp / WPR, t = threadIdx.x % TPR;
  const bool live = row < M + N, is_w = row >= M;
  const int r = is_w ? row - M : row, rows = is_w ? N : M;
  const float4* src = reinterpret_cast<const float4*>((is_w ? W : X) + (size_t)r * K);
  bf16* dst = (is_w ? wp : xp) + (size_t)r * K;
  const int n = live ? K / 4 : 0;
  float4 f[HELD];
  // the largest magnitude of the row; infinity where one of its numbers is not finite
  float top = 0.0f;
  auto see = [&](const float4& q) {
    const float v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 4; ++e)
      top = fmaxf(top, (__float_as_uint(v[e]) & 0x7f800000u) != 0x7f800000u ? fabsf(v[e]) : INFINITY);
  };
#pragma unroll
  for (int i = 0; i < HELD; ++i)
    f[i] = t + i * TPR < n ? src[t + i * TPR] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < HELD; ++i) see(f[i]);
  for (int k = t + HELD * TPR; k < n; k += TPR) see(src[k]);
  top = nb_warp_max(top);
  if constexpr (WPR > 1) {
    if ((threadIdx.x & 31) == 0) s_top[warp] = top;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < WPR; ++i) top = fmaxf(top, s_top[warp / WPR * WPR + i]);
  }
  const bool whole = top <= 0x1p50f;
  const int up = whole && top > 0.0f && top < 0x1p-30f ? -ilogbf(top) : 0;
  if (live && t == 0) (is_w ? w_scale : x_scale)[r] = whole ? ldexpf(1.0f, -up) : 0.0f;
  auto put = [&](int k, const float4& q) {
    float v[4] = {q.x, q.y, q.z, q.w};
    if (up != 0 || !whole) {
#pragma unroll
      for (int e = 0; e < 4; ++e) v[e] = whole ? ldexpf(v[e], up) : 0.0f;
    }
    bf16 p[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split3(v[e], p[0][e], p[1][e], p[2][e]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
      *reinterpret_cast<uint2*>(dst + (size_t)i * rows * K + k * 4) = *reinterpret_cast<const uint2*>(p[i]);
  };
#pragma unroll
  for (int i = 0; i < HELD; ++i)
    if (t + i * TPR < n) put(t + i * TPR, f[i]);
  for (int k = t + HELD * TPR; k < n; k += TPR) put(k, src[k]);
}

template <int BN, typename TOut>
__global__ void __launch_bounds__(Tile<BN>::THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                   const float* X, const float* __restrict__ W, const float* x_scale, const float* w_scale,
                   const float* __restrict__ bias, const float* residual, TOut* out, int ld, int M, int N,
                   int K, int act, int tiles_n, int run, int* err_word) {
  constexpr int XPIECE = Tile<BN>::XPIECE, WPIECE = Tile<BN>::WPIECE, BLOCK_BYTES = Tile<BN>::BLOCK_BYTES;
  constexpr int EPI = Tile<BN>::EPI, OLD = Tile<BN>::OLD;
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;          // swizzle atoms are 1024 bytes
  float* tile_s = reinterpret_cast<float*>(smem_dyn + (base - raw));       // [BM][OLD], over the ring
  const uint32_t bars = base + STAGES * BLOCK_BYTES;
  auto full = [&](int s, int p) { return bars + 8u * (s * 3 + p); };       // one a piece
  auto empty = [&](int s) { return bars + 8u * (3 * STAGES + s); };
  // accumulators 0 and 1: large terms, 2: small terms, in two halves
  auto acc_full = [&](int b) { return bars + 8u * (4 * STAGES + b); };
  auto acc_empty = [&](int b) { return bars + 8u * (4 * STAGES + 3 + b); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem_dyn + (bars - raw) + 8 * (4 * STAGES + 6));
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = (int)(blockIdx.x / tiles_n) * BM, n0 = (int)(blockIdx.x % tiles_n) * BN;
  const int blocks = (K + BK - 1) / BK;

  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      for (int p = 0; p < 3; ++p) mbar_init(full(s, p), 1);
      mbar_init(empty(s), 1);
    }
    for (int b = 0; b < 3; ++b) {
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
  const uint32_t tmem = *tmem_slot;          // accumulator b in columns 128 b ...
  nb_grid_dependency_wait();
  nb_launch_dependents();

  if (warp == 0) {
    if (lane == 0) {
      for (int kb = 0; kb < blocks; ++kb) {
        const int s = kb % STAGES;
        if (!mbar_wait(empty(s), (((uint32_t)(kb / STAGES)) & 1u) ^ 1u, abort_flag)) break;
        const uint32_t st = base + (uint32_t)(s * BLOCK_BYTES);
        for (int p = 0; p < 3; ++p) {        // a box beyond its piece's rows brings rows nobody stores
          mbar_expect_tx(full(s, p), (uint32_t)(XPIECE + WPIECE));
          tma_load_2d(st + (uint32_t)(p * XPIECE), &map_x, kb * BK, p * M + m0, full(s, p));
          tma_load_2d(st + (uint32_t)(3 * XPIECE + p * WPIECE), &map_w, kb * BK, p * N + n0, full(s, p));
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t one = instr_desc_bf16(BM, BN), two = instr_desc_bf16(BM, 2 * BN);
      bool ok = true;
      for (int kb = 0; kb < blocks; ++kb) {
        const int s = kb % STAGES, g = kb / SMALL;
        const bool first = kb % SMALL == 0, last = kb % SMALL == SMALL - 1 || kb + 1 == blocks;
        const uint32_t phase = (uint32_t)(kb / STAGES) & 1u;
        const uint32_t st = base + (uint32_t)(s * BLOCK_BYTES);
        // 16 of K, from `k` of the block on: X's piece px times W's piece pw, or times that and the next
        // one, which follows it in shared memory as 2 BN rows of one operand: the results lie side by side
        auto product = [&](uint32_t idesc, int px, int pw, int k, int col, bool fresh) {
          const uint64_t da = smem_desc_sw128(st + (uint32_t)(px * XPIECE));
          const uint64_t db = smem_desc_sw128(st + (uint32_t)(3 * XPIECE + pw * WPIECE));
          tc05_mma_bf16(tmem + (uint32_t)col, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc,
                        fresh ? 0u : 1u);
        };
        // the large terms, half a block at a time, for the epilogue to take out
        ok = mbar_wait(full(s, 0), phase, abort_flag);
        for (int b = 0; b < 2 && ok; ++b) {
          ok = mbar_wait(acc_empty(b), ((uint32_t)kb & 1u) ^ 1u, abort_flag);
          if (!ok) break;
          tc05_fence_after();
          product(one, 0, 0, 2 * b, b * 128, true);
          product(one, 0, 0, 2 * b + 1, b * 128, false);
          tc05_commit(acc_full(b));
        }
        if (first && ok) ok = mbar_wait(acc_empty(2), ((uint32_t)g & 1u) ^ 1u, abort_flag);
        ok = ok && mbar_wait(full(s, 1), phase, abort_flag);
        if (!ok) break;
        tc05_fence_after();
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) product(two, 1, 0, k, 256, first && k == 0);      // mh' | mm'
        ok = mbar_wait(full(s, 2), phase, abort_flag);
        if (!ok) break;
        tc05_fence_after();
#pragma unroll
        for (int k = 0; k < BK / 16; ++k) {
          product(two, 0, 1, k, 256, false);         // hm' | hl'
          product(two, 2, 0, k, 256, false);         // lh' | lm'
          product(one, 1, 2, k, 256, false);         // ml'
        }
        tc05_commit(empty(s));
        if (last) tc05_commit(acc_full(2));
      }
    }
    __syncwarp();
  } else {
    const int quarter = warp & 3, part = (warp - 2) >> 2;       // 32 rows, 32 columns
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * 32);
    // u: the sums of up to `run` blocks, f: the runs' sums
    float f[32], u[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = u[j] = 0.0f;
    auto take_out = [&](int b, uint32_t parity) {
      if (!__all_sync(0xffffffffu, mbar_wait(acc_full(b), parity, abort_flag))) return false;
      tc05_fence_after();
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        uint32_t v[16];
        tc05_ld_32x32b_x16(lanes + (uint32_t)(b * 128 + q * 16), v);
        if (b == 2) {      // the two halves are added up first: that rounds 2^-8 of the result
          uint32_t w[16];
          tc05_ld_32x32b_x16(lanes + (uint32_t)(b * 128 + BN + q * 16), w);
          tc05_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
        }
        tc05_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) u[q * 16 + j] += __uint_as_float(v[j]);
      }
      tc05_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(acc_empty(b)) : "memory");
      return true;
    };
    bool ok = true;
    for (int kb = 0, left = run; kb < blocks && ok; ++kb) {
      const int g = kb / SMALL;
      ok = take_out(0, (uint32_t)kb & 1u) && take_out(1, (uint32_t)kb & 1u);
      if (ok && (kb % SMALL == SMALL - 1 || kb + 1 == blocks)) ok = take_out(2, (uint32_t)g & 1u);
      if (--left == 0 || kb + 1 == blocks) {
        left = run;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          f[j] += u[j];
          u[j] = 0.0f;
        }
      }
    }
    if (ok) {
      // all MMAs are done: the ring is free
      float* row = tile_s + (size_t)(quarter * 32 + lane) * OLD + part * 32;
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        *reinterpret_cast<float4*>(row + j) = make_float4(f[j], f[j + 1], f[j + 2], f[j + 3]);
    }
  }
  tc05_fence_before();
  __syncthreads();
  const bool aborted = *abort_flag != 0;
  if (!aborted && warp >= 2) {
    // a warp a row at a time: four columns a lane (of a narrower tile the first lanes only)
    const bool vec = ld % 4 == 0 && (uintptr_t)out % (4 * sizeof(TOut)) == 0 && (uintptr_t)residual % 16 == 0;
    const int n = lane * 4 < BN ? n0 + lane * 4 : N;
    float b4[4], ws[4];
    unsigned odd_w = 0;               // the lanes with a column that could not be split
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      b4[j] = (bias != nullptr && n + j < N) ? __ldg(bias + n + j) : 0.0f;
      ws[j] = n + j < N ? w_scale[n + j] : 1.0f;
      odd_w |= __ballot_sync(0xffffffffu, ws[j] == 0.0f);
    }
    const unsigned all = __ballot_sync(0xffffffffu, n < N);
#pragma unroll 2
    for (int i = warp - 2; i < BM; i += EPI) {
      const int m = m0 + i;
      if (m >= M) break;
      const float4 t = *reinterpret_cast<const float4*>(tile_s + (size_t)i * OLD + (lane * 4 < BN ? lane * 4 : 0));
      const float xs = x_scale[m];
      float y[4] = {t.x * xs * ws[0], t.y * xs * ws[1], t.z * xs * ws[2], t.w * xs * ws[3]}, r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      // what could not be split, four columns at a time with the warp's lanes along K (1024x768x768 us:
      // 36 without such rows, 74 with one, 415 with nothing else, as a prompt whose activations
      // have overflowed; with a thread a result that walked K alone 130 and 6,860)
      for (unsigned odd = xs == 0.0f ? all : odd_w; odd != 0; odd &= odd - 1) {
        const int q = __ffs(odd) - 1, nq = n0 + q * 4;
        const float4* xr = reinterpret_cast<const float4*>(X + (size_t)m * K);
        const float4* wr[4];                   // (beyond the last column: that one again)
#pragma unroll
        for (int j = 0; j < 4; ++j) wr[j] = reinterpret_cast<const float4*>(W + (size_t)min(nq + j, N - 1) * K);
        float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 2
        for (int k = lane; k < K / 4; k += 32) {
          const float4 x = xr[k];
          float4 w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) w[j] = wr[j][k];
#pragma unroll
          for (int j = 0; j < 4; ++j)
            a[j] = fmaf(x.w, w[j].w, fmaf(x.z, w[j].z, fmaf(x.y, w[j].y, fmaf(x.x, w[j].x, a[j]))));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          a[j] = nb_warp_sum(a[j]);
          if (lane == q && (xs == 0.0f || ws[j] == 0.0f)) y[j] = a[j];
        }
      }
      if (n >= N) continue;
      const size_t o = (size_t)m * ld + n;
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

// The rows and the columns that one pair of launches takes: their pieces stay within PIECES_MAX
// bytes of scratch memory each, however large the product is (128 rows of them at least).  Rows
// in equal parts; columns in parts of which the last wave of tiles leaves the fewest SMs idle.
// With 96 MB a part of the widest head (1,600 numbers of K) has a CTA for half the SMs and one of 768 for
// all of them: 66x50257x768 144 us whole, 155 cut so, 182 cut to 64 MB; 997x50257x768 694, 709, 704.
constexpr long long PIECES_MAX = 96LL << 20;
struct Cut { int rows, cols; };
Cut cut_of(int M, int N, int K) {
  constexpr int BN = 128;
  const long long sms = nb_device_sms(), tm = (M + BM - 1) / BM, tn = (N + BN - 1) / BN;
  const long long most = PIECES_MAX / (6LL * K * BM) > 1 ? PIECES_MAX / (6LL * K * BM) : 1;
  const long long parts = (tm + most - 1) / most, rows = (tm + parts - 1) / parts;
  long long cols = tn;
  if (tn > most) {
    long long best = 0;
    for (long long c = most; c > most / 2; --c) {
      const long long waves = tn / c * ((rows * c + sms - 1) / sms) + (rows * (tn % c) + sms - 1) / sms;
      if (best == 0 || waves < best) { best = waves; cols = c; }
    }
  }
  Cut cut;
  cut.rows = (int)(rows * BM < M ? rows * BM : M);
  cut.cols = (int)(cols * BN < N ? cols * BN : N);
  return cut;
}

template <int BN, typename TOut>
int launch_tiles(const float* X, const float* W, const bf16* xp, const bf16* wp, const float* x_scale, const float* w_scale,
                 const float* bias, const float* residual, TOut* out, int ld, int M, int N, int K, int act,
                 cudaStream_t stream) {
  auto kern = gemm_f32_tc_kernel<BN, TOut>;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<BN>::SMEM));
    configured = true;
  }
  CUtensorMap mx, mw;
  int rc = make_map(&mx, xp, 3LL * M, K, BM, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  rc = make_map(&mw, wp, 3LL * N, K, BN, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  int run = 1;                      // blocks of a run: as many as there are runs
  while (run * run < (K + BK - 1) / BK) ++run;
  int* w = nb_error_words();
  const int tiles_n = (N + BN - 1) / BN;
  NB_CUDA(nb_launch(kern, dim3((unsigned)(tiles_n * ((M + BM - 1) / BM))), dim3(Tile<BN>::THREADS),
                    (size_t)Tile<BN>::SMEM, stream, mx, mw, X, W, x_scale, w_scale, bias, residual, out, ld, M, N, K,
                    act, tiles_n, run, w ? w + NB_ERRW_GEMM_F32_TC : nullptr));
  return 0;
}

// Columns of a tile: the width with the least waves of tiles x time of a block of K in it.
int g_force_bn = 0;
double block_us(int bn) { return bn == 96 ? 1.53 : 1.65; }
double waves(long long M, long long N, int bn) {
  return ceil((double)((M + BM - 1) / BM) * (double)((N + bn - 1) / bn) / nb_device_sms());
}
int tile_width(int M, int N) {
  if (g_force_bn) return g_force_bn;
  return waves(M, N, 96) * block_us(96) < waves(M, N, 128) * block_us(128) ? 96 : 128;
}

template <typename TOut>
int launch(const float* X, const float* W, const float* bias, const float* residual, void* out, int M,
           int N, int K, int act, unsigned char* scratch, cudaStream_t stream) {
  const Cut cut = cut_of(M, N, K);
  bf16* xp = (bf16*)scratch;
  bf16* wp = (bf16*)(scratch + align256(6LL * cut.rows * K));
  float* x_scale = (float*)(scratch + align256(6LL * cut.rows * K) + align256(6LL * cut.cols * K));
  float* w_scale = x_scale + cut.rows;
  for (int n0 = 0; n0 < N; n0 += cut.cols) {
    const int nc = N - n0 < cut.cols ? N - n0 : cut.cols;
    for (int m0 = 0; m0 < M; m0 += cut.rows) {
      const int mc = M - m0 < cut.rows ? M - m0 : cut.rows;
      const float* Xc = X + (size_t)m0 * K;
      const float* Wc = W + (size_t)n0 * K;
      const size_t o = (size_t)m0 * N + n0;
      // (pieces that the launch before made are there still)
      const int xs = n0 == 0 || cut.rows < M ? mc : 0, ws = m0 == 0 ? nc : 0;
      if (K <= 4 * 32 * HELD)         // a warp holds the row
        NB_CUDA(nb_launch(split_kernel<1>, dim3((unsigned)((xs + ws + 7) / 8)), dim3(256), 0, stream, Xc, Wc, xp, wp,
                          x_scale, w_scale, xs, ws, K));
      else
        NB_CUDA(nb_launch(split_kernel<4>, dim3((unsigned)((xs + ws + 1) / 2)), dim3(256), 0, stream, Xc, Wc, xp, wp,
                          x_scale, w_scale, xs, ws, K));
      const float* bc = bias == nullptr ? nullptr : bias + n0;
      const float* rc = residual == nullptr ? nullptr : residual + o;
      const int e = tile_width(mc, nc) == 96
                        ? launch_tiles<96>(Xc, Wc, xp, wp, x_scale, w_scale, bc, rc, (TOut*)out + o, N, mc, nc, K, act, stream)
                        : launch_tiles<128>(Xc, Wc, xp, wp, x_scale, w_scale, bc, rc, (TOut*)out + o, N, mc, nc, K, act, stream);
      if (e) return e;
    }
  }
  return 0;
}

}  // namespace

// 1 if this kernel takes the product.
NB_EXPORT int nb_gemm_f32_tc_supported(int M, int N, int K) {
  return M >= 1 && N >= 1 && K >= 8 && K % 8 == 0 && (long long)M + N < (1 << 28) ? 1 : 0;
}

// 1 where it is faster than the multiply-adds of gemm_f32.cu, by what the two take (us): this one 7 a
// wave of tiles and 1.65 a block of K in it, and the pieces' bytes at 4 TB/s; the other 6, and for a
// block of 16 of its part of K 1.03 up to 1.75 CTAs an SM, 1.8 up to 3.5, and beyond 0.46 a CTA and SM,
// or 0.62 where K is cut (clusters leave SMs out); where it leaves K of under 256 to gemm_simt.cu that
// one's 4 and 0.045 a number of K.  Measured, this kernel and the other:
// 2024x2304x768 57 and 173, 2024x3072x768 82 and 251, 2024x768x3072 84 and 320, 1000x768x768 26 and 49,
// 333x2304x768 27 and 49, 200x2304x768 26 and 40, 66x50257x768 138 and 244, 128x4800x1600 55 and 92,
// 512x768x3072 76 and 88; but 333x768x768 25 and 23.5, 100x2304x768 25 and 23.6, 256x768x3072 75 and 47,
// 128x768x3072 74 and 30.  (The line's constants are from before the tiles of 96 columns and rows split in one
// reading.  It leaves a few to the multiply-adds that are faster here now: 512x768x768 25.3 and 26.7,
// 997x512x512 19.9 and 21.8, 300x1600x1600 46 and 52, 300x1600x6400 161 and 191.)  Not below 128 of K, where gemm_simt.cu's tiles take as long as a wave here or
// less (512x768x64 6.8 and 9.5) and, with a step or two of 16, the one cut a step leaves more than the few
// roundings of multiply-adds (K = 8, one large term a row: 5.7e-8 against 4.8e-8).
NB_EXPORT int nb_gemm_f32_tc_preferred(int M, int N, int K) {
  if (!nb_gemm_f32_tc_supported(M, N, K) || M < 65 || K < 128) return 0;
  const double sms = nb_device_sms(), blocks = (K + BK - 1) / BK;
  const int bn = tile_width(M, N);
  const double here = waves(M, N, bn) * (7.0 + blocks * block_us(bn)) + ((double)M + N) * K * 10.0 / 4e6;
  const int cut = nb_gemm_f32_cut(M, N, K);
  const double small = (double)((M + 63) / 64) * ((N + 63) / 64) / sms;            // 64 x 64 tiles an SM
  if (cut == 0) return here < 4.0 + 0.045 * K * (small > 0.87 ? 1.15 * small : 1.0) ? 1 : 0;
  const double ctas = small * cut, block = ctas <= 1.75 ? 1.03 : ctas <= 3.5 ? 1.8 : (cut > 1 ? 0.62 : 0.46) * ctas;
  return here < 6.0 + ceil(K / (16.0 * cut)) * block ? 1 : 0;
}

// Bytes of scratch memory of nb_gemm_f32_tc (256-byte aligned): at most twice PIECES_MAX and a little
// (997x50257x768, the head over a text's places: 98 MB; whole, its pieces are 236).
NB_EXPORT long long nb_gemm_f32_tc_scratch(int M, int N, int K) {
  const Cut cut = cut_of(M, N, K);
  return align256(6LL * cut.rows * K) + align256(6LL * cut.cols * K) + 4LL * (cut.rows + cut.cols);
}

// How it cuts a product whose pieces would be larger (tests and reports): rows, columns.
NB_EXPORT void nb_gemm_f32_tc_cut(int M, int N, int K, int* out2) {
  const Cut cut = cut_of(M, N, K);
  out2[0] = cut.rows;
  out2[1] = cut.cols;
}

// Tuning and tests: columns of a tile (96, 128; 0 = choose).
NB_EXPORT int nb_gemm_f32_tc_force(int columns) {
  NB_REQUIRE(columns == 0 || columns == 96 || columns == 128, NB_ERR_BAD_ARG, "gemm_f32_tc: no tile of %d columns", columns);
  g_force_bn = columns;
  return 0;
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
