// Matrix product for 17 to 128 rows (a decode step of a larger batch, a short prompt):
// out[M,N] = act(X[M,K] * W[N,K]^T + bias) (+ residual), bf16 operands, fp32 accumulation.
//
// What bounds such a product is how many SMs take part and what each has to bring in: the
// 64- and 128-wide tiles of the tcgen05 kernels put a product of 768 columns on 6 to 12 CTAs, and
// one thread issues all of a CTA's instructions at some 80 clocks each.  Here a CTA takes
// all rows and 16 to 64 columns, K is cut among the CTAs of a cluster until the launch covers
// the SMs, and eight warps issue mma.sync side by side (the weights are the 16-row operand, the
// rows of X the 8-wide one), splitting the columns and, beyond that, K.  With so few rows the
// warp-level instructions keep up with the loads.
//
// One warp brings 64-column blocks of W and X into a ring of stages by TMA (128-byte swizzle); the
// weights of the first stages are asked for before the wait on the kernel in front.  The warps'
// sums meet in shared memory (where the ring was), those of a cluster's CTAs through distributed
// shared memory: each CTA finishes its share of the rows, adding in rank order.
//
// Every wait on an mbarrier has a clock budget; one that runs out raises the kernel's error
// word, all roles leave their loops, pass the same barriers and return.
//
// Reference analogue: Mat::gemm_into (src/model.rs:94-133).
#include "mma_common.cuh"
#include "tc05_common.cuh"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BK = 64;                // numbers of K in a block: 128 bytes
constexpr int WARPS = 8;              // that multiply; one more brings the operands in
constexpr int THREADS = WARPS * 32 + 32;
constexpr int MAX_STAGES = 16;
constexpr int MAX_SPLIT = 8;          // portable cluster size
constexpr int MAX_ROWS = 128;
constexpr int AHEAD = 2;              // 16-byte pieces of the residual a thread asks for ahead

struct MidShape {
  int wn;            // warps side by side along the columns: a CTA takes 16 * wn columns
  int split;         // CTAs of a cluster = runs of K
  int kb_per;        // blocks of K a CTA
  int stages, stage_bytes, smem;
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

// NT: 8-row tiles of X.  WN: see MidShape.
template <int NT, int WN, typename TOut>
__global__ void __launch_bounds__(THREADS, NT <= 8 ? 2 : 1)
gemm_mid_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                const float* __restrict__ bias, const float* residual, TOut* out, int M, int N, int K,
                int act, MidShape sh, bool vec, int* err_word) {
  constexpr int C = 16 * WN, WK = WARPS / WN, ROWS = NT * 8, LD = C + 4;
  extern __shared__ unsigned char smem_dyn[];
  const uint32_t raw = smem_u32(smem_dyn);
  const uint32_t base = (raw + 1023u) & ~1023u;          // swizzle atoms are 1024 bytes
  float* red = reinterpret_cast<float*>(smem_dyn + (base - raw));          // [WK][ROWS][LD], over the ring
  const uint32_t bars = base + (uint32_t)sh.smem;                          // full, empty
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem_dyn + (bars - raw) + 2 * MAX_STAGES * 8);
  auto full = [&](int s) { return bars + 8u * s; };
  auto empty = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % sh.split, n0 = (int)(blockIdx.x / sh.split) * C;
  const int blocks = (K + BK - 1) / BK;
  const int b_lo = min(blocks, rank * sh.kb_per), n_blocks = min(blocks, b_lo + sh.kb_per) - b_lo;

  if (tid == 0) {
    for (int s = 0; s < sh.stages; ++s) {
      mbar_init(full(s), 1);
      mbar_init(empty(s), WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  }
  __syncthreads();

  const int chunk = (M + sh.split - 1) / sh.split;           // rows a CTA of the cluster finishes
  const int m_lo = min(M, rank * chunk), m_hi = min(M, m_lo + chunk);
  constexpr int Q = C / 4;                                   // 16-byte pieces of a row's columns
  float4 ahead[AHEAD];

  if (warp == WARPS) {
    const int first = min(n_blocks, sh.stages);
    if (lane == 0) {
      for (int b = 0; b < first; ++b) {
        mbar_expect_tx(full(b), (uint32_t)sh.stage_bytes);
        tma_load_2d(base + (uint32_t)(b * sh.stage_bytes), &map_w, (b_lo + b) * BK, n0, full(b));
      }
    }
    nb_grid_dependency_wait();
    nb_launch_dependents();
    if (lane == 0) {
      for (int b = 0; b < first; ++b)
        tma_load_2d(base + (uint32_t)(b * sh.stage_bytes + C * 128), &map_x, (b_lo + b) * BK, 0, full(b));
      int s = 0;
      uint32_t phase = 0;
      for (int b = first; b < n_blocks; ++b) {
        if (!mbar_wait(empty(s), phase, abort_flag)) break;
        mbar_expect_tx(full(s), (uint32_t)sh.stage_bytes);
        tma_load_2d(base + (uint32_t)(s * sh.stage_bytes), &map_w, (b_lo + b) * BK, n0, full(s));
        tma_load_2d(base + (uint32_t)(s * sh.stage_bytes + C * 128), &map_x, (b_lo + b) * BK, 0, full(s));
        if (++s == sh.stages) { s = 0; phase ^= 1u; }
      }
    }
    __syncwarp();
    __syncthreads();
  } else {
    nb_grid_dependency_wait();
    nb_launch_dependents();
    // the residual of the outputs this thread finishes first
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int e = tid + i * THREADS, m = m_lo + e / Q, n = n0 + (e % Q) * 4;
      ahead[i] = (vec && residual != nullptr && m < m_hi && n < N)
                     ? *reinterpret_cast<const float4*>(residual + (size_t)m * N + n)
                     : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    const int wn = warp % WN, kp = warp / WN;
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    // this lane's rows and 16-byte pieces in the swizzled boxes (row & 7 is lane & 7 throughout)
    const uint32_t sw = lane & 7;
    const uint32_t a_row = (uint32_t)((wn * 16 + (lane & 15)) * 128), a_hi = lane >> 4;
    const uint32_t x_row = (uint32_t)(C * 128 + ((lane & 7) + ((lane >> 4) << 3)) * 128), x_hi = (lane >> 3) & 1;
    int s = 0;
    uint32_t phase = 0;
    for (int b = 0; b < n_blocks; ++b) {
      const bool ok = mbar_wait(full(s), phase, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
      const uint32_t st = base + (uint32_t)(s * sh.stage_bytes);
#pragma unroll
      for (int j = 0; j < BK / 16; ++j) {
        if (((b * (BK / 16) + j) & (WK - 1)) != kp) continue;
        uint32_t a[4];
        nbmma::ldmatrix_x4(a, st + a_row + (((2 * j + a_hi) ^ sw) << 4));
#pragma unroll
        for (int i = 0; i < NT; i += 2) {
          uint32_t x[4];
          nbmma::ldmatrix_x4(x, st + x_row + i * 1024 + (((2 * j + x_hi) ^ sw) << 4));
          nbmma::mma_bf16(acc[i], a, x[0], x[1]);
          nbmma::mma_bf16(acc[i + 1], a, x[2], x[3]);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty(s));
      if (++s == sh.stages) { s = 0; phase ^= 1u; }
    }
    __syncthreads();           // all blocks have landed and been read: the ring is free
    float* mine = red + (size_t)kp * ROWS * LD + wn * 16 + (lane >> 2) + (lane & 3) * 2 * LD;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      float* p = mine + i * 8 * LD;
      p[0] = acc[i][0];
      p[LD] = acc[i][1];
      p[8] = acc[i][2];
      p[LD + 8] = acc[i][3];
    }
  }
  __syncthreads();

  if (sh.split > 1) {
    if (WK > 1) {              // this CTA's sums in one place before the others ask for them
      for (int e = tid; e < M * Q; e += THREADS) {
        float* p = red + (size_t)(e / Q) * LD + (e % Q) * 4;
        float4 v = *reinterpret_cast<const float4*>(p);
#pragma unroll
        for (int k = 1; k < WK; ++k) {
          const float4 w = *reinterpret_cast<const float4*>(p + (size_t)k * ROWS * LD);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        *reinterpret_cast<float4*>(p) = v;
      }
    }
    cluster_sync();
  }
  const bool aborted = *abort_flag != 0;
  if (!aborted) {
    int i = 0;
    for (int e = tid; e < (m_hi - m_lo) * Q; e += THREADS, ++i) {
      const int m = m_lo + e / Q, n = n0 + (e % Q) * 4;
      if (n >= N) continue;
      const uint32_t off = (uint32_t)((m * LD + (e % Q) * 4) * 4);
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (sh.split > 1) {
        for (int r = 0; r < sh.split; ++r) {
          const float4 w = ld_cluster4(cluster_addr(base, r) + off);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
      } else {
#pragma unroll
        for (int k = 0; k < WK; ++k) {
          const float4 w = *reinterpret_cast<const float4*>(red + off / 4 + (size_t)k * ROWS * LD);
          v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
      }
      const size_t o = (size_t)m * N + n;
      float y[4] = {v.x, v.y, v.z, v.w};
      float r[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      if (residual != nullptr) {
        if (vec) {
          float4 q;
          if (i < AHEAD && warp < WARPS) q = i == 0 ? ahead[0] : ahead[1];
          else q = *reinterpret_cast<const float4*>(residual + o);
          r[0] = q.x; r[1] = q.y; r[2] = q.z; r[3] = q.w;
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < N) r[j] = residual[o + j];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (bias != nullptr && n + j < N) y[j] += __ldg(bias + n + j);
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
  if (sh.split > 1) cluster_sync();      // nobody leaves while another reads its shared memory
  if (aborted) {
    if (tid == 0) {
      nb_report_timeout(err_word);
      // let copies that are still in flight land before the shared memory goes away
      const long long t0 = clock64();
      while (clock64() - t0 < 4000000LL) {}
    }
    __syncthreads();
  }
}

int g_force_wn = 0, g_force_split = 0;     // tuning and tests: 0 = choose

// The layout, from sweeps over both numbers on products of 32, 40, 64 and 128 rows (us; columns a
// CTA, CTAs a cluster): 64 columns are the best or within 3 % of it (64x768x768: 64 by 4 4.3, 32 by 4
// 4.3, 16 by 3 5.3, 16 by 1 4.7; 64x768x3072: 64 by 8 6.0, 32 by 4 6.5), but
//  * 65 to 128 rows over few columns like 32 (128x768x768: 32 by 4 5.6, 64 by 4 6.4);
//  * 33 to 64 rows with so many columns that 16 a CTA fill the GPU like those uncut where K is short
//    against them.  Uncut, a product takes 2.1 and 0.18 a block of K whatever its columns; cut, it takes
//    0.08 a block and 0.013 a CTA, so the two meet near N = 2 K (64 rows, 16 by 1 and 64 by 4:
//    1024x768 4.2 and 4.0, 1536x768 4.2 and 4.4, 2048x768 4.3 and 4.8, 2304x768 4.3 and 5.2, 1536x1024
//    5.0 and 4.6, 2048x1024 5.0 and 5.1, 2304x1280 5.8 and 6.1).  Up to 8 blocks K can only be cut in
//    two (next rule) and uncut is the faster one at any number of columns (1024x512 3.4 and 4.4).
// K is cut as far as a CTA keeps three blocks and the launch stays within a CTA an SM, or within
// two where a CTA's walk is still long (64x1600x6400: 64 by 8 11.2, by 5 11.7, by 4 over 12;
// 64x1600x1600: by 5 6.4, by 8 over 6.9).
bool plan_mid(int M, int N, int K, MidShape* out) {
  if (M < 1 || M > MAX_ROWS || N < 1 || K < 8 || K % 8 != 0) return false;
  const int sms = nb_device_sms(), blocks = (K + BK - 1) / BK;
  const int rows = (M <= 32 ? 4 : (M <= 64 ? 8 : 16)) * 8;
  MidShape s;
  s.wn = 4;
  bool cut = true;
  if (M > 64 && (N + 31) / 32 * 4 <= sms) s.wn = 2;
  if (M > 32 && M <= 64 && (N >= 2 * K || blocks <= 8) && (N + 15) / 16 <= sms) {
    s.wn = 1;
    cut = false;
  }
  if (g_force_wn) s.wn = g_force_wn;
  const int c = 16 * s.wn;
  const long long groups = (N + c - 1) / c;
  s.split = 1;
  for (int split : {2, 4, 5, 8}) {
    const int kb = (blocks + split - 1) / split;
    if (!cut || kb < 3 || (split - 1) * kb >= blocks) continue;       // no CTA without a block
    if (groups * split <= (M <= 64 && kb >= 12 ? 2 * sms : sms)) s.split = split;
  }
  if (g_force_split) s.split = g_force_split;
  s.kb_per = (blocks + s.split - 1) / s.split;
  if ((s.split - 1) * s.kb_per >= blocks && s.split > 1) return false;
  s.stage_bytes = (c + rows) * 128;
  const int red = (WARPS / s.wn) * rows * (c + 4) * 4;
  s.stages = s.kb_per < MAX_STAGES ? s.kb_per : MAX_STAGES;
  while (s.stages > 1 && s.stages * s.stage_bytes > 104 * 1024) --s.stages;     // two CTAs an SM
  s.smem = s.stages * s.stage_bytes > red ? s.stages * s.stage_bytes : red;
  s.smem = (s.smem + 15) & ~15;
  *out = s;
  return s.smem <= 200 * 1024;
}

int* error_word() {
  int* w = nb_error_words();
  return w ? w + NB_ERRW_GEMM_MID : nullptr;
}

template <int NT, int WN, typename TOut>
int launch(const void* X, const void* W, const float* bias, const float* residual, void* out, int M,
           int N, int K, int act, const MidShape& sh, cudaStream_t stream) {
  constexpr int C = 16 * WN;
  CUtensorMap mx, mw;
  int rc = make_map(&mx, X, M, K, NT * 8, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  rc = make_map(&mw, W, N, K, C, BK, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2);
  if (rc) return rc;
  auto kern = gemm_mid_kernel<NT, WN, TOut>;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024));
    configured = true;
  }
  const bool vec = N % 4 == 0 && (uintptr_t)out % (4 * sizeof(TOut)) == 0 && (uintptr_t)residual % 16 == 0;
  const int smem = sh.smem + 1024 + 2 * MAX_STAGES * 8 + 16;
  NB_CUDA(nb_launch_clusters(kern, dim3((unsigned)((N + C - 1) / C * sh.split)), dim3(THREADS), (size_t)smem,
                             stream, sh.split, mx, mw, bias, residual, (TOut*)out, M, N, K, act, sh, vec,
                             error_word()));
  return 0;
}

template <int NT, typename TOut>
int launch_wn(const void* X, const void* W, const float* bias, const float* residual, void* out, int M,
              int N, int K, int act, const MidShape& sh, cudaStream_t stream) {
  switch (sh.wn) {
    case 1: return launch<NT, 1, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
    case 2: return launch<NT, 2, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
    default: return launch<NT, 4, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  }
}

template <typename TOut>
int launch_nt(const void* X, const void* W, const float* bias, const float* residual, void* out, int M,
              int N, int K, int act, const MidShape& sh, cudaStream_t stream) {
  if (M <= 32) return launch_wn<4, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  if (M <= 64) return launch_wn<8, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  return launch_wn<16, TOut>(X, W, bias, residual, out, M, N, K, act, sh, stream);
}

}  // namespace

// 1 if this kernel takes the product.
NB_EXPORT int nb_gemm_mid_supported(int M, int N, int K) {
  MidShape s;
  return plan_mid(M, N, K, &s) ? 1 : 0;
}

// 1 where this kernel is the fastest of the tensor-core products (us, this kernel and the others, back
// to back over twelve weights):
//  * 17 to 64 rows, up to 2048 columns: 64x768x768 4.0 and 4.8, 64x768x3072 5.5 and 8.4, 64x1600x6400 10.6
//    and 11.9, 33x512x64 2.1 and 2.8, 48x2048x1024 4.9 and 5.3.  Up to 32 rows also over more columns
//    (32x2304x768 4.2 and 4.7, 32x4800x1600 7.1 and 8.0); 33 to 64 rows where the layout is the uncut one
//    (64x2304x768 4.3 and 4.9).  Beyond, the tcgen05 kernels (64x3072x768 5.4 and 4.9, 64x4800x1600
//    9.3 and 8.0).
//  * 65 to 128 rows, up to 2048 columns, from a K on below which the tcgen05 kernels' tiles, with work for
//    more of their rows, are the faster ones; the sooner, the more their epilogue has to do, which
//    costs them 0.7 us for 32-bit results or an activation and 1.4 for rows that TMA cannot store
//    (128 rows; 512 columns, plain: K = 512 4.9 and 4.2, 640 4.5 and 4.5; 32-bit: 256 4.9 and 4.4, 384 4.9
//    and 5.0; GELU: 64 3.7 and 3.9, 512 5.3 and 5.0, 640 4.6 and 5.3; 333 columns, plain: 64 3.7 and 4.5;
//    2048 columns, plain: 1024 6.9 and 5.7, 1600 8.3 and 7.9, 2048 8.8 and 10.1; 32-bit: 768 6.6 and 6.2,
//    1024 7.0 and 6.9; GELU: 1024 7.1 and 6.6; 1999 columns, plain: 512 6.8 and 5.8, 768 6.6 and 6.6).
//  * up to 16 rows, up to 2048 columns, where the rows take half (96 KB) of what the kernel that keeps
//    them and its weights in shared memory together has there, so that little is left for weights in
//    flight (16x768x3072 4.6 and 6.3, 12x1600x4096 6.9 and 8.5, 10x2048x5120 8.8 and 10.6, 8x1600x6400 8.4 and
//    9.8, 16x1600x6400 8.3 and 30.4, 6x2048x8192 10.6 and 11.6).  Short of that line it depends on the
//    columns and is never far from even up to 8 rows (8x768x5120 5.6 and 6.8, 8x2048x5120 8.8 and 8.4,
//    8x1600x4096 6.9 and 6.2, 4x1600x5120 8.0 and 6.3); with 9 to 15 rows this kernel leads a little
//    earlier (9x768x3072 4.5 and 5.5, 9x2048x3072 6.1 and 6.8, 9x1280x2048 5.0 and 4.5).
NB_EXPORT int nb_gemm_mid_preferred(int M, int N, int K, int act, int out_dtype) {
  MidShape s;
  if (!plan_mid(M, N, K, &s)) return 0;
  if (M <= 16) return N <= 2048 && (long long)M * K * 2 >= 96 * 1024;
  if (M <= 64) return N <= 2048 || (M <= 32 && N <= 5120) || s.wn == 1;
  if (N > 2048) return 0;
  const bool few = N <= 1024, wide = out_dtype == NB_F32;
  int from = few ? 640 : 1536;
  if (wide && from > (few ? 384 : 1024)) from = few ? 384 : 1024;
  if (act != NB_ACT_NONE && from > (few ? 8 : 1280)) from = few ? 8 : 1280;
  if (N % (wide ? 4 : 8) != 0 && from > (few ? 8 : 768)) from = few ? 8 : 768;
  return K >= from;
}

// The layout chosen for a shape (tests and reports): columns a CTA, CTAs a cluster, blocks of K a
// CTA, stages.
NB_EXPORT int nb_gemm_mid_plan(int M, int N, int K, int* out4) {
  MidShape s;
  if (!plan_mid(M, N, K, &s)) return 0;
  out4[0] = 16 * s.wn; out4[1] = s.split; out4[2] = s.kb_per; out4[3] = s.stages;
  return 1;
}

// Tuning and tests: columns a CTA (16, 32, 64) and cluster size (1 to 8) to use; 0 = choose.
NB_EXPORT int nb_gemm_mid_force(int columns, int split) {
  NB_REQUIRE((columns == 0 || columns == 16 || columns == 32 || columns == 64) && split >= 0 && split <= MAX_SPLIT,
             NB_ERR_BAD_ARG, "gemm_mid: no layout of %d columns by %d", columns, split);
  g_force_wn = columns / 16;
  g_force_split = split;
  return 0;
}

NB_EXPORT int nb_gemm_mid_set_wait_budget(long long cycles) { return set_wait_budget(cycles); }

NB_EXPORT int nb_gemm_mid(const void* X, const void* W, const float* bias, const float* residual, void* out,
                          int out_dtype, int M, int N, int K, int act, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  MidShape sh;
  NB_REQUIRE(plan_mid(M, N, K, &sh), NB_ERR_UNSUPPORTED,
             "gemm_mid: takes 1 to %d rows and K a multiple of 8 (M=%d N=%d K=%d)", MAX_ROWS, M, N, K);
  NB_REQUIRE((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0, NB_ERR_UNSUPPORTED,
             "gemm_mid: operands must be 16-byte aligned");
  int rc;
  if (out_dtype == NB_F32) rc = launch_nt<float>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  else if (out_dtype == NB_BF16) rc = launch_nt<bf16>(X, W, bias, residual, out, M, N, K, act, sh, stream);
  else NB_REQUIRE(false, NB_ERR_BAD_ARG, "gemm_mid: unknown output type %d", out_dtype);
  if (rc) return rc;
  NB_CHECK_LAUNCH("gemm_mid");
  return 0;
}
