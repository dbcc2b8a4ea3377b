// Products of a decode step in the true 32-bit path (few rows, fp32 weights):
// out[M,N] = act(X W^T + bias) (+ residual), every product and sum in fp32.
//
// Bound by bringing the weights in once.  A CTA owns COLS output columns at a time and its
// threads share K: each thread holds its 16-byte pieces of the COLS weight rows in registers,
// asked for before it waits for the kernel ahead (and, for the next columns it takes, before
// the sums of the present ones are added up), so that a whole SM keeps some 100 KB of weights
// in flight.  The rows need no staging: a thread reads from each row just the pieces that face
// its weights.  Sums are dealt out over a warp by halving exchanges and added over the warps
// through shared memory.
//
// Measured against one column a warp with the weights asked for after the wait (us, back to back,
// rows x columns x K): 8x2304x768 4.2 (7.0), 8x768x768 2.7 (5.7), 8x3072x768 5.3 (9.4),
// 8x768x3072 6.3 (13.2), 8x50257x768 53 (91), 1x768x3072 5.9 (11.6), 32x768x3072 17 (40),
// 64x768x768 11 (35).
//
// Reference analogue: Mat::gemv_into (src/model.rs:65-86).
#include "gemm_f32.cuh"

namespace {

constexpr int ROWS = 8;       // rows multiplied at a time

// Adds `v` over the 32 lanes; afterwards lane l holds the sums of elements l * N / 32 ... in
// v[0 .. N / 32 - 1] (N is 32 or 64).
template <int N>
__device__ __forceinline__ void deal_out(float (&v)[N], int lane) {
#pragma unroll
  for (int half = N / 2, bit = 16; bit > 0; half >>= 1, bit >>= 1) {
    const bool up = lane & bit;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = up ? v[i] : v[half + i];
      const float keep = up ? v[half + i] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
  }
}

// NQ: 16-byte pieces of a weight row that a thread holds.
template <int COLS, int NQ, typename TOut>
__global__ void __launch_bounds__(256)
gemm_rows_f32_kernel(const float* X, const float* __restrict__ W, const float* __restrict__ bias,
                     const float* residual, TOut* out, int M, int N, int K, int act) {
  constexpr int VALUES = ROWS * COLS, EACH = VALUES / 32;
  __shared__ float red[8][VALUES];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, threads = blockDim.x;
  const int quads = K >> 2;
  const int n_groups = (N + COLS - 1) / COLS;

  float4 w[COLS][NQ];
  auto load_weights = [&](int grp) {
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int n = grp * COLS + c, k = tid + q * threads;
        w[c][q] = (n < N && k < quads)
                      ? __ldg(reinterpret_cast<const float4*>(W + (size_t)n * K) + k)
                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
  };
  load_weights(blockIdx.x);
  nb_grid_dependency_wait();

  for (int grp = blockIdx.x; grp < n_groups; grp += gridDim.x) {
    for (int m0 = 0; m0 < M; m0 += ROWS) {
      const int rows = min(ROWS, M - m0);
      float acc[VALUES];
#pragma unroll
      for (int i = 0; i < VALUES; ++i) acc[i] = 0.0f;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int k = tid + q * threads;
        float4 x[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
          x[r] = (r < rows && k < quads) ? *(reinterpret_cast<const float4*>(X + (size_t)(m0 + r) * K) + k)
                                         : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
          for (int c = 0; c < COLS; ++c) {
            float a = acc[r * COLS + c];
            a = fmaf(x[r].x, w[c][q].x, a);
            a = fmaf(x[r].y, w[c][q].y, a);
            a = fmaf(x[r].z, w[c][q].z, a);
            acc[r * COLS + c] = fmaf(x[r].w, w[c][q].w, a);
          }
      }
      if (m0 + ROWS >= M) {
        if (grp + (int)gridDim.x < n_groups) load_weights(grp + gridDim.x);
        else nb_launch_dependents();     // this CTA's weights are all in
      }
      deal_out(acc, lane);
      __syncthreads();                   // the sums before these have been read
#pragma unroll
      for (int i = 0; i < EACH; ++i) red[warp][lane * EACH + i] = acc[i];
      __syncthreads();
      for (int i = tid; i < VALUES; i += threads) {
        const int m = m0 + i / COLS, n = grp * COLS + i % COLS;
        if (m >= M || n >= N) continue;
        float v = 0.0f;
        for (int s = 0; s < (threads >> 5); ++s) v += red[s][i];
        if (bias) v += __ldg(bias + n);
        v = nb_apply_act(v, act);
        const size_t o = (size_t)m * N + n;
        if (residual) v += residual[o];
        out[o] = nb_from_f32<TOut>(v);
      }
    }
  }
}

// Threads that share K, and CTAs of so many that fit on the GPU at once.
int threads_for(int K, int nq) { return ((K / 4 + nq - 1) / nq + 31) / 32 * 32; }
template <int COLS, int NQ, typename TOut>
cudaError_t fitting(int threads, int* fit) {
  static int resident[9] = {};       // by warps
  if (resident[threads / 32] == 0) {
    int per_sm = 0;
    const cudaError_t e =
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, gemm_rows_f32_kernel<COLS, NQ, TOut>, threads, 0);
    if (e != cudaSuccess) return e;
    resident[threads / 32] = (per_sm > 0 ? per_sm : 1) * nb_device_sms();
  }
  *fit = resident[threads / 32];
  return cudaSuccess;
}

template <int COLS, int NQ, typename TOut>
cudaError_t launch(const float* X, const float* W, const float* bias, const float* residual, TOut* out,
                   int M, int N, int K, int act, cudaStream_t stream) {
  const int threads = threads_for(K, NQ), n_groups = (N + COLS - 1) / COLS;
  int fit = 0;
  const cudaError_t e = fitting<COLS, NQ, TOut>(threads, &fit);
  if (e != cudaSuccess) return e;
  return nb_launch(gemm_rows_f32_kernel<COLS, NQ, TOut>, dim3(n_groups < fit ? n_groups : fit), dim3(threads), 0,
                   stream, X, W, bias, residual, out, M, N, K, act);
}

}  // namespace

template <typename TOut>
bool nb_gemm_f32_rows(const float* X, const float* W, const float* bias, const float* residual,
                      TOut* out, int M, int N, int K, int act, cudaStream_t stream,
                      cudaError_t* err) {
  // 16-byte pieces; a row of weights is held in at most three of them a thread (with more the weights
  // of four columns no longer fit beside the rows in registers)
  if (K % 4 || K < 4 || K > 3 * 1024 || (uintptr_t)X % 16 || (uintptr_t)W % 16) return false;
  // eight columns a CTA where that leaves a CTA for every SM and all CTAs run at once, else four: a second
  // walk over groups of eight costs more than one over groups of four (1 row us, eight and four:
  // 2304x768 3.6 and 3.9, 1184x1024 2.5 and 3.0; but 3072x640 4.7 and 4.2, 50257x768 57 and 51, and above 768
  // of K, where the registers leave an SM one CTA of 256 threads, 1600x1024 4.4 and 3.1, 4096x1024 10.1
  // and 8.3, 50257x1024 98 and 70)
  bool wide = false;
  if (K <= 1024 && N >= 8 * nb_device_sms()) {
    int fit = 0;
    *err = fitting<8, 1, TOut>(threads_for(K, 1), &fit);
    if (*err != cudaSuccess) return true;
    wide = (N + 7) / 8 <= fit;
  }
#define NB_GO(C_, Q_) *err = launch<C_, Q_, TOut>(X, W, bias, residual, out, M, N, K, act, stream)
  if (K <= 1024) { if (wide) NB_GO(8, 1); else NB_GO(4, 1); }
  else if (K <= 2048) NB_GO(4, 2);
  else NB_GO(4, 3);
#undef NB_GO
  return true;
}

template bool nb_gemm_f32_rows<float>(const float*, const float*, const float*, const float*, float*,
                                      int, int, int, int, cudaStream_t, cudaError_t*);
template bool nb_gemm_f32_rows<__nv_bfloat16>(const float*, const float*, const float*, const float*,
                                              __nv_bfloat16*, int, int, int, int, cudaStream_t,
                                              cudaError_t*);
