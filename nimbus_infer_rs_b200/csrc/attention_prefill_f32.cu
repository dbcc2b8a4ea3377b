// Prefill attention in true 32-bit arithmetic: many query rows per sequence over the paged
// key/value cache, every product and sum an fp32 multiply-add on the CUDA cores (no tensor
// cores, no rounding of operands).  It is the attention of the whole-model 32-bit path for
// prompts; heads of 64 or 128, pages of 64 tokens.
//
// A CTA takes 64 consecutive query rows of one sequence and one head and walks over the
// sequence's pages up to the last key its rows may see, or over half of them (below).  The multiply-adds
// are the floor (2 x 1,024 tokens x 12 heads of 64: 45 us at 128 a clock and SM); what bounds it is a warp's
// chain of instructions, so as few of them as possible surround the multiply-adds: a thread has 8 rows
// x 4 keys of the scores and 8 rows x 4 columns of the result (8 columns with heads of 128) as packed pairs of
// rows, so three 16-byte reads and four doubled numbers feed 16 packed multiply-adds; queries, keys and
// probabilities lie transposed, their 16-byte pieces exchanged by a few bits of the row so that neither
// the transposing stores nor the reads meet in a bank.  The next page's keys are asked for while P V
// runs and go from registers to shared memory after it, its values by cp.async beside the next scores.
// Scale, causal limit and window; running maximum per row (fp32, maximum subtracted,
// src/ops.rs:6-18) through shuffles among the threads that share a row, the sums per thread until
// the end.  Keys after a row's own position, before its window or beyond the sequence get no weight, and
// the rows of the last page that hold no key yet are never read.
//
// Tiles see as many pages as lie before them, from 1 to all, and a tile of 16 pages alone took as long as
// all others together (192 us; an SM's pages are 22 on average).  So, where a chunk has several tiles,
// the pages of a tile are halved between the two CTAs of a cluster, the second of which hands its maxima, sums
// and weighted values to the first through shared memory; and the CTAs are dealt out longest first,
// every other turn over the SMs backwards, so that an SM's CTAs add up to about the same.
//
// Reference: src/model.rs:401-422 (scores = dot(q,k)*scale for keys 0..P+i, softmax, weighted
// values); head h reads key/value head h / group (src/model.rs:390).
#include "attention_common.cuh"

namespace {

constexpr int TQ = 64;            // query rows per CTA
constexpr int PAGE_TOKENS = 64;   // keys per page
constexpr int LD = 64;            // floats between rows of a transposed tile
constexpr int THREADS = 128;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair_of(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 unpair(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;\n" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ void mul2(f32x2& c, f32x2 a) {
  asm("mul.rn.f32x2 %0, %0, %1;\n" : "+l"(c) : "l"(a));
}

// Four consecutive numbers, widened; one load where the caller has seen that they are aligned.
__device__ __forceinline__ float4 load4(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p, bool vec) {
  if (!vec)
    return make_float4(__bfloat162float(p[0]), __bfloat162float(p[1]), __bfloat162float(p[2]),
                       __bfloat162float(p[3]));
  const uint2 u = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}

// Where piece `c` (four columns) of row `d` of a transposed query or key tile lies: eight rows of the
// source times four pieces of it, which a warp turns over at once, then lie in 32 banks.
__device__ __forceinline__ int piece_of(int d, int c) { return d * LD + ((c ^ (((d >> 2) & 3) << 1)) << 2); }
// The same for row `j` (a key) of the probabilities: a thread writes the keys 4 x, 4 x + 1, ...
__device__ __forceinline__ int prob_of(int j, int c) { return j * LD + ((c ^ ((j >> 2) & 7)) << 2); }

enum : int { VEC_Q = 1, VEC_KV = 2, VEC_OUT = 4 };   // operands whose rows may be taken 4 numbers at a time

template <typename T, int HD, typename TOut>
__global__ void __launch_bounds__(THREADS, HD == 64 ? 3 : 1)
attention_prefill_f32_kernel(const T* q, int q_stride, int q_col,
                             const int* cu_rows, const int* seq_slot,
                             const int* seq_pos0, NbPagedKV kv, int group,
                             TOut* out, int out_stride, float scale, int window, int vec, int sms, int cut) {
  constexpr int TX = 16;                // threads that share a row
  constexpr int KPT = PAGE_TOKENS / TX; // keys a thread
  constexpr int CH = HD / TX / 4;       // pieces of four columns of the result a thread, HD / CH apart
  constexpr int NL = PAGE_TOKENS * HD / 4 / THREADS;       // pieces of four numbers of a page's keys a thread
  extern __shared__ __align__(16) float sm[];
  float* Qt = sm;                       // [HD][LD]: column d of row i
  float* Kt = Qt + HD * LD;             // [HD][LD]: column d of key j
  float* Pt = Kt + HD * LD;             // [64][LD]: probability of key j in row i
  float* Vs = Pt + PAGE_TOKENS * LD;    // [64][HD]

  nb_grid_dependency_wait();
  nb_launch_dependents();
  // this CTA's place in the order of work (see the head of the file); `cut`: CTAs that share a tile
  const unsigned half = blockIdx.x % cut, tiles = gridDim.x / cut, per_turn = (unsigned)sms / cut;
  const unsigned long long b = blockIdx.x / cut + (unsigned long long)tiles * (blockIdx.y + (unsigned long long)gridDim.y * blockIdx.z);
  const unsigned long long total = (unsigned long long)tiles * gridDim.y * gridDim.z;
  const unsigned long long first = b - b % per_turn;
  const unsigned long long turn = total - first < per_turn ? total - first : per_turn;
  const unsigned long long rank = (b / per_turn) & 1 ? first + (turn - 1 - (b - first)) : b;
  const unsigned hs = gridDim.y * gridDim.z, rest = (unsigned)(rank % hs);
  const int tile = (int)(tiles - 1 - (unsigned)(rank / hs)), h = (int)(rest % gridDim.y), s = (int)(rest / gridDim.y);
  const int row0 = cu_rows[s], n_q = cu_rows[s + 1] - row0;
  const int q0 = tile * TQ;
  const int slot = seq_slot[s];
  if (q0 >= n_q || slot < 0) return;
  const int pos0 = seq_pos0[s];
  const int kvh = h / group;
  const int tid = threadIdx.x, ty = tid / TX, tx = tid % TX;
  const int rows_here = min(TQ, n_q - q0);
  const int last_pos = pos0 + q0 + rows_here - 1;                    // newest key any row sees
  const int first_key = (window > 0) ? max(0, pos0 + q0 + 1 - window) : 0;
  const int p_first = first_key / PAGE_TOKENS, p_last = last_pos / PAGE_TOKENS + 1;
  const int p_middle = cut > 1 ? p_first + (p_last - p_first + 1) / 2 : p_last;
  const int p_begin = half ? p_middle : p_first, p_end = half ? p_last : p_middle;
  const int* table = kv.block_table + (size_t)slot * kv.max_pages;

  // Which pieces this thread turns over: a warp takes 8 source rows x 4 pieces at a time, so a row's 64
  // consecutive bytes come with one instruction.  Piece n of NL: row turn_j + 8 * (..), piece turn_d + ..
  const int wj = (tid & 31) >> 2, wd = tid & 3, w = tid >> 5;
  auto turn_row = [&](int n) { return wj + 8 * (n & 7); };
  auto turn_piece = [&](int n) { return wd + 4 * (w + (n >> 3) * (THREADS / 32)); };
  auto put = [&](float* t, int n, const float4& v) {
    const int j = turn_row(n), d = turn_piece(n) * 4;
    float* at = t + piece_of(d, j >> 2) + (j & 3);      // the four rows d .. d + 3 share their exchange
    at[0] = v.x; at[LD] = v.y; at[2 * LD] = v.z; at[3 * LD] = v.w;
  };
  const float4 zero4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float4 kn[NL];                        // a page's keys on their way
  auto ask_keys = [&](int p) {
    const T* src = (const T*)kv.k + ((size_t)table[p] * kv.n_kv_heads + kvh) * PAGE_TOKENS * HD;
    const int keys_here = last_pos + 1 - p * PAGE_TOKENS;      // what lies beyond is an earlier owner's
#pragma unroll
    for (int n = 0; n < NL; ++n)
      kn[n] = turn_row(n) < keys_here ? load4(src + turn_row(n) * HD + turn_piece(n) * 4, vec & VEC_KV) : zero4;
  };
  auto bring_values = [&](int p) {
    const T* src = (const T*)kv.v + ((size_t)table[p] * kv.n_kv_heads + kvh) * PAGE_TOKENS * HD;
    const int keys_here = last_pos + 1 - p * PAGE_TOKENS;
#pragma unroll 4
    for (int idx = tid; idx < PAGE_TOKENS * HD / 4; idx += THREADS) {
      float* dst = Vs + idx * 4;
      if (idx / (HD / 4) >= keys_here) *reinterpret_cast<float4*>(dst) = zero4;
      else if (sizeof(T) == 4 && (vec & VEC_KV)) cp_async16(dst, src + idx * 4);
      else *reinterpret_cast<float4*>(dst) = load4(src + idx * 4, vec & VEC_KV);
    }
    cp_async_commit();
  };

  if (p_begin < p_end) ask_keys(p_begin);
  // the query tile; rows beyond the sequence are zero
#pragma unroll 4
  for (int n = 0; n < NL; ++n) {
    const int i = turn_row(n);
    put(Qt, n, i < rows_here ? load4(q + (size_t)(row0 + q0 + i) * q_stride + q_col + (size_t)h * HD + turn_piece(n) * 4, vec & VEC_Q)
                             : zero4);
  }
  if (p_begin < p_end) {
#pragma unroll
    for (int n = 0; n < NL; ++n) put(Kt, n, kn[n]);
  }
  __syncthreads();
  if (p_begin < p_end) bring_values(p_begin);

  f32x2 o[4][4 * CH];       // rows ty * 8 + 2 i, 2 i + 1; columns tx * 4 + (0 .. 3), and HD / 2 further
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 4 * CH; ++c) o[i][c] = 0ull;
  float m_run[8], l_run[8];  // the sum of this thread's keys only
#pragma unroll
  for (int i = 0; i < 8; ++i) { m_run[i] = -INFINITY; l_run[i] = 0.0f; }

  for (int p = p_begin; p < p_end; ++p) {
    // scores: rows ty * 8 + 2 i, 2 i + 1, keys tx * 4 + (0 .. 3)
    f32x2 sc[4][KPT];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < KPT; ++c) sc[i][c] = 0ull;
#pragma unroll 4
    for (int d = 0; d < HD; ++d) {
      const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(Qt + piece_of(d, ty * 2));
      const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(Qt + piece_of(d, ty * 2 + 1));
      const float4 k4 = *reinterpret_cast<const float4*>(Kt + piece_of(d, tx));
      const f32x2 av[4] = {a0.x, a0.y, a1.x, a1.y};
      const f32x2 kv2[4] = {pair_of(k4.x, k4.x), pair_of(k4.y, k4.y), pair_of(k4.z, k4.z), pair_of(k4.w, k4.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < KPT; ++c) fma2(sc[i][c], av[i], kv2[c]);
    }
    // scale, causal limit, window; the row's maximum among the threads of the row
    const bool all = (p + 1) * PAGE_TOKENS <= pos0 + q0 + 1 && window <= 0;   // every row sees every key
    float pr[8][KPT], resc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int qp = pos0 + q0 + ty * 8 + i;           // absolute position of the row's query
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < KPT; ++c) {
        const int key = p * PAGE_TOKENS + tx * 4 + c;
        const float2 v = unpair(sc[i >> 1][c]);
        const bool ok = all || (key <= qp && (window <= 0 || key > qp - window));
        pr[i][c] = ok ? ((i & 1) ? v.y : v.x) * scale : -INFINITY;
        mx = fmaxf(mx, pr[i][c]);
      }
#pragma unroll
      for (int off = TX / 2; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
      const float m_new = fmaxf(m_run[i], mx);
      const float m_use = (m_new == -INFINITY) ? 0.0f : m_new;
      resc[i] = (m_run[i] == -INFINITY) ? 0.0f : expf(m_run[i] - m_use);
      m_run[i] = m_new;
      float sum = 0.0f;
#pragma unroll
      for (int c = 0; c < KPT; ++c) {
        pr[i][c] = (pr[i][c] == -INFINITY) ? 0.0f : expf(pr[i][c] - m_use);
        sum += pr[i][c];
      }
      l_run[i] = l_run[i] * resc[i] + sum;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const f32x2 r2 = pair_of(resc[2 * i], resc[2 * i + 1]);
#pragma unroll
      for (int c = 0; c < 4 * CH; ++c) mul2(o[i][c], r2);
    }
    // a warp reads only what its own threads wrote (its rows)
    __syncwarp();
#pragma unroll
    for (int c = 0; c < KPT; ++c) {
      const int j = tx * 4 + c;
      *reinterpret_cast<float4*>(Pt + prob_of(j, ty * 2)) = make_float4(pr[0][c], pr[1][c], pr[2][c], pr[3][c]);
      *reinterpret_cast<float4*>(Pt + prob_of(j, ty * 2 + 1)) = make_float4(pr[4][c], pr[5][c], pr[6][c], pr[7][c]);
    }
    cp_async_wait<0>();
    __syncthreads();       // the values are there; nobody reads the keys any more
    const bool more = p + 1 < p_end;
    if (more) ask_keys(p + 1);

    // o += P V
#pragma unroll 4
    for (int j = 0; j < PAGE_TOKENS; ++j) {
      const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(Pt + prob_of(j, ty * 2));
      const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(Pt + prob_of(j, ty * 2 + 1));
      const f32x2 av[4] = {a0.x, a0.y, a1.x, a1.y};
#pragma unroll
      for (int q4 = 0; q4 < CH; ++q4) {
        const float4 t = *reinterpret_cast<const float4*>(Vs + j * HD + q4 * (HD / 2) + tx * 4);
        const f32x2 vv[4] = {pair_of(t.x, t.x), pair_of(t.y, t.y), pair_of(t.z, t.z), pair_of(t.w, t.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) fma2(o[i][q4 * 4 + c], av[i], vv[c]);
      }
    }
    if (more) {
#pragma unroll
      for (int n = 0; n < NL; ++n) put(Kt, n, kn[n]);
    }
    __syncthreads();       // the next keys are there; nobody reads the values any more
    if (more) bring_values(p + 1);
  }

#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int off = TX / 2; off > 0; off >>= 1) l_run[i] += __shfl_xor_sync(0xffffffffu, l_run[i], off);
  // The second CTA's maxima, sums and weighted values, where its tiles were (all pages are done with):
  // [64 rows][HD], maxima [64], sums [64].
  float* part = sm;
  if (cut > 1) {
    if (half) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = ty * 8 + i;
#pragma unroll
        for (int q4 = 0; q4 < CH; ++q4) {
          float y[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float2 v = unpair(o[i >> 1][q4 * 4 + c]);
            y[c] = (i & 1) ? v.y : v.x;
          }
          *reinterpret_cast<float4*>(part + r * HD + q4 * (HD / 2) + tx * 4) = make_float4(y[0], y[1], y[2], y[3]);
        }
        if (tx == 0) { part[TQ * HD + r] = m_run[i]; part[TQ * HD + TQ + r] = l_run[i]; }
      }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
  }
  if (half == 0) {
    uint32_t other = 0;
    if (cut > 1) {
      const uint32_t own = (uint32_t)__cvta_generic_to_shared(part);
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(other) : "r"(own), "r"(1));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = ty * 8 + i;
      if (r >= rows_here) continue;
      float l = l_run[i], own = 1.0f, more = 0.0f;        // factors of the two parts
      if (cut > 1) {
        float m1, l1;
        asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(m1) : "r"(other + (uint32_t)(TQ * HD + r) * 4u) : "memory");
        asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(l1) : "r"(other + (uint32_t)(TQ * HD + TQ + r) * 4u) : "memory");
        const float m = fmaxf(m_run[i], m1);
        own = m_run[i] == -INFINITY ? 0.0f : expf(m_run[i] - m);
        more = m1 == -INFINITY ? 0.0f : expf(m1 - m);
        l = l * own + l1 * more;
      }
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
      for (int q4 = 0; q4 < CH; ++q4) {
        float y[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float2 v = unpair(o[i >> 1][q4 * 4 + c]);
          y[c] = (i & 1) ? v.y : v.x;
        }
        if (cut > 1) {
          float4 t;
          asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                       : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
                       : "r"(other + (uint32_t)(r * HD + q4 * (HD / 2) + tx * 4) * 4u)
                       : "memory");
          y[0] = y[0] * own + t.x * more; y[1] = y[1] * own + t.y * more;
          y[2] = y[2] * own + t.z * more; y[3] = y[3] * own + t.w * more;
        }
        TOut* dst = out + (size_t)(row0 + q0 + r) * out_stride + (size_t)h * HD + q4 * (HD / 2) + tx * 4;
        if (sizeof(TOut) == 4 && (vec & VEC_OUT)) {
          *reinterpret_cast<float4*>(dst) = make_float4(y[0] * inv, y[1] * inv, y[2] * inv, y[3] * inv);
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[c] = nb_from_f32<TOut>(y[c] * inv);
        }
      }
    }
  }
  if (cut > 1)      // the second CTA stays until it has been read
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

template <typename T, int HD, typename TOut>
int launch(const void* q, int q_stride, int q_col, const int* cu_rows, const int* seq_slot,
           const int* seq_pos0, const NbPagedKV& kv, int n_heads, void* out, int out_stride,
           float scale, int window, int n_seqs, int max_q_len, cudaStream_t stream) {
  const size_t smem = (size_t)(2 * HD * LD + PAGE_TOKENS * (HD + LD)) * sizeof(float);
  auto kern = attention_prefill_f32_kernel<T, HD, TOut>;
  static bool configured = false;   // per instantiation
  if (!configured) {
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured = true;
  }
  const bool vec_q = (uintptr_t)q % (4 * sizeof(T)) == 0 && q_stride % 4 == 0 && q_col % 4 == 0;
  const bool vec_kv = (uintptr_t)kv.k % 16 == 0 && (uintptr_t)kv.v % 16 == 0;
  const bool vec_out = (uintptr_t)out % 16 == 0 && out_stride % 4 == 0;
  const int vec = (vec_q ? VEC_Q : 0) | (vec_kv ? VEC_KV : 0) | (vec_out ? VEC_OUT : 0);
  const int tiles = (max_q_len + TQ - 1) / TQ, cut = tiles > 1 && tiles < (1 << 30) ? 2 : 1;
  dim3 grid(tiles * cut, n_heads, n_seqs);
  NB_CUDA(nb_launch_clusters(kern, grid, dim3(THREADS), smem, stream, cut, (const T*)q, q_stride, q_col, cu_rows,
                    seq_slot, seq_pos0, kv, n_heads / kv.n_kv_heads, (TOut*)out, out_stride, scale,
                    window, vec, nb_device_sms(), cut));
  return 0;
}

}  // namespace

// 1 if the 32-bit prefill kernel takes this shape (otherwise the caller uses the generic kernel).
NB_EXPORT int nb_attention_prefill_f32_supported(int head_dim, int n_heads, int n_kv_heads, int page) {
  if (page != PAGE_TOKENS || n_kv_heads < 1 || n_heads % n_kv_heads != 0) return 0;
  return head_dim == 64 || head_dim == 128;
}

// Rows of sequence s are cu_rows[s]..cu_rows[s+1] of the packed batch, at positions
// seq_pos0[s].. of slot seq_slot[s]; their keys and values are already in the cache.  `dtype`:
// element type of the queries and of the cache (fp32, or bf16 widened on the way in).
NB_EXPORT int nb_attention_prefill_f32(const void* q, int dtype, int q_stride, int q_col,
                                       const int* cu_rows, const int* seq_slot, const int* seq_pos0,
                                       const void* k_cache, const void* v_cache,
                                       const int* block_table, int max_pages, int page, int n_heads,
                                       int n_kv_heads, int head_dim, void* out, int out_dtype,
                                       int out_stride, float scale, int window, int n_seqs,
                                       int max_q_len, cudaStream_t stream) {
  if (n_seqs == 0 || max_q_len == 0) return 0;
  NB_REQUIRE(nb_attention_prefill_f32_supported(head_dim, n_heads, n_kv_heads, page), NB_ERR_UNSUPPORTED,
             "attention_prefill_f32: unsupported shape (head size %d, %d/%d heads, page %d)", head_dim,
             n_heads, n_kv_heads, page);
  NB_REQUIRE(n_seqs <= 65535 && n_heads <= 65535, NB_ERR_UNSUPPORTED, "attention_prefill_f32: grid too large");
  NbPagedKV kv{(void*)k_cache, (void*)v_cache, block_table, max_pages, page, n_kv_heads, head_dim};
  typedef __nv_bfloat16 bf16;
  int rc = NB_ERR_BAD_ARG;
#define NB_ARGS q, q_stride, q_col, cu_rows, seq_slot, seq_pos0, kv, n_heads, out, out_stride, scale, window, n_seqs, max_q_len, stream
#define NB_HD(T_, TO_) rc = head_dim == 64 ? launch<T_, 64, TO_>(NB_ARGS) : launch<T_, 128, TO_>(NB_ARGS)
  if (dtype == NB_F32 && out_dtype == NB_F32) { NB_HD(float, float); }
  else if (dtype == NB_F32 && out_dtype == NB_BF16) { NB_HD(float, bf16); }
  else if (dtype == NB_BF16 && out_dtype == NB_F32) { NB_HD(bf16, float); }
  else if (dtype == NB_BF16 && out_dtype == NB_BF16) { NB_HD(bf16, bf16); }
#undef NB_HD
#undef NB_ARGS
  NB_REQUIRE(rc != NB_ERR_BAD_ARG, NB_ERR_BAD_ARG, "attention_prefill_f32: unknown dtypes %d/%d", dtype, out_dtype);
  if (rc) return rc;
  NB_CHECK_LAUNCH("attention_prefill_f32");
  return 0;
}
