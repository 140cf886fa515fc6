// Causal grouped-query attention over the paged cache in true float32 (no tensor cores), heads of 64 or 128 channels:
// one kernel for steps of many tokens, one (with a short joining kernel) for steps of one token per sequence.
//
// Every sum's order depends only on the query's own position and window, so a token's result is the same bits whether it
// came in a prompt, in a portion or alone, whatever else the step holds:
//   * a score is the sum of two chains over the even and the odd channels, each fmaf with channels ascending, times the scale;
//   * keys go in pages of 64 positions, two pages a chunk (both counted from position 0 of the sequence). Within a chunk an
//     online softmax runs page by page: maximum, then sum and weighted values scaled by exp(old - new maximum), the page's
//     weights summed in four runs of 16 ((0 + 1) + (2 + 3)), weighted values added one fmaf per key, keys ascending;
//   * chunks are joined in ascending order, each time to the larger of the two maxima.
// A page without a visible key changes nothing. Values of keys that a query does not see are not multiplied by a zero weight
// but left out. Formulas as in the general kernel (attention_generic.cu), which serves what these do not take: other head
// sizes, other score rules, bfloat16.
//
// Before, the general kernel read every key and value row once per query and head. 16 / 8 heads of 128, us before / now: eight
// prompts of 400 tokens 2,034 / 197, single tokens at a context of 700 (batch 8) 41 / 16, at 4,000 (batch 1) 184 / 23.
#include <math.h>

#include "packed_f32.cuh"

namespace slb {

struct AttnF32Args {
  const float* q;        // [tokens, H, hd]
  const float* k_pool;   // [pages, K, 64, hd]
  const float* v_pool;
  float* out;            // [tokens, H * hd]
  const int* seq_start;  // [n] first token row of each sequence
  const int* past;       // [n] position of that token
  const int* counts;     // [n]
  const int* block_table;
  int table_stride, n_seqs, heads, kv_heads, window;
  float scale;
  const float* sinks;    // [H] or null
  float* scratch;        // single tokens: per (sequence, head, chunk) hd weighted values, maximum, sum
  int chunks;            // chunks a sequence can have
};

constexpr int kChunkPages = 2;
constexpr int kMostGroup = 16;      // query heads per kv head

__device__ __forceinline__ float max_nan(float a, float b) {      // a NaN score stays visible
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
__device__ __forceinline__ float exp_diff(float a, float b) { return expf(__fsub_rn(a, b)); }

// One more chunk (maximum m, sum l) joins what came before (M, L): the factors for both sides' weighted values.
__device__ __forceinline__ void join_factors(float m, float l, float& M, float& L, float& fa, float& fb) {
  if (m == -INFINITY) { fa = 1.0f; fb = 0.0f; return; }
  const float top = max_nan(M, m);
  fa = exp_diff(M, top);
  fb = exp_diff(m, top);
  L = __fmaf_rn(l, fb, __fmul_rn(L, fa));
  M = top;
}
__device__ __forceinline__ float join_value(float acc, float o, float fa, float fb) { return __fmaf_rn(acc, fb, __fmul_rn(o, fa)); }
// What the joined weighted values are multiplied by; a sink counts once in the denominator.
__device__ __forceinline__ float last_factor(const float* sinks, int head, float M, float L) {
  if (sinks == nullptr) return __fdiv_rn(1.0f, L);
  const float sink = sinks[head], top = max_nan(M, sink), e = exp_diff(M, top);
  return __fdiv_rn(e, __fmaf_rn(L, e, exp_diff(sink, top)));
}

// ---- many tokens ----------------------------------------------------------------------------------------------
// A block takes 64 rows = (64 / G) tokens x G query heads of one kv head, so that a page of keys and values is read once for
// the whole group; 256 threads, 4 x 4 scores and 4 x HD / 16 outputs each. Bound by the FMA pipe: per four channels 8
// sixteen-byte shared-memory reads for 32 packed FMAs in the scores, per four keys 12 for 64 in the weighted sum. The next
// page's keys are copied while the current weights are applied, its values while its scores are formed. Queries, keys and
// weights lie in shared memory with the 16-byte groups of row r exchanged by r % 8, without padding: 112 KB, two blocks an SM.
constexpr int kRows = 64;
template <int HD> constexpr int prompt_smem() { return (3 * 64 * HD + 64 * 64 + 3 * 64) * 4; }

template <int HD>
__device__ __forceinline__ int swz(int row, int group) { return row * HD + ((group ^ (row & 7)) << 2); }

template <int HD>
__global__ void __launch_bounds__(256, 2) attn_f32_prompt_kernel(AttnF32Args a) {
  pdl_enter();
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;
  float* ks = qs + 64 * HD;
  float* vs = ks + 64 * HD;
  float* ps = vs + 64 * HD;
  float* alpha_s = ps + 64 * 64;
  float* fa_s = alpha_s + 64;
  float* fb_s = fa_s + 64;
  constexpr int kGroups = HD / 4;       // 16-byte groups of a row
  constexpr int CH = HD / 64;           // 16-byte groups of output channels per thread
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = a.heads / a.kv_heads, tile_tokens = kRows / G;
  const int kh = blockIdx.x, seq = blockIdx.y;
  const int count = a.counts[seq];
  const int tile = gridDim.z - 1 - blockIdx.z;      // the longest first
  const int t0 = tile * tile_tokens;
  if (t0 >= count) return;
  const int tokens = min(tile_tokens, count - t0), rows = tokens * G;
  const int pos0 = a.past[seq] + t0, pos1 = pos0 + tokens - 1;
  const size_t token0 = (size_t)a.seq_start[seq] + t0;
  const int* table = a.block_table + (size_t)seq * a.table_stride;

  const int page_lo = first_key(pos0, a.window) / kPageTokens, page_hi = pos1 / kPageTokens;
  auto ask_page = [&](float* dst, const float* pool, int page, bool swizzle) {
    const float* src = pool + ((size_t)table[page] * a.kv_heads + kh) * (kPageTokens * HD);
#pragma unroll
    for (int e = tid; e < 64 * kGroups; e += 256) {
      const int r = e / kGroups, g = e % kGroups;
      copy_async<true>(dst + (swizzle ? swz<HD>(r, g) : e * 4), src + e * 4, 16);
    }
  };
  for (int e = tid; e < 64 * kGroups; e += 256) {
    const int r = e / kGroups, g = e % kGroups;
    const bool live = r < rows;
    const float* src = live ? a.q + ((token0 + r / G) * a.heads + kh * G + r % G) * HD + g * 4 : a.q;
    copy_async<true>(qs + swz<HD>(r, g), src, live ? 16 : 0);
  }
  ask_page(ks, a.k_pool, page_lo, true);
  copies_commit();
  ask_page(vs, a.v_pool, page_lo, false);
  copies_commit();

  // scores and outputs: rows r0 + 4 i; keys c0 + 8 j; output channels o0 + 32 h .. + 3
  const int r0 = (warp & 3) * 16 + (lane >> 3), c0 = (warp >> 2) * 32 + (lane & 7);
  const int o0 = (warp >> 2) * (HD / 2) + (lane & 7) * 4;
  int row_pos[4], row_lo[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 4 * i;
    row_pos[i] = r < rows ? pos0 + r / G : -1;
    row_lo[i] = r < rows ? first_key(row_pos[i], a.window) : 0;
  }
  const int last_lo = first_key(pos1, a.window);
  f32x2 acc[4][2 * CH], o[4][2 * CH];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int c = 0; c < 2 * CH; ++c) acc[i][c] = o[i][c] = 0;
  // softmax: four threads a row, 16 keys each
  const int sr = tid >> 2, sq = tid & 3;
  float m = -INFINITY, l = 0.0f, M = -INFINITY, L = 0.0f;

  for (int page = page_lo; page <= page_hi; ++page) {
    const bool new_chunk = page % kChunkPages == 0 && page != page_lo;
    const bool masked = page * kPageTokens + kPageTokens - 1 > pos0 || page * kPageTokens < last_lo;
    copies_wait<1>();
    __syncthreads();
    {
      f32x2 s[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s[i][j] = 0;
#pragma unroll 4
      for (int g = 0; g < kGroups; ++g) {
        ulonglong2 qv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(qs + swz<HD>(r0 + 4 * i, g));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(ks + swz<HD>(c0 + 8 * j, g));
#pragma unroll
          for (int i = 0; i < 4; ++i) s[i][j] = fma2(qv[i].x, kv.x, s[i][j]);
#pragma unroll
          for (int i = 0; i < 4; ++i) s[i][j] = fma2(qv[i].y, kv.y, s[i][j]);
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int c = c0 + 8 * j, key = page * kPageTokens + c, r = r0 + 4 * i;
          float v = __fmul_rn(halves_sum(s[i][j]), a.scale);
          if (masked && (key > row_pos[i] || key < row_lo[i])) v = -INFINITY;
          ps[swz<64>(r, c >> 2) + (c & 3)] = v;
        }
    }
    __syncthreads();
    if (page < page_hi) ask_page(ks, a.k_pool, page + 1, true);
    copies_commit();
    {
      float4 x[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) x[g] = *reinterpret_cast<const float4*>(ps + swz<64>(sr, 4 * sq + g));
      float top = -INFINITY;
#pragma unroll
      for (int g = 0; g < 4; ++g) top = max_nan(top, max_nan(max_nan(x[g].x, x[g].y), max_nan(x[g].z, x[g].w)));
      top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, 1));
      top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, 2));
      if (new_chunk) {
        float fa, fb;
        join_factors(m, l, M, L, fa, fb);
        if (sq == 0) { fa_s[sr] = fa; fb_s[sr] = fb; }
        m = -INFINITY;
        l = 0.0f;
      }
      const float m_new = max_nan(m, top);
      float alpha = 1.0f, sum = 0.0f;
      if (m_new == -INFINITY) {
#pragma unroll
        for (int g = 0; g < 4; ++g) x[g] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        alpha = exp_diff(m, m_new);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          x[g].x = exp_diff(x[g].x, m_new); x[g].y = exp_diff(x[g].y, m_new);
          x[g].z = exp_diff(x[g].z, m_new); x[g].w = exp_diff(x[g].w, m_new);
          sum = __fadd_rn(sum, x[g].x); sum = __fadd_rn(sum, x[g].y);
          sum = __fadd_rn(sum, x[g].z); sum = __fadd_rn(sum, x[g].w);
        }
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) *reinterpret_cast<float4*>(ps + swz<64>(sr, 4 * sq + g)) = x[g];
      sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, 1));
      sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, 2));
      l = __fmaf_rn(l, alpha, sum);
      m = m_new;
      if (sq == 0) alpha_s[sr] = alpha;
    }
    copies_wait<1>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + 4 * i;
      if (new_chunk) {
        const f32x2 fa = both(fa_s[r]), fb = both(fb_s[r]);
#pragma unroll
        for (int c = 0; c < 2 * CH; ++c) {
          o[i][c] = fma2(acc[i][c], fb, mul2(o[i][c], fa));
          acc[i][c] = 0;
        }
      } else {
        const f32x2 al = both(alpha_s[r]);
#pragma unroll
        for (int c = 0; c < 2 * CH; ++c) acc[i][c] = mul2(acc[i][c], al);
      }
    }
    const int keys = min(kPageTokens, pos1 + 1 - page * kPageTokens);
    if (!masked) {
#pragma unroll 4
      for (int j4 = 0; j4 < 16; ++j4) {
        float4 p[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(ps + swz<64>(r0 + 4 * i, j4));
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
          ulonglong2 v[CH];
#pragma unroll
          for (int h = 0; h < CH; ++h) v[h] = *reinterpret_cast<const ulonglong2*>(vs + (j4 * 4 + jj) * HD + o0 + 32 * h);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const f32x2 w = both(jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w);
#pragma unroll
            for (int h = 0; h < CH; ++h) {
              acc[i][2 * h] = fma2(w, v[h].x, acc[i][2 * h]);
              acc[i][2 * h + 1] = fma2(w, v[h].y, acc[i][2 * h + 1]);
            }
          }
        }
      }
    } else {
#pragma unroll 2
      for (int j = 0; j < keys; ++j) {
        const int key = page * kPageTokens + j;
        ulonglong2 v[CH];
#pragma unroll
        for (int h = 0; h < CH; ++h) v[h] = *reinterpret_cast<const ulonglong2*>(vs + j * HD + o0 + 32 * h);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const f32x2 w = both(ps[swz<64>(r0 + 4 * i, j >> 2) + (j & 3)]);
          if (key > row_pos[i] || key < row_lo[i]) continue;
#pragma unroll
          for (int h = 0; h < CH; ++h) {
            acc[i][2 * h] = fma2(w, v[h].x, acc[i][2 * h]);
            acc[i][2 * h + 1] = fma2(w, v[h].y, acc[i][2 * h + 1]);
          }
        }
      }
    }
    __syncthreads();
    if (page < page_hi) ask_page(vs, a.v_pool, page + 1, false);
    copies_commit();
  }
  copies_wait<0>();
  {
    float fa, fb;
    join_factors(m, l, M, L, fa, fb);
    const float f = sr < rows ? last_factor(a.sinks, kh * G + sr % G, M, L) : 0.0f;
    if (sq == 0) { fa_s[sr] = fa; fb_s[sr] = fb; alpha_s[sr] = f; }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 4 * i;
    if (r >= rows) continue;
    const f32x2 fa = both(fa_s[r]), fb = both(fb_s[r]), f = both(alpha_s[r]);
    float* dst = a.out + ((token0 + r / G) * a.heads + kh * G + r % G) * HD;
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      ulonglong2 v;
      v.x = mul2(fma2(acc[i][2 * h], fb, mul2(o[i][2 * h], fa)), f);
      v.y = mul2(fma2(acc[i][2 * h + 1], fb, mul2(o[i][2 * h + 1], fa)), f);
      *reinterpret_cast<ulonglong2*>(dst + o0 + 32 * h) = v;
    }
  }
}

// ---- single tokens --------------------------------------------------------------------------------------------
// A block takes the chunks z, z + gridDim.z, ... of one (sequence, kv head), all G query heads of it. Bound by the read of keys and
// values: a chunk's keys (128 rows, 64 KB at 128 channels) come by asynchronous copies, its values are asked into L2 at the same
// time and read by the threads that own their channel. Results go to scratch per chunk; attn_f32_join_kernel joins them.
// GP: query heads per kv head, rounded up to 2, 4, 8 or 16.
template <int HD, int GP> constexpr int token_smem() { return (128 * HD + GP * HD + GP * 128 + 3 * GP) * 4; }

template <int HD, int GP>
__global__ void __launch_bounds__(256) attn_f32_token_kernel(AttnF32Args a) {
  pdl_enter();
  extern __shared__ __align__(16) float smem[];
  float* ks = smem;                    // [128][HD], swizzled
  float* qs = ks + 128 * HD;           // [GP][HD]
  float* ps = qs + GP * HD;            // [GP][128]
  float* alpha_s = ps + GP * 128;      // [GP] of the second page
  float* m_s = alpha_s + GP;
  float* l_s = m_s + GP;
  constexpr int kGroups = HD / 4, HQ = GP / 2;
  constexpr int kParts = 256 / HD, HV = GP >= kParts ? GP / kParts : 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = a.heads / a.kv_heads;
  const int kh = blockIdx.x, seq = blockIdx.y;
  const int pos = a.past[seq], lo = first_key(pos, a.window);
  const size_t token = a.seq_start[seq];
  const int* table = a.block_table + (size_t)seq * a.table_stride;
  const int chunk_lo = lo / 128, chunk_hi = pos / 128;
  int chunk = chunk_lo + blockIdx.z;
  if (chunk > chunk_hi) return;
  for (int e = tid; e < GP * HD; e += 256) qs[e] = e < G * HD ? a.q[(token * a.heads + kh * G) * HD + e] : 0.0f;

  for (; chunk <= chunk_hi; chunk += gridDim.z) {
    const int key0 = chunk * 128, first = max(lo - key0, 0), last = min(pos - key0, 127);      // visible keys of the chunk
    for (int p = first / 64; p <= last / 64; ++p) {
      const size_t base = ((size_t)table[chunk * kChunkPages + p] * a.kv_heads + kh) * (kPageTokens * HD);
      if (tid == 0) {
        const uint32_t bytes = (uint32_t)(min(last + 1 - 64 * p, 64) * HD * 4);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.v_pool + base), "r"(bytes) : "memory");
      }
      const int most = min(last + 1 - 64 * p, 64) * kGroups;
      for (int e = tid; e < most; e += 256) copy_async<true>(ks + swz<HD>(64 * p + e / kGroups, e % kGroups), a.k_pool + base + e * 4, 16);
    }
    copies_commit();
    copies_wait<0>();
    __syncthreads();
    {
      const int key = tid & 127, half = tid >> 7;      // heads half, half + 2, ...
      f32x2 s[HQ];
#pragma unroll
      for (int h = 0; h < HQ; ++h) s[h] = 0;
      if (key >= first && key <= last) {
#pragma unroll 8
        for (int g = 0; g < kGroups; ++g) {
          const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(ks + swz<HD>(key, g));
#pragma unroll
          for (int h = 0; h < HQ; ++h) {
            const ulonglong2 qv = *reinterpret_cast<const ulonglong2*>(qs + (half + 2 * h) * HD + 4 * g);
            s[h] = fma2(qv.x, kv.x, s[h]);
            s[h] = fma2(qv.y, kv.y, s[h]);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < HQ; ++h)
        ps[(half + 2 * h) * 128 + key] = (key >= first && key <= last) ? __fmul_rn(halves_sum(s[h]), a.scale) : -INFINITY;
    }
    __syncthreads();
    for (int h = warp; h < G; h += 8) {      // one warp a head: both pages' weights
      float* row = ps + h * 128;
      float m = -INFINITY, l = 0.0f;
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        float x0 = row[64 * p + lane], x1 = row[64 * p + 32 + lane];
        float top = max_nan(x0, x1);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) top = max_nan(top, __shfl_xor_sync(0xffffffffu, top, d));
        const float m_new = max_nan(m, top);
        float alpha = 1.0f, sum = 0.0f;
        if (m_new == -INFINITY) {
          x0 = x1 = 0.0f;
        } else {
          alpha = exp_diff(m, m_new);
          x0 = exp_diff(x0, m_new);
          x1 = exp_diff(x1, m_new);
        }
        row[64 * p + lane] = x0;
        row[64 * p + 32 + lane] = x1;
        __syncwarp();
        if (lane < 4)
#pragma unroll
          for (int j = 0; j < 16; ++j) sum = __fadd_rn(sum, row[64 * p + 16 * lane + j]);
        sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, 1));
        sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, 2));
        l = __fmaf_rn(l, alpha, sum);      // (lanes 0 to 3)
        m = m_new;
        if (p == 1 && lane == 0) alpha_s[h] = alpha;
      }
      if (lane == 0) { m_s[h] = m; l_s[h] = l; }
    }
    __syncthreads();
    {
      const int c = tid % HD, part = tid / HD;         // heads part, part + kParts, ...
      float acc[HV];
#pragma unroll
      for (int h = 0; h < HV; ++h) acc[h] = 0.0f;
      if (part < GP) {
        for (int p = first / 64; p <= last / 64; ++p) {
          const float* v = a.v_pool + ((size_t)table[chunk * kChunkPages + p] * a.kv_heads + kh) * (kPageTokens * HD) + c;
          if (p == 1) {
#pragma unroll
            for (int h = 0; h < HV; ++h) acc[h] = __fmul_rn(acc[h], alpha_s[min(part + kParts * h, G - 1)]);
          }
          const int j0 = max(first - 64 * p, 0), j1 = min(last - 64 * p, 63);
          int j = j0;
          for (; j + 15 <= j1; j += 16) {
            float x[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) x[u] = v[(size_t)(j + u) * HD];
#pragma unroll
            for (int u = 0; u < 16; ++u)
#pragma unroll
              for (int h = 0; h < HV; ++h) acc[h] = __fmaf_rn(ps[(part + kParts * h) * 128 + 64 * p + j + u], x[u], acc[h]);
          }
          for (; j <= j1; ++j) {
            const float x = v[(size_t)j * HD];
#pragma unroll
            for (int h = 0; h < HV; ++h) acc[h] = __fmaf_rn(ps[(part + kParts * h) * 128 + 64 * p + j], x, acc[h]);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < HV; ++h) {
        const int head = part + kParts * h;
        if (head >= G) continue;
        float* dst = a.scratch + (((size_t)seq * a.heads + kh * G + head) * a.chunks + chunk) * (HD + 2);
        dst[c] = acc[h];
        if (c == 0) { dst[HD] = m_s[head]; dst[HD + 1] = l_s[head]; }
      }
    }
    __syncthreads();
  }
}

// The chunks of one (sequence, head), in ascending order; a thread a channel.
template <int HD>
__global__ void __launch_bounds__(HD) attn_f32_join_kernel(AttnF32Args a) {
  pdl_enter();
  const int head = blockIdx.x, seq = blockIdx.y, c = threadIdx.x;
  const int pos = a.past[seq], lo = first_key(pos, a.window);
  const float* src = a.scratch + ((size_t)seq * a.heads + head) * a.chunks * (HD + 2);
  float M = -INFINITY, L = 0.0f, o = 0.0f;
#pragma unroll 4
  for (int chunk = lo / 128; chunk <= pos / 128; ++chunk) {
    const float* p = src + (size_t)chunk * (HD + 2);
    float fa, fb;
    const float acc = p[c];
    join_factors(p[HD], p[HD + 1], M, L, fa, fb);
    o = join_value(acc, o, fa, fb);
  }
  a.out[((size_t)a.seq_start[seq] * a.heads + head) * HD + c] = __fmul_rn(o, last_factor(a.sinks, head, M, L));
}

template <int HD, int GP>
static int launch_token(const AttnF32Args& a, cudaStream_t s) {
  constexpr int smem = token_smem<HD, GP>();
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)attn_f32_token_kernel<HD, GP>, smem, allowed);
  if (e != cudaSuccess) return fail(2, "attention_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  // about four blocks an SM; a block with several chunks takes them in turn
  const int pairs = a.n_seqs * a.kv_heads;
  int z = (4 * sm_count() + pairs - 1) / pairs;
  if (z > a.chunks) z = a.chunks;
  launch(attn_f32_token_kernel<HD, GP>, dim3(a.kv_heads, a.n_seqs, z), dim3(256), smem, s, a);
  launch(attn_f32_join_kernel<HD>, dim3(a.heads, a.n_seqs), dim3(HD), 0, s, a);
  return check_launch("attention_f32 (single tokens)");
}

template <int HD>
static int launch_f32(const AttnF32Args& a, int max_count, cudaStream_t s) {
  const int G = a.heads / a.kv_heads;
  if (max_count == 1) {
    if (G <= 2) return launch_token<HD, 2>(a, s);
    if (G <= 4) return launch_token<HD, 4>(a, s);
    if (G <= 8) return launch_token<HD, 8>(a, s);
    return launch_token<HD, 16>(a, s);
  }
  constexpr int smem = prompt_smem<HD>();
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)attn_f32_prompt_kernel<HD>, smem, allowed);
  if (e != cudaSuccess) return fail(2, "attention_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  const int tile_tokens = kRows / G, tiles = (max_count + tile_tokens - 1) / tile_tokens;
  SLB_REQUIRE(tiles < 65536 && a.n_seqs < 65536, "attention_f32: %d tiles, %d sequences", tiles, a.n_seqs);
  launch(attn_f32_prompt_kernel<HD>, dim3(a.kv_heads, a.n_seqs, tiles), dim3(256), smem, s, a);
  return check_launch("attention_f32 (many tokens)");
}

}  // namespace slb

using namespace slb;

// Float32 attention for heads of 64 or 128 channels, up to 16 query heads per kv head. Sequence i brings counts[i] tokens at
// rows seq_start[i].. with positions past[i]..; max_count is the largest count. With max_count 1 scratch holds
// n_seqs * heads * chunks * (head_dim + 2) floats, chunks = ceil(table_stride / 2).
extern "C" int slb_attention_f32(const float* q, const float* k_pool, const float* v_pool, float* out, const int* seq_start,
                                 const int* past, const int* counts, const int* block_table, int table_stride, int n_seqs,
                                 int max_count, int heads, int kv_heads, int head_dim, int window, float scale,
                                 const float* sinks, float* scratch, long long scratch_floats, void* stream) {
  SLB_REQUIRE(n_seqs >= 0 && max_count >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && heads / kv_heads <= kMostGroup,
              "attention_f32: n_seqs=%d heads=%d kv_heads=%d", n_seqs, heads, kv_heads);
  SLB_REQUIRE(head_dim == 64 || head_dim == 128, "attention_f32: head_dim %d is not supported (64 or 128)", head_dim);
  SLB_REQUIRE(window > -(1 << 30) && table_stride > 0, "attention_f32: window=%d table_stride=%d", window, table_stride);
  SLB_REQUIRE((uintptr_t)q % 16 == 0 && (uintptr_t)k_pool % 16 == 0 && (uintptr_t)v_pool % 16 == 0 && (uintptr_t)out % 16 == 0,
              "attention_f32: q, out and the pools must be 16-byte aligned");
  if (n_seqs == 0 || max_count == 0) return 0;
  SLB_REQUIRE(kv_heads < 65536 && heads < 65536 && n_seqs < 65536, "attention_f32: n_seqs=%d heads=%d", n_seqs, heads);
  const int chunks = (table_stride + kChunkPages - 1) / kChunkPages;
  SLB_REQUIRE(max_count > 1 || (scratch != nullptr && scratch_floats >= (long long)n_seqs * heads * chunks * (head_dim + 2)),
              "attention_f32: single tokens need %lld floats of scratch, got %lld",
              (long long)n_seqs * heads * chunks * (head_dim + 2), scratch_floats);
  const AttnF32Args a{q, k_pool, v_pool, out, seq_start, past, counts, block_table, table_stride, n_seqs, heads, kv_heads, window,
                      scale, sinks, scratch, chunks};
  return head_dim == 128 ? launch_f32<128>(a, max_count, (cudaStream_t)stream) : launch_f32<64>(a, max_count, (cudaStream_t)stream);
}
