// Causal grouped-query attention over the paged cache in true float32 (no tensor cores), heads of 64 or 128 channels:
// one kernel for steps of many tokens, one for steps of few (up to 16 rows a group: a token's query heads are rows), and a short
// kernel that joins what their blocks found where several blocks share a sequence's keys.
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
// prompts of 400 tokens 2,034 / 197, single tokens at a context of 700 (batch 8) 41 / 16, at 4,000 (batch 1) 184 / 23. Portions (cold caches),
// the general kernel / tiles of 64 rows walking all keys / now: 2 tokens on 4,000 keys 366 / 606 / 40, 32 391 / 610 / 67; 64 sequences of 2 on 500
// 239 / 281 / 108. Where the general kernel was as fast: up to a dozen keys in all (12 against 13), 16 query heads a group on less than 60 (11 / 22).
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
  float* scratch;        // with several slices: per (chunk, row of the step, head) hd weighted values, maximum, sum
  int tile_rows;         // many tokens: rows of a block's tile, 64 or (where SMs are idle) 32
  int slices;            // blocks that share a sequence's chunks, each every slices-th of them
  int rows;              // scratch rows a chunk: sequences in steps of single tokens, else token rows
  int row_is_sequence;
};

// Where the results of one chunk wait for the joining kernel. Chunk by chunk, so that what a step writes lies together however long
// a sequence may become (a row's chunks side by side: 64 tokens on 60 keys 56 us where up to 40,960 keys are allowed, unsliced 33).
template <int HD>
__device__ __forceinline__ float* chunk_slot(const AttnF32Args& a, int seq, size_t token, int head, int chunk) {
  return a.scratch + (((size_t)chunk * a.rows + (a.row_is_sequence ? (size_t)seq : token)) * a.heads + head) * (HD + 2);
}

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
// A page costs a block 9 us at 128 channels, so a portion on a long past whose tiles leave SMs idle is cut along its keys (SLICED):
// a block takes every slices-th chunk and leaves each chunk's results in scratch.
constexpr int kRows = 64;
template <int HD> constexpr int prompt_smem() { return (3 * 64 * HD + 64 * 64 + 3 * 64) * 4; }

template <int HD>
__device__ __forceinline__ int swz(int row, int group) { return row * HD + ((group ^ (row & 7)) << 2); }

template <int HD, bool SLICED>
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
  const int G = a.heads / a.kv_heads, tile_tokens = a.tile_rows / G;
  const int kh = blockIdx.x, seq = blockIdx.y;
  const int count = a.counts[seq];
  // the longest tiles first, and the slices that every tile has before those that may be empty: the blocks with work get SMs of their own
  const int slices = SLICED ? a.slices : 1, tiles = gridDim.z / slices, slice = SLICED ? blockIdx.z / tiles : 0;
  const int tile = tiles - 1 - (SLICED ? blockIdx.z % tiles : blockIdx.z);
  const int t0 = tile * tile_tokens;
  if (t0 >= count) return;
  const int tokens = min(tile_tokens, count - t0), rows = tokens * G;
  const int pos0 = a.past[seq] + t0, pos1 = pos0 + tokens - 1;
  const size_t token0 = (size_t)a.seq_start[seq] + t0;
  const int* table = a.block_table + (size_t)seq * a.table_stride;

  const int page_hi = pos1 / kPageTokens;
  int page_lo = first_key(pos0, a.window) / kPageTokens;
  if (SLICED) {
    page_lo = max(page_lo, (page_lo / kChunkPages + slice) * kChunkPages);
    if (page_lo > page_hi) return;
  }
  auto after = [&](int page) { return SLICED && page % kChunkPages == kChunkPages - 1 ? page + 1 + (slices - 1) * kChunkPages : page + 1; };
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
  // (the warps of tokens that do not exist have nothing to do; those that do lie on different quarters of the SM)
  const int r0 = (warp >> 1) * 16 + (lane >> 3), c0 = (warp & 1) * 32 + (lane & 7);
  const int o0 = (warp & 1) * (HD / 2) + (lane & 7) * 4;
  const bool busy = (warp >> 1) * 16 < rows;
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
  auto put_chunk = [&](int r, int chunk, const f32x2* v) {      // a row's weighted values of a chunk (slots are 8-byte aligned)
    float* slot = chunk_slot<HD>(a, seq, token0 + r / G, kh * G + r % G, chunk);
#pragma unroll
    for (int h = 0; h < CH; ++h) {
      *reinterpret_cast<f32x2*>(slot + o0 + 32 * h) = v[2 * h];
      *reinterpret_cast<f32x2*>(slot + o0 + 32 * h + 2) = v[2 * h + 1];
    }
  };
  // softmax: four threads a row, 16 keys each
  const int sr = tid >> 2, sq = tid & 3;
  float m = -INFINITY, l = 0.0f, M = -INFINITY, L = 0.0f;

  int chunk = page_lo / kChunkPages;
  for (int page = page_lo; page <= page_hi; page = after(page)) {
    const bool new_chunk = page % kChunkPages == 0 && page != page_lo;
    const int coming = after(page);
    const bool masked = page * kPageTokens + kPageTokens - 1 > pos0 || page * kPageTokens < last_lo;
    copies_wait<1>();
    __syncthreads();
    if (busy) {
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
    if (coming <= page_hi) ask_page(ks, a.k_pool, coming, true);
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
        if (SLICED) {
          if (sq == 0 && sr < rows) {
            float* slot = chunk_slot<HD>(a, seq, token0 + sr / G, kh * G + sr % G, chunk);
            slot[HD] = m;
            slot[HD + 1] = l;
          }
        } else {
          float fa, fb;
          join_factors(m, l, M, L, fa, fb);
          if (sq == 0) { fa_s[sr] = fa; fb_s[sr] = fb; }
        }
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
      if (new_chunk && SLICED) {
        if (r < rows) put_chunk(r, chunk, acc[i]);
#pragma unroll
        for (int c = 0; c < 2 * CH; ++c) acc[i][c] = 0;
      } else if (new_chunk) {
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
    if (new_chunk) chunk = page / kChunkPages;
    const int keys = min(kPageTokens, pos1 + 1 - page * kPageTokens);
    if (!busy) {
    } else if (!masked) {
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
    if (coming <= page_hi) ask_page(vs, a.v_pool, coming, false);
    copies_commit();
  }
  copies_wait<0>();
  if (SLICED) {
    if (sq == 0 && sr < rows) {
      float* slot = chunk_slot<HD>(a, seq, token0 + sr / G, kh * G + sr % G, chunk);
      slot[HD] = m;
      slot[HD + 1] = l;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (r0 + 4 * i < rows) put_chunk(r0 + 4 * i, chunk, acc[i]);
    return;
  }
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

// ---- few tokens -----------------------------------------------------------------------------------------------
// A block takes the chunks z, z + gridDim.z, ... of one (sequence, kv head) for all its rows: row r is token r / G, query head r % G
// of the group. Bound by the read of keys and values: a chunk's keys (128 rows, 64 KB at 128 channels) come by asynchronous copies, its
// values are asked into L2 at the same time and read by the threads that own their channel. With several slices each chunk's results
// go to scratch for attn_f32_join_kernel; a block that has a sequence to itself joins them as it goes and needs none.
// GP: rows, rounded up to 2, 4, 8 or 16.
template <int HD, int GP> constexpr int few_smem() { return (128 * HD + GP * HD + GP * 128 + 5 * GP) * 4; }
constexpr int few_blocks(int hd, int gp) { return (hd == 128 ? 3 : 4) - (gp > 8); }      // an SM (shared memory at 128 channels, registers)

template <int HD, int GP>
__global__ void __launch_bounds__(256, few_blocks(HD, GP)) attn_f32_few_kernel(AttnF32Args a) {
  pdl_enter();
  extern __shared__ __align__(16) float smem[];
  float* ks = smem;                    // [128][HD], swizzled
  float* qs = ks + 128 * HD;           // [GP][HD]
  float* ps = qs + GP * HD;            // [GP][128]
  float* alpha_s = ps + GP * 128;      // [GP] of the second page
  float* m_s = alpha_s + GP;
  float* l_s = m_s + GP;
  int* lo_s = reinterpret_cast<int*>(l_s + GP);      // [GP] first and last key that a row sees; none for rows that do not exist
  int* pos_s = lo_s + GP;
  constexpr int kGroups = HD / 4, HQ = GP / 2;
  constexpr int kParts = 256 / HD, HV = GP >= kParts ? GP / kParts : 1;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int G = a.heads / a.kv_heads;
  const int kh = blockIdx.x, seq = blockIdx.y;
  const int count = a.counts[seq], rows = count * G;
  if (count <= 0) return;
  const int pos0 = a.past[seq], pos1 = pos0 + count - 1;
  const int lo0 = first_key(pos0, a.window), lo1 = first_key(pos1, a.window);
  const size_t token0 = a.seq_start[seq];
  const int* table = a.block_table + (size_t)seq * a.table_stride;
  const bool joined = a.slices == 1;
  const int chunk_hi = pos1 / 128;
  int chunk = lo0 / 128 + blockIdx.z;
  if (chunk > chunk_hi) return;
  for (int e = tid; e < GP * HD; e += 256) {
    const int r = e / HD;
    qs[e] = r < rows ? a.q[((token0 + r / G) * a.heads + kh * G + r % G) * HD + e % HD] : 0.0f;
  }
  if (tid < GP) {
    const int pos = tid < rows ? pos0 + tid / G : -1;
    lo_s[tid] = tid < rows ? first_key(pos, a.window) : 0;
    pos_s[tid] = pos;
  }
  float o[HV], M[HV], L[HV];
#pragma unroll
  for (int h = 0; h < HV; ++h) { o[h] = 0.0f; M[h] = -INFINITY; L[h] = 0.0f; }
  const int c = tid % HD, part = tid / HD;         // values: rows part, part + kParts, ... of channel c

  for (; chunk <= chunk_hi; chunk += gridDim.z) {
    const int key0 = chunk * 128, first = max(lo0 - key0, 0), last = min(pos1 - key0, 127);      // keys of the chunk that some row sees
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
      const int key = tid & 127, half = tid >> 7;      // rows half, half + 2, ...
      f32x2 s[HQ];
#pragma unroll
      for (int h = 0; h < HQ; ++h) s[h] = 0;
      if (key >= first && key <= last) {
#pragma unroll 4
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
      for (int h = 0; h < HQ; ++h) {
        const int r = half + 2 * h;
        ps[r * 128 + key] = (key0 + key >= lo_s[r] && key0 + key <= pos_s[r]) ? __fmul_rn(halves_sum(s[h]), a.scale) : -INFINITY;
      }
    }
    __syncthreads();
    for (int r = warp; r < rows; r += 8) {      // one warp a row: the weights of the pages that hold a visible key
      float* row = ps + r * 128;
      float m = -INFINITY, l = 0.0f;
      for (int p = first / 64; p <= last / 64; ++p) {
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
        if (p == 1 && lane == 0) alpha_s[r] = alpha;
      }
      if (lane == 0) { m_s[r] = m; l_s[r] = l; }
    }
    __syncthreads();
    {
      float acc[HV];
#pragma unroll
      for (int h = 0; h < HV; ++h) acc[h] = 0.0f;
      if (part < GP) {
        for (int p = first / 64; p <= last / 64; ++p) {
          const float* v = a.v_pool + ((size_t)table[chunk * kChunkPages + p] * a.kv_heads + kh) * (kPageTokens * HD) + c;
          if (p == 1) {
#pragma unroll
            for (int h = 0; h < HV; ++h) acc[h] = __fmul_rn(acc[h], alpha_s[min(part + kParts * h, rows - 1)]);
          }
          // keys j0 .. j1 are seen by some row, c0 .. c1 by all; sixteen values are asked for together
          const int at = key0 + 64 * p, j0 = max(first - 64 * p, 0), j1 = min(last - 64 * p, 63);
          const int c0 = max(lo1 - at, j0), c1 = min(pos0 - at, j1);
          const float* weights = ps + part * 128 + 64 * p;
          for (int j = j0 & ~15; j <= j1; j += 16) {
            float x[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) x[u] = v[(size_t)min(max(j + u, j0), j1) * HD];
            if (j >= c0 && j + 15 <= c1) {
#pragma unroll
              for (int u = 0; u < 16; u += 4)
#pragma unroll
                for (int h = 0; h < HV; ++h) {
                  const float4 w = *reinterpret_cast<const float4*>(weights + kParts * h * 128 + j + u);
                  acc[h] = __fmaf_rn(w.x, x[u], acc[h]);
                  acc[h] = __fmaf_rn(w.y, x[u + 1], acc[h]);
                  acc[h] = __fmaf_rn(w.z, x[u + 2], acc[h]);
                  acc[h] = __fmaf_rn(w.w, x[u + 3], acc[h]);
                }
            } else {      // each row takes the keys that it sees
#pragma unroll
              for (int h = 0; h < HV; ++h) {
                const int r = part + kParts * h, lo = lo_s[r] - at - j, hi = min(pos_s[r] - at - j, 15);
                const unsigned sees = hi < 0 || lo > 15 ? 0u : (0xffffu >> (15 - hi)) & (0xffffu << max(lo, 0));
#pragma unroll
                for (int u = 0; u < 16; u += 4) {
                  const float4 w = *reinterpret_cast<const float4*>(weights + kParts * h * 128 + j + u);
                  if (sees >> u & 1) acc[h] = __fmaf_rn(w.x, x[u], acc[h]);
                  if (sees >> u & 2) acc[h] = __fmaf_rn(w.y, x[u + 1], acc[h]);
                  if (sees >> u & 4) acc[h] = __fmaf_rn(w.z, x[u + 2], acc[h]);
                  if (sees >> u & 8) acc[h] = __fmaf_rn(w.w, x[u + 3], acc[h]);
                }
              }
            }
          }
        }
      }
#pragma unroll
      for (int h = 0; h < HV; ++h) {
        const int r = part + kParts * h;
        if (r >= rows) continue;
        if (joined) {
          float fa, fb;
          join_factors(m_s[r], l_s[r], M[h], L[h], fa, fb);
          if (m_s[r] != -INFINITY) o[h] = join_value(acc[h], o[h], fa, fb);
        } else {
          float* slot = chunk_slot<HD>(a, seq, token0 + r / G, kh * G + r % G, chunk);
          slot[c] = acc[h];
          if (c == 0) { slot[HD] = m_s[r]; slot[HD + 1] = l_s[r]; }
        }
      }
    }
    __syncthreads();
  }
  if (!joined) return;
#pragma unroll
  for (int h = 0; h < HV; ++h) {
    const int r = part + kParts * h;
    if (r >= rows) continue;
    a.out[((token0 + r / G) * a.heads + kh * G + r % G) * HD + c] = __fmul_rn(o[h], last_factor(a.sinks, kh * G + r % G, M[h], L[h]));
  }
}

// The chunks of one (token, head), in ascending order; a thread a channel.
template <int HD>
__global__ void __launch_bounds__(HD) attn_f32_join_kernel(AttnF32Args a) {
  pdl_enter();
  const int head = blockIdx.x, seq = blockIdx.y, t = blockIdx.z, c = threadIdx.x;
  if (t >= a.counts[seq]) return;
  const int pos = a.past[seq] + t, lo = first_key(pos, a.window);
  const size_t token = (size_t)a.seq_start[seq] + t;
  const float* src = chunk_slot<HD>(a, seq, token, head, 0);
  const size_t stride = (size_t)a.rows * a.heads * (HD + 2);
  float M = -INFINITY, L = 0.0f, o = 0.0f;
#pragma unroll 4
  for (int chunk = lo / 128; chunk <= pos / 128; ++chunk) {
    const float* p = src + chunk * stride;
    float fa, fb;
    const float acc = p[c];
    join_factors(p[HD], p[HD + 1], M, L, fa, fb);
    o = join_value(acc, o, fa, fb);
  }
  a.out[(token * a.heads + head) * HD + c] = __fmul_rn(o, last_factor(a.sinks, head, M, L));
}

// How a step is cut: which kernel, into how many slices, and the scratch that takes.
struct F32Plan {
  bool few;
  int tile_rows, slices, rows;
  long long floats;
};
constexpr long long kMostScratch = 1ll << 26;      // floats (256 MB): beyond, blocks keep a sequence to themselves

static F32Plan plan_f32(int n_seqs, long long tokens, int max_count, int heads, int kv_heads, int head_dim, int table_stride, int max_keys) {
  F32Plan p;
  const int G = heads / kv_heads;
  const long long sms = sm_count();
  p.tile_rows = kRows;
  p.few = (long long)max_count * G <= kMostGroup;
  long long chunks = (table_stride + kChunkPages - 1) / kChunkPages;
  if (max_keys > 0 && (max_keys + 127) / 128 < chunks) chunks = (max_keys + 127) / 128;
  long long slices;
  if (p.few) {                     // about four blocks an SM; a block with several chunks takes them in turn
    // (four fit at 64 channels, and no more than fit; at 128 three, and shorter blocks even out the second round: 64 sequences of 500
    // keys in one / two slices 52 / 58 us at 64 channels, 101 / 93 at 128)
    const long long pairs = (long long)n_seqs * kv_heads;
    slices = (4 * sms + (head_dim == 128 ? pairs - 1 : 0)) / pairs;
  } else {                         // as many as two blocks an SM take at once
    auto blocks = [&](int tile_rows) { return (long long)n_seqs * kv_heads * ((max_count + tile_rows / G - 1) / (tile_rows / G)); };
    if (blocks(kRows / 2) <= sms) p.tile_rows = kRows / 2;      // half a tile takes two thirds of its time (32 tokens on 60 keys, G = 2: 38 -> 28 us)
    slices = 2 * sms / blocks(p.tile_rows);
  }
  if (slices > chunks) slices = chunks;
  p.rows = max_count == 1 ? n_seqs : (int)tokens;
  p.floats = (long long)p.rows * heads * chunks * (head_dim + 2);
  if (slices <= 1 || p.floats > kMostScratch) { slices = 1; p.floats = 0; }
  p.slices = (int)slices;
  return p;
}

template <int HD, int GP>
static int launch_few(const AttnF32Args& a, cudaStream_t s) {
  constexpr int smem = few_smem<HD, GP>();
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)attn_f32_few_kernel<HD, GP>, smem, allowed);
  if (e != cudaSuccess) return fail(2, "attention_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  launch(attn_f32_few_kernel<HD, GP>, dim3(a.kv_heads, a.n_seqs, a.slices), dim3(256), smem, s, a);
  return check_launch("attention_f32 (few tokens)");
}

template <int HD, bool SLICED>
static int launch_prompt(const AttnF32Args& a, int max_count, cudaStream_t s) {
  constexpr int smem = prompt_smem<HD>();
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)attn_f32_prompt_kernel<HD, SLICED>, smem, allowed);
  if (e != cudaSuccess) return fail(2, "attention_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
  const int tile_tokens = a.tile_rows / (a.heads / a.kv_heads), tiles = (max_count + tile_tokens - 1) / tile_tokens;
  SLB_REQUIRE(tiles < 65536 && a.n_seqs < 65536, "attention_f32: %d tiles, %d sequences", tiles, a.n_seqs);
  launch(attn_f32_prompt_kernel<HD, SLICED>, dim3(a.kv_heads, a.n_seqs, tiles * a.slices), dim3(256), smem, s, a);
  return check_launch("attention_f32 (many tokens)");
}

template <int HD>
static int launch_f32(const AttnF32Args& a, bool few, int max_count, cudaStream_t s) {
  const int rows = max_count * (a.heads / a.kv_heads);
  int rc;
  if (!few) rc = a.slices > 1 ? launch_prompt<HD, true>(a, max_count, s) : launch_prompt<HD, false>(a, max_count, s);
  else if (rows <= 2) rc = launch_few<HD, 2>(a, s);
  else if (rows <= 4) rc = launch_few<HD, 4>(a, s);
  else if (rows <= 8) rc = launch_few<HD, 8>(a, s);
  else rc = launch_few<HD, 16>(a, s);
  if (rc || a.slices == 1) return rc;
  SLB_REQUIRE(max_count < 65536, "attention_f32: %d tokens a sequence", max_count);
  launch(attn_f32_join_kernel<HD>, dim3(a.heads, a.n_seqs, max_count), dim3(HD), 0, s, a);
  return check_launch("attention_f32 (join)");
}

}  // namespace slb

using namespace slb;

// Floats of scratch with which slb_attention_f32 cuts a step of n_seqs sequences, `tokens` rows and at most max_count tokens a sequence
// along its keys; 0 where it does not. max_keys: no sequence has more keys after the step (0: the table's width bounds them).
extern "C" long long slb_attention_f32_scratch(int n_seqs, int tokens, int max_count, int heads, int kv_heads, int head_dim, int table_stride,
                                               int max_keys) {
  if (n_seqs <= 0 || max_count <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || heads / kv_heads > kMostGroup || table_stride <= 0) return 0;
  return plan_f32(n_seqs, tokens, max_count, heads, kv_heads, head_dim, table_stride, max_keys).floats;
}

// Float32 attention for heads of 64 or 128 channels, up to 16 query heads per kv head. Sequence i brings counts[i] tokens at
// rows seq_start[i].. with positions past[i]..; max_count is the largest count, `tokens` the rows of q. Scratch as
// slb_attention_f32_scratch says; steps of more than one token a sequence run without it too, on fewer SMs.
extern "C" int slb_attention_f32(const float* q, const float* k_pool, const float* v_pool, float* out, const int* seq_start,
                                 const int* past, const int* counts, const int* block_table, int table_stride, int n_seqs, int tokens,
                                 int max_count, int max_keys, int heads, int kv_heads, int head_dim, int window, float scale,
                                 const float* sinks, float* scratch, long long scratch_floats, void* stream) {
  SLB_REQUIRE(n_seqs >= 0 && tokens >= 0 && max_count >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && heads / kv_heads <= kMostGroup,
              "attention_f32: n_seqs=%d heads=%d kv_heads=%d", n_seqs, heads, kv_heads);
  SLB_REQUIRE(head_dim == 64 || head_dim == 128, "attention_f32: head_dim %d is not supported (64 or 128)", head_dim);
  SLB_REQUIRE(window > -(1 << 30) && table_stride > 0, "attention_f32: window=%d table_stride=%d", window, table_stride);
  SLB_REQUIRE((uintptr_t)q % 16 == 0 && (uintptr_t)k_pool % 16 == 0 && (uintptr_t)v_pool % 16 == 0 && (uintptr_t)out % 16 == 0,
              "attention_f32: q, out and the pools must be 16-byte aligned");
  SLB_REQUIRE((uintptr_t)scratch % 8 == 0, "attention_f32: scratch must be 8-byte aligned");
  if (n_seqs == 0 || max_count == 0) return 0;
  SLB_REQUIRE(kv_heads < 65536 && heads < 65536 && n_seqs < 65536, "attention_f32: n_seqs=%d heads=%d", n_seqs, heads);
  F32Plan plan = plan_f32(n_seqs, tokens, max_count, heads, kv_heads, head_dim, table_stride, max_keys);
  const bool enough = plan.floats == 0 || (scratch != nullptr && scratch_floats >= plan.floats);
  SLB_REQUIRE(max_count > 1 || enough, "attention_f32: single tokens need %lld floats of scratch, got %lld", plan.floats, scratch_floats);
  if (!enough) plan.slices = 1;
  const AttnF32Args a{q, k_pool, v_pool, out, seq_start, past, counts, block_table, table_stride, n_seqs, heads, kv_heads, window,
                      scale, sinks, scratch, plan.tile_rows, plan.slices, plan.rows, max_count == 1};
  return head_dim == 128 ? launch_f32<128>(a, plan.few, max_count, (cudaStream_t)stream) : launch_f32<64>(a, plan.few, max_count, (cudaStream_t)stream);
}
