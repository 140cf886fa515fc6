// The 32-bit matrix product on the tensor cores: C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]), float32 in, float32 out.
//
// A float32 value is the sum of three bfloat16 values exactly (8 + 8 + 8 bits of its 24): x = x1 + x2 + x3 with x1 = bf16(x),
// x2 = bf16(x - x1), x3 = x - x1 - x2, |x2| <= 2^-8 |x|, |x3| <= 2^-16 |x|. A product of two bfloat16 values is exact in float32, so a
// float32 product is w1 a1 + (w1 a2 + w2 a1) + (w1 a3 + w2 a2 + w3 a1) and parts of either sign below 2^-24 of it, typically 2^-27,
// which are left out: six tcgen05 products of kind f16 in place of one FMA a value (splitting into exact partial products:
// Dekker, 1971; Ozaki et al., 2012).
//
// Order of the sums: K is cut into chunks of 64. A chunk's six products are summed by the tensor core, the small ones first, so that
// of the 24 instructions only the last four add at full size (its float32 sums are truncated, half a unit each on average). A chunk's
// sum is then taken out of tensor memory, and the chunks' sums are added in float32, rounded to nearest, in ascending order:
//     C = ((chunk 0 + chunk 1) + chunk 2) + ...   (+ bias, then added to the old value)
// Every form below does exactly this, whatever tile it takes, however many blocks share K and whatever M is, so that a row's bits
// depend neither on the rows beside it nor on how a sequence was cut into steps. Which products come here depends on W alone
// (ops.f32_on_tensor_cores). Against the FMA kernels' chains of K / 8 roundings the sums are shorter. Error (2-norm, against 64 bits),
// FMA chains / here: K 256 2.1e-7 / 0.9e-7, 1,024 2.1e-7 / 1.1e-7, 3,072 3.6e-7 / 1.5e-7, 9,728 6.3e-7 / 2.4e-7.
// A result that is not finite (infinite or NaN operands, whose parts are NaN; a sum beyond the range) is formed again as one FMA chain.
//
// One block: 128 features (the instruction's rows, so that few tokens waste nothing) by NT tokens. Per chunk, for the unit u:
//   * the last warp asks TMA for the raw 128 x 64 weights, a ring of R chunks ahead;
//   * eight or sixteen warps split them into tensor memory (operand A of the instruction) and the tokens' values, which they have fetched a
//     unit ahead into registers, into shared memory in the 128-byte swizzle (operand B), both double-buffered; while unit u is
//     multiplied they take the sums of unit u - 1 out of tensor memory (double-buffered too), add them in registers and split unit u + 1;
//   * one more warp issues the 24 instructions.
// Blocks of a cluster may share a tile's K (few tokens: the weights' stream wants all SMs): each sends its chunks' sums as they come to
// the block that owns the feature, through distributed shared memory, and each adds up its features, all chunks in order. The first
// chunk of weights is split before the wait for the kernel in front.
#include "packed_f32.cuh"
#include "tcgen05.cuh"

namespace slb {

constexpr int kFtChunk = 64, kFtFeatures = 128, kFtRaw = kFtFeatures * kFtChunk * 4;

struct GemmF32TcArgs {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int M, N, K, lda, ldw, ldc, accumulate;
  int early;             // no kernel writes W: it is fetched before the wait for the kernel in front
  int vec;               // A's rows can be read 16 bytes at a time
  int rows;              // tokens of a tile (NT; fewer where the chunks' sums of NT would not fit shared memory)
  int splits;            // blocks that share a tile's K (the cluster's size)
  int m_tiles;           // tiles of a.rows tokens
  GateAct gate;          // GATED: W holds N gate rows, then N up rows; C = act(gate) * up
  int* status;
};

// NT tokens, WORKERS warps that split and add.
template <int NT, int WORKERS>
struct FtShape {
  static constexpr int kThreads = (WORKERS + 2) * 32;
  static constexpr int kPlane = NT * 128;                  // bytes: NT rows of 64 bfloat16
  static constexpr int kB = 2 * 3 * kPlane;
  static constexpr int kParts = WORKERS / 4;               // warps that share a quarter of tensor memory's lanes
  static constexpr int kOut = NT / kParts;                 // columns of a worker thread
  static constexpr int kPieces = 16 / kParts;              // 16-byte pieces of a feature's chunk that a worker thread splits
  static constexpr int kRowsAPass = WORKERS * 4;           // tokens whose values the workers split at once
  static constexpr int kPasses = NT > kRowsAPass ? NT / kRowsAPass : 1;
  static constexpr int kColumns = 2 * NT + 192 > 256 ? 512 : 256;
};
// Shared memory: the ring, the tokens' parts, and the chunks' sums (K shared) or the up values on their way to the gate values.
__host__ __device__ constexpr int ft_smem(int nt, int ring, int chunks, int rows, bool gated = false) {
  return ring * kFtRaw + 2 * 3 * nt * 128 + (chunks > 0 ? chunks * rows * kFtFeatures * 4 : gated ? nt * kFtFeatures * 2 : 0) + 256 + 1024;
}

// Two values into their three parts, packed as the tensor core reads them (the first in the low half).
__device__ __forceinline__ void split2(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  const f32x2 minus = both(-1.0f);
  auto pack = [](f32x2 w) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(low_half(w), high_half(w));
    return *reinterpret_cast<const uint32_t*>(&b);
  };
  auto rest = [&](uint32_t p) {      // what the parts leave, exactly
    f32x2 h;
    asm("mov.b64 %0, {%1, %2};" : "=l"(h) : "r"(p << 16), "r"(p & 0xffff0000u));
    v = fma2(h, minus, v);
  };
  p1 = pack(v);
  rest(p1);
  p2 = pack(v);
  rest(p2);
  p3 = pack(v);
}

__device__ __forceinline__ void tmem_st8_nowait(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_ld4_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
// N consecutive columns of this warp's lanes, all there on return.
template <int N>
__device__ __forceinline__ void ft_take_out(uint32_t taddr, uint32_t (&r)[N]) {
  if constexpr (N == 4) tmem_ld4_nowait(taddr, r);
  else if constexpr (N == 8) tmem_ld8_nowait(taddr, r);
  else {
#pragma unroll
    for (int j = 0; j < N; j += 16) tmem_ld16_nowait(taddr + j, r + j);
  }
  tmem_wait_ld();
}

// The result of one output in plain float32, for results that are not finite.
__device__ __noinline__ float ft_plain_dot(const GemmF32TcArgs& a, int m, int n) {
  float v = 0.0f;
  for (int k = 0; k < a.K; ++k) v = fmaf(a.A[(size_t)m * a.lda + k], a.W[(size_t)n * a.ldw + k], v);
  return v;
}
__device__ __forceinline__ float ft_checked(const GemmF32TcArgs& a, int m, int n, float v) { return isfinite(v) ? v : ft_plain_dot(a, m, n); }
__device__ __forceinline__ float ft_old(const GemmF32TcArgs& a, int m, int n) { return a.accumulate ? a.C[(size_t)m * a.ldc + n] : 0.0f; }
__device__ __forceinline__ void ft_store(const GemmF32TcArgs& a, int m, int n, float v, float old) {
  v = ft_checked(a, m, n, v);
  if (a.bias) v += a.bias[n];
  a.C[(size_t)m * a.ldc + n] = a.accumulate ? old + v : v;
}

// A chunk's 24 products: the small ones first. wa: the three parts of W in tensor memory, 32 columns each; x1, x2, x3: the tokens' parts.
__device__ __forceinline__ void ft_multiply(uint32_t d, uint32_t wa, uint64_t x1, uint64_t x2, uint64_t x3, uint32_t idesc) {
#pragma unroll
  for (int k4 = 0; k4 < 4; ++k4) {
    mma_bf16_ts(d, wa + 64 + k4 * 8, x1 + k4 * 2, idesc, k4 > 0 ? 1u : 0u);
    mma_bf16_ts(d, wa + k4 * 8, x3 + k4 * 2, idesc, 1u);
    mma_bf16_ts(d, wa + 32 + k4 * 8, x2 + k4 * 2, idesc, 1u);
  }
#pragma unroll
  for (int k4 = 0; k4 < 4; ++k4) {
    mma_bf16_ts(d, wa + 32 + k4 * 8, x1 + k4 * 2, idesc, 1u);
    mma_bf16_ts(d, wa + k4 * 8, x2 + k4 * 2, idesc, 1u);
  }
#pragma unroll
  for (int k4 = 0; k4 < 4; ++k4) mma_bf16_ts(d, wa + k4 * 8, x1 + k4 * 2, idesc, 1u);
}

// Waits for the cluster's sums and forms this block's share of the outputs: its features, from n0 + rank * share on, for the tile's tokens.
// Called by all threads of all blocks; no block's shared memory is read by others after it.
template <bool GATED, int THREADS>
__device__ __forceinline__ void ft_add_up(const GemmF32TcArgs& a, const float* sums, int chunks_all, int mine, int m0, int live, int n0, int rank) {
  const int tid = threadIdx.x, cols = GATED ? mine / 2 : mine, outputs = live * cols;
  n0 += rank * cols;
  float old = !GATED && tid < outputs && n0 + tid % cols < a.N ? ft_old(a, m0 + tid / cols, n0 + tid % cols) : 0.0f;
  cluster_sync_all();
  for (int i = tid; i < outputs; i += THREADS) {
    const int t = i / cols, f = i % cols, m = m0 + t, n = n0 + f;
    if (n >= a.N) continue;
    auto total_of = [&](int at) {
      float v = 0.0f;
#pragma unroll 8
      for (int g = 0; g < chunks_all; ++g) v += sums[(g * a.rows + t) * mine + at];
      return v;
    };
    if constexpr (GATED) {
      const float g = ft_checked(a, m, n, total_of(f)), up = ft_checked(a, m, a.N + n, total_of(cols + f));
      a.C[(size_t)m * a.ldc + n] = gated(a.gate, g, up);
    } else {
      if (i != tid) old = ft_old(a, m, n);
      ft_store(a, m, n, total_of(f), old);
    }
  }
}

// GATED: a tile is 64 gate rows of W and the 64 up rows that match them. SPLIT: K is shared by a cluster, which has one tile.
template <int NT, int R, int WORKERS, bool SPLIT, bool GATED>
__global__ void __launch_bounds__(FtShape<NT, WORKERS>::kThreads, WORKERS == 8 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, GemmF32TcArgs a) {
  using S = FtShape<NT, WORKERS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = smem + R * kFtRaw;
  unsigned char* after = planes + S::kB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(after);      // full[R], empty[R], ready[2], done[2], up values there, up values read; then the tensor memory's address
  // SPLIT: [chunk][token][feature], of this block's share of the features (of GATED tiles, of the gate rows and then of the up rows that
  // match them); else GATED: the up values [token][64]
  float* sums = reinterpret_cast<float*>(after + 256);
  constexpr int kCols = GATED ? kFtFeatures / 2 : kFtFeatures;      // of C in a tile
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * R, ready0 = empty0 + 8 * R, done0 = ready0 + 16, up_there = done0 + 16, up_read = up_there + 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * R + 6);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int n_tiles = (a.N + kCols - 1) / kCols, m_tiles = (a.M + a.rows - 1) / a.rows, total = n_tiles * m_tiles;
  const int chunks_all = (a.K + kFtChunk - 1) / kFtChunk;
  const int rank = SPLIT ? (int)cluster_ctarank() : 0, shares = SPLIT ? a.splits : 1;
  const int per = (chunks_all + shares - 1) / shares;       // chunks of a share
  const int c_first = rank * per, chunks = max(0, min(per, chunks_all - c_first));
  const int worker = SPLIT ? (int)blockIdx.x / shares : (int)blockIdx.x, n_workers = SPLIT ? (int)gridDim.x / shares : (int)gridDim.x;
  const int my_tiles = worker < total ? (total - worker + n_workers - 1) / n_workers : 0;
  const int units = my_tiles * chunks;

  if (tid == 0) {
    for (int s = 0; s < R; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, WORKERS);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(ready0 + 8 * i, WORKERS);
      mbar_init(done0 + 8 * i, 1);
    }
    mbar_init(up_there, WORKERS / 2);
    mbar_init(up_read, WORKERS / 2);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(S::kColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot, tA = tmem + 2 * NT;
  if (SPLIT) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (no sums go to a block that has not begun)
  pdl_launch_dependents();
  const int mine = kFtFeatures / shares;                    // features of an output share

  if (warp == WORKERS + 1) {
    if (elect_one()) {
      if (!a.early) pdl_wait();
      int tile = worker, c = 0;
      for (int u = 0; u < units; ++u) {
        const int s = u % R;
        if (u >= R && !mbar_wait(empty0 + 8 * s, ((u / R) - 1) & 1)) { atomicExch(a.status, 61); break; }
        const int n0 = (tile / m_tiles) * kCols, n1 = GATED ? a.N + n0 : n0 + 64, k0 = (c_first + c) * kFtChunk;
        mbar_expect_tx(full0 + 8 * s, kFtRaw);
        const uint32_t dst = smem_addr(smem) + s * kFtRaw;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tma_load_2d(dst + h * (kFtRaw / 2), &map_w, k0 + 32 * h, n0, full0 + 8 * s);
          tma_load_2d(dst + h * (kFtRaw / 2) + kFtRaw / 4, &map_w, k0 + 32 * h, n1, full0 + 8 * s);
        }
        if (++c == chunks) { c = 0; tile += n_workers; }
      }
    }
  } else if (warp == WORKERS) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(kFtFeatures, NT);
      for (int u = 0; u < units; ++u) {
        const int b = u & 1;
        if (!mbar_wait(ready0 + 8 * b, (u >> 1) & 1)) { atomicExch(a.status, 62); break; }
        tc_fence_after();
        const uint32_t d = tmem + b * NT, wa = tA + b * 96;
        const uint64_t x1 = smem_desc(smem_addr(planes) + b * 3 * S::kPlane), x2 = x1 + S::kPlane / 16, x3 = x2 + S::kPlane / 16;
        ft_multiply(d, wa, x1, x2, x3, idesc);
        mma_commit(done0 + 8 * b);
      }
    }
  } else {
    const int quad = warp & 3, part = warp >> 2;             // tensor memory's lanes; a share of the chunk's k values and of the tile's tokens
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const int b_row = tid >> 3, b_k = (tid & 7) * 8;         // this thread's row of each pass of tokens and its eight k values
    float raw[S::kPasses][8];
    const float* rows_at[S::kPasses];
    uint32_t there = 0;                                      // bit p: this thread's row of pass p exists
    auto aim = [&](int tile) {
      const int m0 = (tile % m_tiles) * a.rows, m_end = min(a.M, m0 + a.rows);
      there = 0;
#pragma unroll
      for (int p = 0; p < S::kPasses; ++p) {
        const int m = m0 + S::kRowsAPass * p + b_row;
        if (m < m_end) there |= 1u << p;
        rows_at[p] = a.A + (size_t)min(m, a.M - 1) * a.lda + c_first * kFtChunk + b_k;
      }
    };
    auto fetch_tokens = [&](int c) {
      const int left = a.K - (c_first + c) * kFtChunk - b_k;
#pragma unroll
      for (int p = 0; p < S::kPasses; ++p) {
        const float* src = rows_at[p] + c * kFtChunk;
        if (a.vec && left >= 8) {
          float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
          if (there >> p & 1u) {
            lo = *reinterpret_cast<const float4*>(src);
            hi = *reinterpret_cast<const float4*>(src + 4);
          }
          *reinterpret_cast<float4*>(raw[p]) = lo;
          *reinterpret_cast<float4*>(raw[p] + 4) = hi;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) raw[p][e] = (there >> p & 1u) && e < left ? src[e] : 0.0f;
        }
      }
    };
    float acc[S::kOut];
#pragma unroll
    for (int j = 0; j < S::kOut; ++j) acc[j] = 0.0f;
    int tile = worker, c = 0;                                // of unit u
    int d_tile = worker, d_c = 0;                            // of the unit that is taken out
    bool ok = true;
    auto split_tokens = [&](int b) {       // 8 lanes a row, 4 rows a store, which the swizzle spreads over all banks
      if (NT < S::kRowsAPass && b_row >= NT) return;
      unsigned char* dst = planes + b * 3 * S::kPlane + b_row * 128 + ((((tid & 7) ^ b_row) & 7) << 4);
#pragma unroll
      for (int p = 0; p < S::kPasses; ++p) {
        uint4 q1, q2, q3;
        split2(raw[p][0], raw[p][1], q1.x, q2.x, q3.x);
        split2(raw[p][2], raw[p][3], q1.y, q2.y, q3.y);
        split2(raw[p][4], raw[p][5], q1.z, q2.z, q3.z);
        split2(raw[p][6], raw[p][7], q1.w, q2.w, q3.w);
        unsigned char* at = dst + p * S::kRowsAPass * 128;
        *reinterpret_cast<uint4*>(at) = q1;
        *reinterpret_cast<uint4*>(at + S::kPlane) = q2;
        *reinterpret_cast<uint4*>(at + 2 * S::kPlane) = q3;
      }
    };
    auto split_weights = [&](int u) {      // lane = feature, this warp's share of the chunk's k values
      const int b = u & 1, s = u % R, row = quad * 32 + lane;
      ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (u / R) & 1));
      if (!ok) {
        if (lane == 0) atomicExch(a.status, 63);
        return;
      }
#pragma unroll
      for (int j0 = 0; j0 < S::kPieces; j0 += 4) {
        const int piece = part * S::kPieces + j0;            // of the chunk's sixteen a feature; eight lie side by side
        const unsigned char* src = smem + s * kFtRaw + (piece >> 3) * (kFtRaw / 2) + row * 128;
        uint32_t w1[8], w2[8], w3[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(src + ((((piece & 7) + j) ^ (row & 7)) << 4));
          split2(v.x, v.y, w1[2 * j], w2[2 * j], w3[2 * j]);
          split2(v.z, v.w, w1[2 * j + 1], w2[2 * j + 1], w3[2 * j + 1]);
        }
        const uint32_t wa = tA + lanes + b * 96 + piece * 2;
        tmem_st8_nowait(wa, w1);
        tmem_st8_nowait(wa + 32, w2);
        tmem_st8_nowait(wa + 64, w3);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * s);
    };
    if (units) split_weights(0);           // (the kernel in front may still be running)
    pdl_wait();
    if (SPLIT) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (units) {
      aim(tile);
      fetch_tokens(c);
    }
    for (int u = 0; u <= units && ok; ++u) {
      if (u < units) {
        split_tokens(u & 1);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        fence_smem_to_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready0 + 8 * (u & 1));
        if (++c == chunks) {
          c = 0;
          tile += n_workers;
          if (u + 1 < units) aim(tile);
        }
        if (u + 1 < units) fetch_tokens(c);
      }
      if (u >= 1) {
        const int v = u - 1, b = v & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(done0 + 8 * b, (v >> 1) & 1));
        if (!ok) {
          if (lane == 0) atomicExch(a.status, 64);
          break;
        }
        tc_fence_after();
        uint32_t r[S::kOut];
        ft_take_out<S::kOut>(tmem + lanes + b * NT + part * S::kOut, r);
        if constexpr (SPLIT) {             // to the block that adds up this feature
          const int live = min(a.rows, a.M - (worker % m_tiles) * a.rows) - part * S::kOut, f = quad * 32 + lane;
          const int half = mine / 2, owner = GATED ? (f & 63) / half : f / mine, at_f = GATED ? (f >> 6) * half + (f & 63) % half : f % mine;
          const uint32_t at = cluster_map(smem_addr(sums) + (uint32_t)((((c_first + v) * a.rows + part * S::kOut) * mine + at_f) * 4), (uint32_t)owner);
#pragma unroll
          for (int j = 0; j < S::kOut; ++j)
            if (j < live) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(at + (uint32_t)(j * mine * 4)), "r"(r[j]) : "memory");
        } else {
#pragma unroll
          for (int j = 0; j < S::kOut; ++j) acc[j] += __uint_as_float(r[j]);
          if (++d_c == chunks) {
            const int m0 = (d_tile % m_tiles) * a.rows + part * S::kOut, rows = min(a.M, (d_tile % m_tiles + 1) * a.rows) - m0;
            const int n = (d_tile / m_tiles) * kCols + (GATED ? (quad & 1) * 32 : quad * 32) + lane;
            if constexpr (GATED) {         // the up values go to the threads that have the gate values
              float* up = sums + part * S::kOut * 64 + (quad & 1) * 32 + lane;
              const int t = (d_tile - worker) / n_workers;
              ok = __all_sync(0xffffffffu, quad >= 2 ? t == 0 || mbar_wait(up_read, (t - 1) & 1) : mbar_wait(up_there, t & 1));
              if (!ok) {
                if (lane == 0) atomicExch(a.status, 65);
                break;
              }
              if (n < a.N) {
#pragma unroll
                for (int j = 0; j < S::kOut; ++j) {
                  if (j >= rows) break;
                  const float v = ft_checked(a, m0 + j, quad >= 2 ? a.N + n : n, acc[j]);
                  if (quad >= 2) up[j * 64] = v;
                  else a.C[(size_t)(m0 + j) * a.ldc + n] = gated(a.gate, v, up[j * 64]);
                }
              }
              __syncwarp();
              if (lane == 0) mbar_arrive(quad >= 2 ? up_there : up_read);
            } else if (n < a.N) {
#pragma unroll
              for (int j = 0; j < S::kOut; ++j)
                if (j < rows) ft_store(a, m0 + j, n, acc[j], ft_old(a, m0 + j, n));
            }
#pragma unroll
            for (int j = 0; j < S::kOut; ++j) acc[j] = 0.0f;
            d_c = 0;
            d_tile += n_workers;
          }
        }
        __syncwarp();
      }
      if (u + 1 < units) split_weights(u + 1);
    }
  }
  __syncwarp();
  tc_fence_before();
  if constexpr (SPLIT) {
    if (warp >= WORKERS) {
      pdl_wait();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const int m0 = (worker % m_tiles) * a.rows;      // (a cluster has one tile)
    ft_add_up<GATED, S::kThreads>(a, sums, chunks_all, mine, m0, min(a.rows, a.M - m0), (worker / m_tiles) * kCols, rank);
  } else {
    __syncthreads();
  }
  if (warp == WORKERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kColumns) : "memory");
}

// ---- up to 16 tokens, K shared by a cluster ----
// The same sums with nothing but latency in mind: what a narrow matrix's few chunks a block cost above is the way from the workers to the
// tensor core and back (0.8 us a chunk) and the prologue in front of the first load (1.8 us). Here the last warp asks for weights before
// anything else, four chunks have buffers of their own, so that they go through in one go, and the tokens of all four are fetched at once, by
// four warps each. A cluster has one tile of 128 features (64 gate and 64 up rows) and all of a.rows tokens.
constexpr int kFewTokens = 16, kFewBuffers = 4, kFewThreads = 18 * 32, kFewPlane = kFewTokens * 128;
__host__ __device__ constexpr int few_smem(int chunks_all, int rows, int splits) {
  return kFewBuffers * (kFtRaw + 3 * kFewPlane) + chunks_all * rows * (kFtFeatures / splits) * 4 + 256 + 1024;
}

template <bool GATED>
__global__ void __launch_bounds__(kFewThreads, 1) gemm_f32_few_kernel(const __grid_constant__ CUtensorMap map_w, GemmF32TcArgs a) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = smem + kFewBuffers * kFtRaw;
  unsigned char* after = planes + kFewBuffers * 3 * kFewPlane;
  uint64_t* bars = reinterpret_cast<uint64_t*>(after);                 // full[4], empty[4], ready, done; then the tensor memory's address
  float* sums = reinterpret_cast<float*>(after + 256);                 // [chunk][token][feature], of this block's share of the features
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kFewBuffers + 2);
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * kFewBuffers, ready = empty0 + 8 * kFewBuffers, done = ready + 8;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int chunks_all = (a.K + kFtChunk - 1) / kFtChunk, rank = (int)cluster_ctarank(), tile = (int)blockIdx.x / a.splits;
  const int per = (chunks_all + a.splits - 1) / a.splits, c_first = rank * per, chunks = max(0, min(per, chunks_all - c_first));
  const int n0 = (GATED ? kFtFeatures / 2 : kFtFeatures) * (tile / a.m_tiles), m0 = tile % a.m_tiles * a.rows, live = min(a.rows, a.M - m0);

  auto ask = [&](int c) {
    const uint32_t bar = full0 + 8 * (c % kFewBuffers), dst = smem_addr(smem) + (c % kFewBuffers) * kFtRaw;
    const int k0 = (c_first + c) * kFtChunk;
    mbar_expect_tx(bar, kFtRaw);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      tma_load_2d(dst + h * (kFtRaw / 2), &map_w, k0 + 32 * h, n0, bar);
      tma_load_2d(dst + h * (kFtRaw / 2) + kFtRaw / 4, &map_w, k0 + 32 * h, GATED ? a.N + n0 : n0 + 64, bar);
    }
  };
  if (warp == 17) {
    if (elect_one()) {
      for (int i = 0; i < kFewBuffers; ++i) {
        mbar_init(full0 + 8 * i, 1);
        mbar_init(empty0 + 8 * i, 16);
      }
      mbar_init(ready, 16);
      mbar_init(done, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      fence_smem_to_async();
    }
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"n"(kFewThreads) : "memory");      // the barriers are there; this warp goes on to the loads
    if (elect_one()) {
      if (!a.early) pdl_wait();
      for (int c = 0; c < min(chunks, kFewBuffers); ++c) ask(c);
    }
    __syncwarp();
  } else if (warp == 16) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(tmem_slot)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  if (warp != 17) asm volatile("bar.sync 1, %0;" ::"n"(kFewThreads) : "memory");
  tc_fence_after();
  const uint32_t tmem = warp != 17 ? *tmem_slot : 0u, tA = tmem + kFewBuffers * kFewTokens;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // (no sums go to a block that has not begun)
  // Not by the loading warp, which has not waited for the allocation: a block of the next kernel that found this one's tensor memory still
  // free would take it and then wait for this grid, which could not go on without it.
  if (warp != 17) pdl_launch_dependents();
  const int mine = kFtFeatures / a.splits, half = mine / 2;                  // features of an output share

  if (warp == 17) {
    if (elect_one()) {
      for (int c = kFewBuffers; c < chunks; ++c) {
        if (!mbar_wait(empty0 + 8 * (c % kFewBuffers), ((c / kFewBuffers) - 1) & 1)) { atomicExch(a.status, 61); break; }
        ask(c);
      }
    }
  } else if (warp == 16) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(kFtFeatures, kFewTokens);
      for (int s = 0; s * kFewBuffers < chunks; ++s) {
        if (!mbar_wait(ready, s & 1)) { atomicExch(a.status, 62); break; }
        tc_fence_after();
        for (int i = 0; i < min(kFewBuffers, chunks - s * kFewBuffers); ++i) {
          const uint32_t d = tmem + i * kFewTokens, wa = tA + i * 96;
          const uint64_t x1 = smem_desc(smem_addr(planes) + i * 3 * kFewPlane), x2 = x1 + kFewPlane / 16, x3 = x2 + kFewPlane / 16;
          ft_multiply(d, wa, x1, x2, x3, idesc);
        }
        mma_commit(done);
      }
    }
  } else {
    const int quad = warp & 3, part = warp >> 2, row = quad * 32 + lane;
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const int t_row = (tid >> 3) & 15, t_k = (tid & 7) * 8;
    const float* src = a.A + (size_t)(m0 + min(t_row, live - 1)) * a.lda + t_k;
    bool ok = true;
    for (int s = 0; s * kFewBuffers < chunks; ++s) {
      const int c0 = s * kFewBuffers, n = min(kFewBuffers, chunks - c0);
      for (int i = 0; i < n; ++i) {        // lane = feature, this warp's quarter of the chunk's k values
        ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * i, s & 1)) && ok;
        const unsigned char* from = smem + i * kFtRaw + (part >> 1) * (kFtRaw / 2) + row * 128;
        uint32_t w1[8], w2[8], w3[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(from + ((((part & 1) * 4 + j) ^ (row & 7)) << 4));
          split2(v.x, v.y, w1[2 * j], w2[2 * j], w3[2 * j]);
          split2(v.z, v.w, w1[2 * j + 1], w2[2 * j + 1], w3[2 * j + 1]);
        }
        const uint32_t wa = tA + lanes + i * 96 + part * 8;
        tmem_st8_nowait(wa, w1);
        tmem_st8_nowait(wa + 32, w2);
        tmem_st8_nowait(wa + 64, w3);
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * i);
      }
      if (s == 0) pdl_wait();
      if (part < n) {                      // 8 lanes a row, 4 rows a store, which the swizzle spreads over all banks
        const int k0 = (c_first + c0 + part) * kFtChunk, left = a.K - k0 - t_k;
        float x[8];
        if (a.vec && left >= 8) {
          *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(src + k0);
          *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(src + k0 + 4);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = e < left ? src[k0 + e] : 0.0f;
        }
        if (t_row >= live) {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] = 0.0f;
        }
        uint4 q1, q2, q3;
        split2(x[0], x[1], q1.x, q2.x, q3.x);
        split2(x[2], x[3], q1.y, q2.y, q3.y);
        split2(x[4], x[5], q1.z, q2.z, q3.z);
        split2(x[6], x[7], q1.w, q2.w, q3.w);
        unsigned char* dst = planes + part * 3 * kFewPlane + t_row * 128 + ((((tid & 7) ^ t_row) & 7) << 4);
        *reinterpret_cast<uint4*>(dst) = q1;
        *reinterpret_cast<uint4*>(dst + kFewPlane) = q2;
        *reinterpret_cast<uint4*>(dst + 2 * kFewPlane) = q3;
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      fence_smem_to_async();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(ready);
      if (s == 0) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      ok = __all_sync(0xffffffffu, mbar_wait(done, s & 1)) && ok;
      tc_fence_after();
      if (!ok) {
        if (lane == 0) atomicExch(a.status, 64);
        break;
      }
      if (part < n) {                      // chunk `part`'s sums go to the block that adds up the feature
        uint32_t r[kFewTokens];
        tmem_ld16(tmem + lanes + part * kFewTokens, r);
        const int f = row, owner = GATED ? (f & 63) / half : f / mine, at_f = GATED ? (f >> 6) * half + (f & 63) % half : f % mine;
        const uint32_t at = cluster_map(smem_addr(sums) + (uint32_t)(((c_first + c0 + part) * a.rows * mine + at_f) * 4), (uint32_t)owner);
#pragma unroll
        for (int j = 0; j < kFewTokens; ++j)
          if (j < live) asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(at + (uint32_t)(j * mine * 4)), "r"(r[j]) : "memory");
      }
      tc_fence_before();
    }
    if (chunks == 0) {
      pdl_wait();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
  __syncwarp();
  tc_fence_before();
  if (warp >= 16) {
    pdl_wait();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  ft_add_up<GATED, kFewThreads>(a, sums, chunks_all, mine, m0, live, n0, rank);
  if (warp == 16) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// W [N, K] float32 seen through boxes of 64 rows by 32 values (128 bytes, 128-byte swizzle).
static int ft_map(CUtensorMap* map, const float* W, int N, int K, int ldw) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(2, "gemm_f32_tc: the driver does not offer cuTensorMapEncodeTiled");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
  cuuint64_t strides[1] = {(cuuint64_t)ldw * 4};
  cuuint32_t box[2] = {32, kFtFeatures / 2};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(2, "gemm_f32_tc: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

template <bool GATED>
static int launch_few(const CUtensorMap& map, const GemmF32TcArgs& a, cudaStream_t s) {
  const auto kernel = gemm_f32_few_kernel<GATED>;
  constexpr int kCols = GATED ? kFtFeatures / 2 : kFtFeatures;
  const int smem = few_smem((a.K + kFtChunk - 1) / kFtChunk, a.rows, a.splits);
  SLB_REQUIRE(smem <= 227 * 1024, "gemm_f32_tc: %d bytes of shared memory", smem);
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, 227 * 1024, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32_tc: %s", cudaGetErrorString(e));
  const bool early = a.early ? pdl_mode() != 0 : pdl_mode() == 1;
  launch_clusters(early, (unsigned)a.splits, kernel, dim3((unsigned)((a.N + kCols - 1) / kCols * a.m_tiles * a.splits)), dim3(kFewThreads), (size_t)smem, s, map, a);
  return check_launch("gemm_f32_tc (few tokens)");
}

template <int NT, int R, int WORKERS, bool SPLIT, bool GATED>
static int launch_ft_form(const CUtensorMap& map, const GemmF32TcArgs& a, cudaStream_t s) {
  const auto kernel = gemm_f32_tc_kernel<NT, R, WORKERS, SPLIT, GATED>;
  constexpr int kCols = GATED ? kFtFeatures / 2 : kFtFeatures;
  const int tiles = ((a.N + kCols - 1) / kCols) * ((a.M + a.rows - 1) / a.rows), all = (a.K + kFtChunk - 1) / kFtChunk;
  const int smem = ft_smem(NT, R, SPLIT ? (all + a.splits - 1) / a.splits : 0, a.rows, GATED);
  SLB_REQUIRE(smem <= 227 * 1024, "gemm_f32_tc: %d bytes of shared memory", smem);
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, 227 * 1024, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32_tc: cannot reserve shared memory: %s", cudaGetErrorString(e));
  const bool early = a.early ? pdl_mode() != 0 : pdl_mode() == 1;
  const dim3 block(FtShape<NT, WORKERS>::kThreads);
  const int room = sm_count() * (WORKERS == 8 ? 2 : 1);
  if (SPLIT) launch_clusters(early, (unsigned)a.splits, kernel, dim3((unsigned)(tiles * a.splits)), block, (size_t)smem, s, map, a);
  else launch_with(early, kernel, dim3((unsigned)(tiles < room ? tiles : room)), block, (size_t)smem, s, map, a);
  return check_launch("gemm_f32_tc");
}

// A form: tokens of a tile, blocks that share its K, warps that split (8: two blocks an SM, with a ring of two chunks; 16: one). The bits are
// the same for all. Per chunk and for what comes once a tile, in ns, fitted to products of 1 to 3,000 rows by 1,024 to 151,936 x 1,024 to 3,072 on a
// B200; `busy`: per chunk where two blocks share an SM. Tiles of 16 tokens want K shared so far that about every SM has a block, wider
// ones less, as each block's sums grow with its tokens.
struct FtForm {
  int nt, splits, workers, rows;
};
struct FtCost {
  int nt, workers, most_splits;
  double chunk, busy, once, once_split;
};
constexpr FtCost kFtCosts[] = {{16, 16, 8, 600, 600, 0, 5000}, {16, 8, 1, 900, 1450, 1000, 0}, {32, 8, 1, 1060, 1670, 1000, 0}, {32, 16, 8, 980, 980, 1000, 7900},
                               {64, 16, 1, 1200, 1200, 2500, 0}, {128, 16, 1, 1750, 1750, 2000, 0}};

// rows of a tile with which the chunks' sums fit beside the ring; 0: none
static int ft_split_rows(int nt, int splits, int K) {
  const int all = (K + kFtChunk - 1) / kFtChunk;
  for (int rows = nt; rows >= 4; rows /= 2)
    if ((nt == kFewTokens ? few_smem(all, rows, splits) : ft_smem(nt, 3, (all + splits - 1) / splits, rows)) <= 227 * 1024) return rows;
  return 0;
}

static FtForm ft_choose(int M, int rows_of_w, int K, bool with_gate) {
  const long long n_tiles = (rows_of_w + kFtFeatures - 1) / kFtFeatures, sms = sm_count(), chunks = (K + kFtChunk - 1) / kFtChunk;
  FtForm best{128, 1, 16, 128};
  double best_cost = 1e30;
  for (const FtCost& f : kFtCosts)
    for (int splits = f.nt == kFewTokens && f.workers == 16 ? 2 : 1; (f.nt <= 32 || !with_gate) && splits <= f.most_splits && splits <= chunks; splits *= 2) {
      const int rows = splits == 1 ? f.nt : ft_split_rows(f.nt, splits, K);
      if (rows == 0) continue;
      const long long blocks = n_tiles * ((M + rows - 1) / rows) * splits, room = f.workers == 8 ? 2 * sms : sms;
      const double cost = (double)((blocks + room - 1) / room) * ((double)((chunks + splits - 1) / splits) * (blocks > sms ? f.busy : f.chunk) + (splits > 1 ? f.once_split : f.once));
      if (cost < best_cost) { best_cost = cost; best = FtForm{f.nt, splits, f.workers, rows}; }
    }
  return best;
}

// (the gated form has tiles of 16 and 32 tokens: with wider ones the exchange of the up values and the shorter ring cost more than the activation
// kernel: 1,500 x 2 x 3,072 x 1,024 181 us against 125 + 15)
template <bool GATED>
static int launch_ft(const CUtensorMap& map, const GemmF32TcArgs& a, const FtForm& f, cudaStream_t s) {
  if (f.nt == 16) return f.splits > 1 ? launch_few<GATED>(map, a, s) : launch_ft_form<16, 2, 8, false, GATED>(map, a, s);
  if (f.nt == 32 && f.workers == 8) return launch_ft_form<32, 2, 8, false, GATED>(map, a, s);
  if (f.nt == 32) return f.splits > 1 ? launch_ft_form<32, 3, 16, true, GATED>(map, a, s) : launch_ft_form<32, 6, 16, false, GATED>(map, a, s);
  if constexpr (!GATED) return f.nt == 64 ? launch_ft_form<64, 5, 16, false, false>(map, a, s) : launch_ft_form<128, 4, 16, false, false>(map, a, s);
  return fail(2, "gemm_f32_tc: a gated product of %d tokens", a.M);
}

}  // namespace slb

using namespace slb;

// gate_kind: -1, or an activation (common.cuh) for a W that holds N gate rows and then N up rows: C [M, N] = act(gate) * up, without bias and not added.
// nt, splits and workers: 0 to let the rule choose, else tokens of a tile, blocks that share K and warps that split: tiles of 16 with 8 warps
// and one block or 16 warps and 2, 4 or 8; of 32 with 8 warps and one block or 16 warps and 1, 2, 4 or 8; of 64 and 128 (not gated) with 16 warps
// and one block. `status` is a device int that the caller zeroed: the kernel writes a code there if one of its bounded waits gave up.
extern "C" int slb_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               int accumulate, int static_weight, int gate_kind, float limit, float alpha, int nt, int splits, int workers, int* status,
                               void* stream) {
  SLB_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_tc: M=%d N=%d K=%d", M, N, K);
  SLB_REQUIRE(lda >= K && ldw >= K && ldc >= N && ldw % 4 == 0 && (uintptr_t)W % 16 == 0 && status != nullptr,
              "gemm_f32_tc: leading dimensions lda=%d ldw=%d ldc=%d for K=%d N=%d, W 16-byte aligned, a status word", lda, ldw, ldc, K, N);
  SLB_REQUIRE((long long)((N + 127) / 128) * ((M + 3) / 4) < (1ll << 28), "gemm_f32_tc: M=%d N=%d are too many tiles", M, N);
  const bool with_gate = gate_kind >= 0;
  SLB_REQUIRE(gate_kind >= -1 && gate_kind <= kGateLast && (!with_gate || (bias == nullptr && !accumulate)), "gemm_f32_tc: gate %d", gate_kind);
  if (M == 0) return 0;
  const int w_rows = with_gate ? 2 * N : N;
  FtForm f = ft_choose(M, w_rows, K, with_gate);
  if (nt) {
    bool known = false;
    for (const FtCost& c : kFtCosts) known = known || (c.nt == nt && c.workers == workers && ((splits == 1 && !(nt == kFewTokens && workers == 16)) || ((splits == 2 || splits == 4 || splits == 8) && splits <= c.most_splits)) && (c.nt <= 32 || !with_gate));
    SLB_REQUIRE(known, "gemm_f32_tc: tiles of %d tokens with %d blocks, %d warps", nt, splits, workers);
    f = FtForm{nt, splits, workers, splits == 1 ? nt : ft_split_rows(nt, splits, K)};
    SLB_REQUIRE(f.rows > 0, "gemm_f32_tc: the sums of K=%d do not fit the shared memory of %d blocks", K, splits);
  }
  GemmF32TcArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, static_weight, (uintptr_t)A % 16 == 0 && lda % 4 == 0, f.rows, f.splits, (M + f.rows - 1) / f.rows,
                  GateAct{with_gate ? gate_kind : 0, limit, alpha}, status};
  CUtensorMap map;
  const int rc = ft_map(&map, W, w_rows, K, ldw);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  return with_gate ? launch_ft<true>(map, a, f, s) : launch_ft<false>(map, a, f, s);
}
