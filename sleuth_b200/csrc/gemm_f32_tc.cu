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
// Blocks of a cluster may share a tile's K (few tokens: the weights' stream wants all SMs): each keeps its chunks' sums in shared
// memory, and each adds up a share of the outputs, all chunks in order, through distributed shared memory.
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
__host__ __device__ constexpr int ft_smem(int nt, int ring, int chunks, int rows) {
  return ring * kFtRaw + 2 * 3 * nt * 128 + chunks * rows * kFtFeatures * 4 + 256 + 1024;
}

// Two values into their three parts, packed as the tensor core reads them (the first in the low half).
__device__ __forceinline__ void split2(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  __nv_bfloat162 b = __floats2bfloat162_rn(x, y);
  p1 = *reinterpret_cast<uint32_t*>(&b);
  x -= __uint_as_float(p1 << 16);
  y -= __uint_as_float(p1 & 0xffff0000u);
  b = __floats2bfloat162_rn(x, y);
  p2 = *reinterpret_cast<uint32_t*>(&b);
  x -= __uint_as_float(p2 << 16);
  y -= __uint_as_float(p2 & 0xffff0000u);
  b = __floats2bfloat162_rn(x, y);
  p3 = *reinterpret_cast<uint32_t*>(&b);
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
__device__ __forceinline__ void ft_store(const GemmF32TcArgs& a, int m, int n, float v) {
  if (!isfinite(v)) v = ft_plain_dot(a, m, n);
  if (a.bias) v += a.bias[n];
  float* c = a.C + (size_t)m * a.ldc + n;
  *c = a.accumulate ? *c + v : v;
}

template <int NT, int R, int WORKERS, bool SPLIT>
__global__ void __launch_bounds__(FtShape<NT, WORKERS>::kThreads, WORKERS == 8 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, GemmF32TcArgs a) {
  using S = FtShape<NT, WORKERS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = smem + R * kFtRaw;
  unsigned char* after = planes + S::kB;
  uint64_t* bars = reinterpret_cast<uint64_t*>(after);      // full[R], empty[R], ready[2], done[2], then the tensor memory's address
  float* sums = reinterpret_cast<float*>(after + 256);      // SPLIT: [chunk of this block][token][feature]
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * R, ready0 = empty0 + 8 * R, done0 = ready0 + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * R + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int n_tiles = (a.N + kFtFeatures - 1) / kFtFeatures, m_tiles = (a.M + a.rows - 1) / a.rows, total = n_tiles * m_tiles;
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
  pdl_launch_dependents();
  if (warp <= WORKERS || !a.early) pdl_wait();

  if (warp == WORKERS + 1) {
    if (elect_one()) {
      int tile = worker, c = 0;
      for (int u = 0; u < units; ++u) {
        const int s = u % R;
        if (u >= R && !mbar_wait(empty0 + 8 * s, ((u / R) - 1) & 1)) { atomicExch(a.status, 61); break; }
        const int n0 = (tile / m_tiles) * kFtFeatures, k0 = (c_first + c) * kFtChunk;
        mbar_expect_tx(full0 + 8 * s, kFtRaw);
        const uint32_t dst = smem_addr(smem) + s * kFtRaw;
        tma_load_2d(dst, &map_w, k0, n0, full0 + 8 * s);
        tma_load_2d(dst + kFtRaw / 2, &map_w, k0 + 32, n0, full0 + 8 * s);
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
        mma_commit(done0 + 8 * b);
      }
    }
  } else {
    const int quad = warp & 3, part = warp >> 2;             // tensor memory's lanes; a share of the chunk's k values and of the tile's tokens
    const uint32_t lanes = (uint32_t)(quad * 32) << 16;
    const int b_row = tid >> 3, b_k = (tid & 7) * 8;         // this thread's row of each pass of tokens and its eight k values
    float raw[S::kPasses][8];
    auto fetch_tokens = [&](int tile, int c) {
      const int m0 = (tile % m_tiles) * a.rows, m_end = min(a.M, m0 + a.rows), k0 = (c_first + c) * kFtChunk + b_k;
#pragma unroll
      for (int p = 0; p < S::kPasses; ++p) {
        const int m = m0 + S::kRowsAPass * p + b_row;
        const float* src = a.A + (size_t)m * a.lda + k0;
        if (m < m_end && a.vec && k0 + 8 <= a.K) {
          *reinterpret_cast<float4*>(raw[p]) = *reinterpret_cast<const float4*>(src);
          *reinterpret_cast<float4*>(raw[p] + 4) = *reinterpret_cast<const float4*>(src + 4);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) raw[p][e] = m < m_end && k0 + e < a.K ? src[e] : 0.0f;
        }
      }
    };
    float acc[S::kOut];
#pragma unroll
    for (int j = 0; j < S::kOut; ++j) acc[j] = 0.0f;
    int tile = worker, c = 0;                                // of unit u
    int d_tile = worker, d_c = 0;                            // of the unit that is taken out
    bool ok = true;
    if (units) fetch_tokens(tile, c);
    for (int u = 0; u <= units && ok; ++u) {
      if (u < units) {
        const int b = u & 1, s = u % R;
        // the tokens' values: 8 lanes a row, 4 rows a store, which the swizzle spreads over all banks
        if (NT >= S::kRowsAPass || b_row < NT) {
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
        }
        if (++c == chunks) { c = 0; tile += n_workers; }
        if (u + 1 < units) fetch_tokens(tile, c);
        // the weights: lane = feature, this warp's share of the chunk's k values
        ok = mbar_wait(full0 + 8 * s, (u / R) & 1);
        const int row = quad * 32 + lane;
#pragma unroll
        for (int j0 = 0; j0 < S::kPieces; j0 += 4) {
          const int piece = part * S::kPieces + j0;          // of the chunk's sixteen a feature; eight lie side by side
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
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        fence_smem_to_async();
        tc_fence_before();
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) atomicExch(a.status, 63);
        } else if (lane == 0) {
          mbar_arrive(empty0 + 8 * s);
          mbar_arrive(ready0 + 8 * b);
        }
      }
      if (u >= 1 && ok) {
        const int v = u - 1, b = v & 1;
        ok = __all_sync(0xffffffffu, mbar_wait(done0 + 8 * b, (v >> 1) & 1));
        if (!ok) {
          if (lane == 0) atomicExch(a.status, 64);
          break;
        }
        tc_fence_after();
        uint32_t r[S::kOut];
        ft_take_out<S::kOut>(tmem + lanes + b * NT + part * S::kOut, r);
        if constexpr (SPLIT) {
          const int live = min(a.rows, a.M - (worker % m_tiles) * a.rows) - part * S::kOut;
          float* dst = sums + ((size_t)v * a.rows + part * S::kOut) * kFtFeatures + quad * 32 + lane;
#pragma unroll
          for (int j = 0; j < S::kOut; ++j)
            if (j < live) dst[j * kFtFeatures] = __uint_as_float(r[j]);
        } else {
#pragma unroll
          for (int j = 0; j < S::kOut; ++j) acc[j] += __uint_as_float(r[j]);
          if (++d_c == chunks) {
            const int m0 = (d_tile % m_tiles) * a.rows + part * S::kOut, rows = min(a.M, (d_tile % m_tiles + 1) * a.rows) - m0;
            const int n = (d_tile / m_tiles) * kFtFeatures + quad * 32 + lane;
            if (n < a.N) {
#pragma unroll
              for (int j = 0; j < S::kOut; ++j)
                if (j < rows) ft_store(a, m0 + j, n, acc[j]);
            }
#pragma unroll
            for (int j = 0; j < S::kOut; ++j) acc[j] = 0.0f;
            d_c = 0;
            d_tile += n_workers;
          }
        }
        __syncwarp();
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  if constexpr (SPLIT) {
    cluster_sync_all();        // every share's sums are in its block's shared memory
    // (a cluster has one tile) this block's part of the outputs, token by token of 128 features
    const int m0 = (worker % m_tiles) * a.rows, live = min(a.rows, a.M - m0), n0 = (worker / m_tiles) * kFtFeatures;
    const uint32_t base = smem_addr(sums), step = (uint32_t)a.rows * kFtFeatures * 4;
    for (int i = rank * S::kThreads + tid; i < live * kFtFeatures; i += shares * S::kThreads) {
      const uint32_t at = base + (uint32_t)i * 4;
      float v = 0.0f;
      int r = 0, c = 0;
      for (int g0 = 0; g0 < chunks_all; g0 += 16) {          // sixteen chunks' sums under way at a time
        float x[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          x[j] = 0.0f;
          if (g0 + j < chunks_all) {
            asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(x[j]) : "r"(cluster_map(at, (uint32_t)r) + (uint32_t)c * step));
            if (++c == per) { c = 0; ++r; }
          }
        }
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (g0 + j < chunks_all) v += x[j];
      }
      const int n = n0 + i % kFtFeatures;
      if (n < a.N) ft_store(a, m0 + i / kFtFeatures, n, v);
    }
    cluster_sync_all();        // no block leaves while another still reads its sums
  } else {
    __syncthreads();
  }
  if (warp == WORKERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kColumns) : "memory");
}

// W [N, K] float32 seen through boxes of 128 rows by 32 values (128 bytes, 128-byte swizzle).
static int ft_map(CUtensorMap* map, const float* W, int N, int K, int ldw) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(2, "gemm_f32_tc: the driver does not offer cuTensorMapEncodeTiled");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
  cuuint64_t strides[1] = {(cuuint64_t)ldw * 4};
  cuuint32_t box[2] = {32, kFtFeatures};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(2, "gemm_f32_tc: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

template <int NT, int R, int WORKERS, bool SPLIT>
static int launch_ft_form(const CUtensorMap& map, const GemmF32TcArgs& a, cudaStream_t s) {
  const auto kernel = gemm_f32_tc_kernel<NT, R, WORKERS, SPLIT>;
  const int tiles = ((a.N + kFtFeatures - 1) / kFtFeatures) * ((a.M + a.rows - 1) / a.rows), all = (a.K + kFtChunk - 1) / kFtChunk;
  const int smem = ft_smem(NT, R, SPLIT ? (all + a.splits - 1) / a.splits : 0, a.rows);
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

// A form: tokens of a tile, blocks that share its K, warps that split (8: two blocks an SM, with a ring of two chunks). The bits are the same for all.
struct FtForm {
  int nt, splits, workers, rows;
};

// rows of a tile with which the chunks' sums fit beside the ring; 0: none
static int ft_split_rows(int nt, int splits, int workers, int K) {
  const int per = ((K + kFtChunk - 1) / kFtChunk + splits - 1) / splits;
  for (int rows = nt; rows >= 4; rows /= 2)
    if (workers == 8 ? ft_smem(nt, 2, per, rows) <= 113 * 1024 : ft_smem(nt, 3, per, rows) <= 227 * 1024) return rows;
  return 0;
}

static FtForm ft_choose(int M, int N, int K) {
  const long long n_tiles = (N + kFtFeatures - 1) / kFtFeatures, sms = sm_count(), chunks = (K + kFtChunk - 1) / kFtChunk;
  FtForm best{128, 1, 16, 128};
  double best_cost = 1e30;
  const int widths[4] = {16, 32, 64, 128};
  const double chunk_ns[4] = {560, 580, 700, 1050};
  for (int i = 0; i < 4; ++i) {
    for (int splits = 1; splits <= 8; splits *= 2) {
      if (splits > 1 && (widths[i] > 32 || splits > chunks)) break;
      const int rows = splits == 1 ? widths[i] : ft_split_rows(widths[i], splits, 16, K);
      if (rows == 0) continue;
      const long long tiles = n_tiles * ((M + rows - 1) / rows);
      const long long rounds = (tiles * splits + sms - 1) / sms;
      const double cost = rounds * (((chunks + splits - 1) / splits) * chunk_ns[i] + (splits > 1 ? 3500.0 : 1500.0));
      if (cost < best_cost) { best_cost = cost; best = FtForm{widths[i], splits, 16, rows}; }
    }
  }
  return best;
}

}  // namespace slb

using namespace slb;

// nt, splits and workers: 0 to let the rule choose, else tokens of a tile (16, 32, 64, 128), blocks that share K (1, 2, 4, 8; above 1 for tiles
// of 16 and 32 only) and warps that split (8 or 16; 8 for tiles of 16 and 32 only). `status` is a device int that the caller zeroed: the kernel writes
// a code there if one of its bounded waits gave up.
extern "C" int slb_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               int accumulate, int static_weight, int nt, int splits, int workers, int* status, void* stream) {
  SLB_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_tc: M=%d N=%d K=%d", M, N, K);
  SLB_REQUIRE(lda >= K && ldw >= K && ldc >= N && ldw % 4 == 0 && (uintptr_t)W % 16 == 0 && status != nullptr,
              "gemm_f32_tc: leading dimensions lda=%d ldw=%d ldc=%d for K=%d N=%d, W 16-byte aligned, a status word", lda, ldw, ldc, K, N);
  SLB_REQUIRE((long long)((N + 127) / 128) * ((M + 3) / 4) < (1ll << 28), "gemm_f32_tc: M=%d N=%d are too many tiles", M, N);
  if (M == 0) return 0;
  FtForm f = ft_choose(M, N, K);
  if (nt) {
    const bool small = nt == 16 || nt == 32;
    SLB_REQUIRE((small || nt == 64 || nt == 128) && (splits == 1 || ((splits == 2 || splits == 4 || splits == 8) && small)) &&
                (workers == 16 || (workers == 8 && small)), "gemm_f32_tc: tiles of %d tokens with %d blocks, %d warps", nt, splits, workers);
    f = FtForm{nt, splits, workers, splits == 1 ? nt : ft_split_rows(nt, splits, workers, K)};
    SLB_REQUIRE(f.rows > 0, "gemm_f32_tc: the sums of K=%d do not fit the shared memory of %d blocks", K, splits);
  }
  GemmF32TcArgs a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, static_weight, (uintptr_t)A % 16 == 0 && lda % 4 == 0, f.rows, f.splits, status};
  CUtensorMap map;
  const int rc = ft_map(&map, W, N, K, ldw);
  if (rc) return rc;
  cudaStream_t s = (cudaStream_t)stream;
  if (f.workers == 8) {
    if (f.splits > 1) return f.nt == 16 ? launch_ft_form<16, 2, 8, true>(map, a, s) : launch_ft_form<32, 2, 8, true>(map, a, s);
    return f.nt == 16 ? launch_ft_form<16, 2, 8, false>(map, a, s) : launch_ft_form<32, 2, 8, false>(map, a, s);
  }
  if (f.splits > 1) return f.nt == 16 ? launch_ft_form<16, 3, 16, true>(map, a, s) : launch_ft_form<32, 3, 16, true>(map, a, s);
  if (f.nt == 16) return launch_ft_form<16, 6, 16, false>(map, a, s);
  if (f.nt == 32) return launch_ft_form<32, 6, 16, false>(map, a, s);
  if (f.nt == 64) return launch_ft_form<64, 5, 16, false>(map, a, s);
  return launch_ft_form<128, 4, 16, false>(map, a, s);
}
