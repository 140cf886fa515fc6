// The 32-bit matrix product on the tensor cores: C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]), float32 in, float32 out.
//
// A float32 value is the sum of three bfloat16 values exactly (8 + 8 + 8 bits of its 24): x = x1 + x2 + x3 with x1 = bf16(x),
// x2 = bf16(x - x1), x3 = x - x1 - x2, |x2| <= 2^-8 |x|, |x3| <= 2^-16 |x|. (bfloat16 ends at 2^-133, so for values below 2^-110 this holds only of the
// value times 2^24: both operands are split after that multiplication, and the result is divided by 2^48.) A product of two bfloat16 values is exact in
// float32, so a product is w1 a1 + (w1 a2 + w2 a1) + (w1 a3 + w2 a2 + w3 a1) and parts of either sign below 2^-24 of it, typically 2^-27,
// which are left out: six tcgen05 products of kind f16 in place of one FMA a value (splitting into exact partial products:
// Dekker, 1971; Ozaki et al., 2012).
//
// Order of the sums: K is cut into chunks of 64, a chunk into two chains of 32. A chain's six products are summed by the tensor core, the small ones first,
// so that of its twelve instructions only the last two add at full size (its float32 sums are truncated, which on operands of one sign is a bias; in
// chains of 64 it came to 1.33 units of 2^-24, 0.8 here). Chains are taken out of tensor memory, and all further sums are float32, rounded to nearest: a
// chunk is chain 0 + chain 1, two chunks make a pair, and the pairs are added in ascending order:
//     C = ((pair 0 + pair 1) + pair 2) + ...   (+ bias, then added to the old value)
// Every form does exactly this, here and in the kernel for few rows (gemm_f32_rows.cu), whatever tile it takes and whatever M is, so that a row's
// bits depend neither on the rows beside it nor on how a sequence was cut into steps. Which products come here depends on W alone
// (ops.f32_on_tensor_cores). Error (2-norm, against 64 bits), FMA chains / here: normal operands, K 1,024 2.1e-7 / 0.9e-7, 3,072 3.6e-7 / 1.2e-7, 9,728
// 6.3e-7 / 1.8e-7; of one sign 0.74e-7 / 0.68e-7, 1.2e-7 / 0.9e-7, 1.7e-7 / 1.3e-7. Below K = 1,024 operands of wide range can lose to the FMA chains.
// A result that is not finite in this form (infinite or NaN operands, whose parts are NaN; operands from 2^104, results from 2^80 on) is formed again as the
// FMA kernels form it.
//
// One block: 128 features (the instruction's rows) by NT tokens. Per chunk, for the unit u:
//   * the last warp asks TMA for the raw 128 x 64 weights, a ring of R chunks ahead;
//   * eight or sixteen warps take the two chains of unit u - 1 out of tensor memory (while the tensor core rests: beside its products, which read tensor
//     memory too, a load from there takes several times as long: 1,500 x 4,096 x 1,024 178 us against 98), then, while unit u is multiplied, split the weights of
//     unit u + 1 into tensor memory (operand A of the instruction) and its tokens' values, fetched a unit ahead into registers, into shared memory in the
//     128-byte swizzle (operand B), both double-buffered; a tile's sums lie in shared memory where registers are short (128 tokens);
//   * one more warp issues the 24 instructions.
// The first chunk of weights is split before the wait for the kernel in front. 1,500 x 4,096 x 1,024: 309 us by FMA, 88.7 with one chain a chunk, 97.5 now: what
// bounds it is the splitting warps' chain a chunk; the tensor core works a third of the time.
#include "gemm_f32_split.cuh"
#include "tcgen05.cuh"

namespace slb {

static_assert(kF32Steps == 2, "two chains a chunk");
constexpr int kFtChunk = kF32Chunk, kFtFeatures = 128, kFtRaw = kFtFeatures * kFtChunk * 4;

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
  static constexpr bool kHeld = kOut > 16;                 // a tile's sums lie in shared memory: registers hold one partial sum's
  static constexpr int kTotals = kHeld ? NT * kFtFeatures * 4 : 0;
  static constexpr int kColumns = 2 * NT + 192 > 256 ? 512 : 256;
};
// Shared memory: the ring, the tokens' parts, a tile's sums, the barriers.
template <int NT, int R, int WORKERS>
constexpr int ft_smem() {
  return R * kFtRaw + FtShape<NT, WORKERS>::kB + FtShape<NT, WORKERS>::kTotals + 256 + 1024;
}

__device__ __forceinline__ void tmem_st4_nowait(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory");
}
__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// One chain: the products of kF32Steps sixteens from sixteen k4 on, the small ones first. wa: the three parts of W in tensor memory, 32
// columns each; x1, x2, x3: the tokens' parts.
__device__ __forceinline__ void ft_multiply(int k0, uint32_t d, uint32_t wa, uint64_t x1, uint64_t x2, uint64_t x3, uint32_t idesc) {
#pragma unroll
  for (int k4 = k0; k4 < k0 + kF32Steps; ++k4) {
    mma_bf16_ts(d, wa + 64 + k4 * 8, x1 + k4 * 2, idesc, k4 > k0 ? 1u : 0u);
    mma_bf16_ts(d, wa + k4 * 8, x3 + k4 * 2, idesc, 1u);
    mma_bf16_ts(d, wa + 32 + k4 * 8, x2 + k4 * 2, idesc, 1u);
  }
#pragma unroll
  for (int k4 = k0; k4 < k0 + kF32Steps; ++k4) {
    mma_bf16_ts(d, wa + 32 + k4 * 8, x1 + k4 * 2, idesc, 1u);
    mma_bf16_ts(d, wa + k4 * 8, x2 + k4 * 2, idesc, 1u);
  }
#pragma unroll
  for (int k4 = k0; k4 < k0 + kF32Steps; ++k4) mma_bf16_ts(d, wa + k4 * 8, x1 + k4 * 2, idesc, 1u);
}

template <int NT, int R, int WORKERS>
__global__ void __launch_bounds__(FtShape<NT, WORKERS>::kThreads, WORKERS == 8 ? 2 : 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ F32Args a) {
  using S = FtShape<NT, WORKERS>;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* planes = smem + R * kFtRaw;
  float4* totals = reinterpret_cast<float4*>(planes + S::kB) + threadIdx.x;      // kHeld: [four values][worker thread]
  unsigned char* after = planes + S::kB + S::kTotals;
  uint64_t* bars = reinterpret_cast<uint64_t*>(after);      // full[R], empty[R], ready[2], done[2]; then the tensor memory's address
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * R, ready0 = empty0 + 8 * R, done0 = ready0 + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * R + 4);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int n_tiles = (a.N + kFtFeatures - 1) / kFtFeatures, m_tiles = (a.M + NT - 1) / NT, total = n_tiles * m_tiles;
  const int chunks = (a.K + kFtChunk - 1) / kFtChunk, worker = (int)blockIdx.x, n_workers = (int)gridDim.x;
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

  if (warp == WORKERS + 1) {
    if (elect_one()) {
      if (!a.early) pdl_wait();
      int tile = worker, c = 0;
      for (int u = 0; u < units; ++u) {
        const int s = u % R;
        if (u >= R && !mbar_wait(empty0 + 8 * s, ((u / R) - 1) & 1)) { atomicExch(a.status, 61); break; }
        const int n0 = (tile / m_tiles) * kFtFeatures, k0 = c * kFtChunk;
        mbar_expect_tx(full0 + 8 * s, kFtRaw);
        const uint32_t dst = smem_addr(smem) + s * kFtRaw;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tma_load_2d(dst + h * (kFtRaw / 2), &map_w, k0 + 32 * h, n0, full0 + 8 * s);
          tma_load_2d(dst + h * (kFtRaw / 2) + kFtRaw / 4, &map_w, k0 + 32 * h, n0 + 64, full0 + 8 * s);
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
        const uint32_t wa = tA + b * 96;
        const uint64_t x1 = smem_desc(smem_addr(planes) + b * 3 * S::kPlane), x2 = x1 + S::kPlane / 16, x3 = x2 + S::kPlane / 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) ft_multiply(h * kF32Steps, tmem + h * NT, wa, x1, x2, x3, idesc);
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
      const int m0 = (tile % m_tiles) * NT, m_end = min(a.M, m0 + NT);
      there = 0;
#pragma unroll
      for (int p = 0; p < S::kPasses; ++p) {
        const int m = m0 + S::kRowsAPass * p + b_row;
        if (m < m_end) there |= 1u << p;
        rows_at[p] = a.A + (size_t)min(m, a.M - 1) * a.lda + b_k;
      }
    };
    auto fetch_tokens = [&](int c) {
      const int left = a.K - c * kFtChunk - b_k;
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
    float sum[S::kOut], acc[S::kHeld ? 1 : S::kOut];         // of the chunks of one partial sum; of the tile
#pragma unroll
    for (int j = 0; j < S::kOut; ++j) sum[j] = 0.0f;
    // The partial sum joins the tile's sums (v: these with it); `begin`: there are none yet.
    auto join = [&](bool begin, bool end, auto&& store) {
      if constexpr (S::kHeld) {
#pragma unroll
        for (int j = 0; j < S::kOut; j += 4) {
          float4 v = begin ? make_float4(0.f, 0.f, 0.f, 0.f) : totals[j / 4 * (WORKERS * 32)];
          v.x += sum[j];
          v.y += sum[j + 1];
          v.z += sum[j + 2];
          v.w += sum[j + 3];
          if (end) {
            store(j, v.x);
            store(j + 1, v.y);
            store(j + 2, v.z);
            store(j + 3, v.w);
          } else {
            totals[j / 4 * (WORKERS * 32)] = v;
          }
          sum[j] = sum[j + 1] = sum[j + 2] = sum[j + 3] = 0.0f;
        }
      } else {
#pragma unroll
        for (int j = 0; j < S::kOut; ++j) {
          acc[j] = (begin ? 0.0f : acc[j]) + sum[j];
          if (end) store(j, acc[j]);
          sum[j] = 0.0f;
        }
      }
    };
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
      for (int j0 = 0; j0 < S::kPieces; j0 += 2) {           // (two pieces at a time: registers)
        const int piece = part * S::kPieces + j0;            // of the chunk's sixteen a feature; eight lie side by side
        const unsigned char* src = smem + s * kFtRaw + (piece >> 3) * (kFtRaw / 2) + row * 128;
        uint32_t w1[4], w2[4], w3[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float4 v = *reinterpret_cast<const float4*>(src + ((((piece & 7) + j) ^ (row & 7)) << 4));
          split2(v.x, v.y, w1[2 * j], w2[2 * j], w3[2 * j]);
          split2(v.z, v.w, w1[2 * j + 1], w2[2 * j + 1], w3[2 * j + 1]);
        }
        const uint32_t wa = tA + lanes + b * 96 + piece * 2;
        tmem_st4_nowait(wa, w1);
        tmem_st4_nowait(wa + 32, w2);
        tmem_st4_nowait(wa + 64, w3);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(empty0 + 8 * s);
    };
    auto take_out = [&](int v) {           // the sum of unit v's two chains joins its partial sum
      ok = __all_sync(0xffffffffu, mbar_wait(done0 + 8 * (v & 1), (v >> 1) & 1));
      if (!ok) {
        if (lane == 0) atomicExch(a.status, 64);
        return;
      }
      tc_fence_after();
#pragma unroll
      for (int j0 = 0; j0 < S::kOut; j0 += 8) {
        uint32_t r[2][8];
        tmem_ld8_nowait(tmem + lanes + part * S::kOut + j0, r[0]);
        tmem_ld8_nowait(tmem + lanes + NT + part * S::kOut + j0, r[1]);
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j0 + j] += __uint_as_float(r[0][j]) + __uint_as_float(r[1][j]);
      }
    };
    if (units) split_weights(0);           // (the kernel in front may still be running)
    pdl_wait();
    // The tokens' values are fetched a unit before they are split.
    int f_tile = worker, f_c = 0, f_left = units;
    auto fetch_next = [&]() {
      if (f_left == 0) return;
      fetch_tokens(f_c);
      --f_left;
      if (++f_c == chunks) {
        f_c = 0;
        f_tile += n_workers;
        if (f_left) aim(f_tile);
      }
    };
    if (units) {
      aim(f_tile);
      fetch_next();
      split_tokens(0);
      fetch_next();
    }
    for (int u = 0; u <= units && ok; ++u) {
      // The sums are taken out while the tensor core rests: beside its products, which read tensor memory themselves, a load from there takes several times as long.
      if (u >= 1) take_out(u - 1);
      if (!ok) break;
      if (u < units) {
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        fence_smem_to_async();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(ready0 + 8 * (u & 1));
        if (u + 1 < units) split_weights(u + 1);
      }
      if (u >= 1) {
        ++d_c;
        if (d_c % kF32Partial == 0 || d_c == chunks) {
          const int m0 = (d_tile % m_tiles) * NT + part * S::kOut, rows = a.M - m0, n = (d_tile / m_tiles) * kFtFeatures + quad * 32 + lane;
          uint32_t again = 0;                // outputs that are not finite: formed again, in one place for the registers' sake
          join(d_c <= kF32Partial, d_c == chunks, [&](int j, float v) {
            if (j >= rows || n >= a.N) return;
            if (isfinite(v)) f32_finish(a, m0 + j, n, v * kF32Unscale, f32_old(a, m0 + j, n));
            else again |= 1u << j;
          });
          while (again) {
            const int j = __ffs(again) - 1;
            again &= again - 1;
            f32_finish(a, m0 + j, n, f32_plain_dot(a, m0 + j, n), f32_old(a, m0 + j, n));
          }
          if (d_c == chunks) {
            d_c = 0;
            d_tile += n_workers;
          }
        }
      }
      if (u + 1 < units && ok) {
        split_tokens((u + 1) & 1);
        fetch_next();
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == WORKERS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kColumns) : "memory");
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

template <int NT, int R, int WORKERS>
static int launch_ft_form(const CUtensorMap& map, const F32Args& a, cudaStream_t s) {
  const auto kernel = gemm_f32_tc_kernel<NT, R, WORKERS>;
  const int tiles = ((a.N + kFtFeatures - 1) / kFtFeatures) * ((a.M + NT - 1) / NT);
  constexpr int smem = ft_smem<NT, R, WORKERS>();
  static_assert(smem <= 227 * 1024, "the ring fits");
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, smem, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32_tc: cannot reserve shared memory: %s", cudaGetErrorString(e));
  const bool early = a.early ? pdl_mode() != 0 : pdl_mode() == 1;
  const int room = sm_count() * (WORKERS == 8 ? 2 : 1);
  launch_with(early, kernel, dim3((unsigned)(tiles < room ? tiles : room)), dim3(FtShape<NT, WORKERS>::kThreads), (size_t)smem, s, map, a);
  return check_launch("gemm_f32_tc");
}

// The forms: 1, the kernel for few rows; else tokens of a tile (32: two blocks of eight splitting warps an SM, with a ring of two chunks; 64 and 128:
// one of sixteen). The bits are the same for all. Per chunk and for what comes once a tile, in ns, fitted to products of 64 to 1,500 rows by 1,024
// to 151,936 x 1,024 to 3,072 on a B200.
struct FtCost {
  int nt, workers;
  double chunk, once;
};
constexpr FtCost kFtCosts[] = {{32, 8, 1600, 1000}, {64, 16, 1250, 2500}, {128, 16, 1920, 2000}};

static int ft_choose(int M, int N, int K) {
  const long long n_tiles = (N + kFtFeatures - 1) / kFtFeatures, sms = sm_count(), chunks = (K + kFtChunk - 1) / kFtChunk;
  int best = 1;
  double best_cost = f32_rows_cost(M, N, K);
  for (const FtCost& f : kFtCosts) {
    const long long blocks = n_tiles * ((M + f.nt - 1) / f.nt), room = f.workers == 8 ? 2 * sms : sms;
    const double cost = (double)((blocks + room - 1) / room) * ((double)chunks * f.chunk + f.once);
    if (cost < best_cost) { best_cost = cost; best = f.nt; }
  }
  return best;
}

}  // namespace slb

using namespace slb;

// gate_kind: -1, or an activation (common.cuh) for a W that holds N gate rows and then N up rows: C [M, N] = act(gate) * up, without bias and not
// added, always in the form for few rows. form: 0 to let the rule choose, 1 the kernel for few rows, else the tokens of a tile (32, 64 or 128, not gated).
// next, next_bytes: the matrix that the kernel after this one reads, or nothing. `status` is a device int that the caller zeroed: a kernel writes a code there if one of its bounded waits gave up.
// The form that the rule chooses.
extern "C" int slb_gemm_f32_form(int M, int N, int K) { return M >= 1 && N >= 1 && K >= 1 ? ft_choose(M, N, K) : 0; }

extern "C" int slb_gemm_f32_tc(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                               int accumulate, int static_weight, int gate_kind, float limit, float alpha, int form, const void* next, long long next_bytes,
                               int* status, void* stream) {
  SLB_REQUIRE(M >= 0 && N > 0 && K > 0 && K % 4 == 0, "gemm_f32_tc: M=%d N=%d K=%d", M, N, K);
  SLB_REQUIRE(lda >= K && ldw >= K && ldc >= N && ldw % 4 == 0 && (uintptr_t)W % 16 == 0 && status != nullptr,
              "gemm_f32_tc: leading dimensions lda=%d ldw=%d ldc=%d for K=%d N=%d, W 16-byte aligned, a status word", lda, ldw, ldc, K, N);
  SLB_REQUIRE((long long)((N + 127) / 128) * ((M + 31) / 32) < (1ll << 28), "gemm_f32_tc: M=%d N=%d are too many tiles", M, N);
  const bool with_gate = gate_kind >= 0;
  SLB_REQUIRE(gate_kind >= -1 && gate_kind <= kGateLast && (!with_gate || (bias == nullptr && !accumulate && form <= 1)), "gemm_f32_tc: gate %d", gate_kind);
  SLB_REQUIRE(form == 0 || form == 1 || form == 32 || form == 64 || form == 128, "gemm_f32_tc: form %d for %d rows", form, M);
  SLB_REQUIRE(next_bytes >= 0 && (uintptr_t)next % 16 == 0, "gemm_f32_tc: the range to prefetch must be 16-byte aligned");
  if (M == 0) return 0;
  const F32Args a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, static_weight, (uintptr_t)A % 16 == 0 && lda % 4 == 0,
                  GateAct{with_gate ? gate_kind : 0, limit, alpha}, status, NextRead{(const char*)next, next_bytes}};
  cudaStream_t s = (cudaStream_t)stream;
  const int chosen = with_gate ? 1 : form ? form : ft_choose(M, N, K);
  if (chosen == 1) return launch_f32_rows(a, with_gate, s);
  CUtensorMap map;
  const int rc = ft_map(&map, W, N, K, ldw);
  if (rc) return rc;
  switch (chosen) {
    case 32: return launch_ft_form<32, 2, 8>(map, a, s);
    case 64: return launch_ft_form<64, 5, 16>(map, a, s);
    default: return launch_ft_form<128, 2, 16>(map, a, s);
  }
}
