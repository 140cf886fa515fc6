// The 32-bit product of few rows on the tensor cores, with the bits of gemm_f32_tc.cu: C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]), or
// act(gate) * up for a W of gate and up rows.
//
// mma.sync and tcgen05.mma add sixteen products and an accumulator in the same way: 30 million sums of normal, one-signed, equal, sparse and
// tiny values and of such over 30 decades agreed in every bit, also with the sixteen in another order (and the tests demand it of every form). So the
// same parts in the same order of instructions give the same result from registers, without tensor memory, its allocation and the
// way there and back, which is what a few rows wait for.
//
// Bound by the stream of the weights where there are many, by latency where there are few. A block has a tile of 16 features and up to 32 rows; its
// warps share K, a chunk each a round, and a warp keeps its own ring of weight chunks, R deep, by cp.async: a lane copies exactly the
// 16-byte pieces that its fragments want (k 4t .. 4t + 3 of rows g and g + 8; within sixteen products the order is free), so the ring needs no
// barrier and no swizzle, and it runs on over the block's tiles. Where no kernel writes W the ring is filled before the wait for the kernel in
// front, and the next product's matrix is asked into L2. The rows of A are fetched a chunk ahead and split by every warp that uses them. The chunks' sums
// of a round meet in shared memory, where one thread an output adds them two by two. A step of one sequence (0.6B sizes) waits for some
// 110 of these one after the other. us in a row of launches, FMA chains / clusters of tcgen05 blocks with the exchange through
// distributed shared memory (this kernel's predecessor) / here: one row of 4,096 x 1,024 4.6 / 6.6 / 5.2, 1,024 x 2,048 4.9 / 5.1 / 4.0, 6,144 x 1,024
// 6.0 / 8.5 / 7.2, 1,024 x 3,072 6.6 / 7.2 / 5.7, 19,456 x 2,560 35 / 56 / 41; eight rows 5.6 / 6.7 / 5.4, 7.4 / 5.3 / 4.5, 8.7 / 9.1 / 7.3, 10.4 / 7.5 / 6.2, 51 / 61 / 43.
#include "gemm_f32_split.cuh"

namespace slb {


constexpr int kFrRows = 16;      // features of a tile (of a gated one half gate, half up rows)

// 8 * NB rows of A, WARPS warps that share K.
template <int NB, int WARPS>
struct FrShape {
  static constexpr int kThreads = WARPS * 32;
  static constexpr int kStage = 8 * 512;                             // bytes of a warp's chunk: 16 bytes a lane and piece
  static constexpr int kTokens = 8 * NB;
  static constexpr int kStride = kFrRows + 4;                        // floats from one token's sums to the next's (spreads the stores over the banks)
  static constexpr int kSums = WARPS * kTokens * kStride;            // floats of a round's sums; two rounds' are held
  static constexpr int kRoom = WARPS == 8 ? 113 * 1024 : 227 * 1024; // two blocks of eight warps an SM, one of sixteen
  static constexpr int kStages = (kRoom - 2 * kSums * 4) / (WARPS * kStage);
  static constexpr int kSmem = WARPS * kStages * kStage + 2 * kSums * 4;
};

// (Not volatile: the two chains' instructions may be interleaved.)
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&w)[4], const uint32_t (&x)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(x[0]), "r"(x[1]));
}

template <int NB, int WARPS, bool GATED>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 2 : 1) gemm_f32_split_rows_kernel(const __grid_constant__ F32Args a, int m_tiles) {
  using S = FrShape<NB, WARPS>;
  constexpr int R = S::kStages, kCols = GATED ? kFrRows / 2 : kFrRows, kOut = kCols * S::kTokens, kOwn = (kOut + S::kThreads - 1) / S::kThreads;
  static_assert(R >= 2 && WARPS % 2 == 0 && kF32Steps == 2, "rounds of whole pairs of chunks");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const float4* ring = reinterpret_cast<const float4*>(smem_raw + (size_t)warp * R * S::kStage) + lane;      // [stage][step][row g or g + 8][lane]
  const uint32_t ring_at = (uint32_t)__cvta_generic_to_shared(ring);
  float* sums = reinterpret_cast<float*>(smem_raw + WARPS * R * S::kStage);                                  // [2][warp][token][feature]
  const int tiles = (a.N + kCols - 1) / kCols * m_tiles, chunks = (a.K + kF32Chunk - 1) / kF32Chunk, rounds = (chunks + WARPS - 1) / WARPS;
  const int my_tiles = ((int)blockIdx.x < tiles) ? (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0, total_rounds = my_tiles * rounds;
  pdl_launch_dependents();

  // A warp has one chunk a round: chunk warp + WARPS * round of the tile, if there is such a chunk.
  struct Walk {
    int tile, chunk, left;             // left: rounds from here on
  };
  auto next = [&](Walk& w) {           // true where another tile begins
    --w.left;
    w.chunk += WARPS;
    if (w.chunk < rounds * WARPS) return false;
    w.chunk = warp;
    w.tile += gridDim.x;
    return true;
  };
  // The ring is filled R chunks ahead. Rows that do not exist are zeros (no bytes copied).
  Walk ask{(int)blockIdx.x, warp, total_rounds};
  const float* from[2];
  int bytes[2];
  auto aim = [&]() {
    const int n0 = ask.tile / m_tiles * kCols;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int row = g + 8 * r, n = n0 + (GATED ? row % kCols : row);
      bytes[r] = n < a.N ? 16 : 0;
      from[r] = a.W + (bytes[r] ? (size_t)(n + (GATED && row >= kCols ? a.N : 0)) * a.ldw + 4 * t : 0);
    }
  };
  aim();
  uint32_t ask_at = ring_at;
  auto ask_chunk = [&]() {
    if (ask.left > 0) {
      if (ask.chunk < chunks) {
        const int k0 = ask.chunk * kF32Chunk;
        const bool whole = k0 + kF32Chunk <= a.K;
#pragma unroll
        for (int s = 0; s < 4; ++s)
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            const bool in = whole || k0 + 16 * s + 4 * t < a.K;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ask_at + (uint32_t)((s * 2 + r) * 512)), "l"(in ? from[r] + k0 + 16 * s : a.W), "r"(in ? bytes[r] : 0) : "memory");
          }
      }
      if (next(ask) && ask.left > 0) aim();
    }
    copies_commit();
    ask_at = ask_at + S::kStage == ring_at + R * S::kStage ? ring_at : ask_at + S::kStage;
  };

  if (!a.early) pdl_wait();
#pragma unroll 1
  for (int i = 0; i < R; ++i) ask_chunk();
  if (tid == 0) prefetch_share(a.next, blockIdx.x, gridDim.x);

  // The parts of a chunk of weights, formed a round ahead; its stage of the ring is free then.
  uint32_t w[3][4][4];
  int stage = 0;
  auto split_weights = [&](bool there) {
    if (there) {
      copies_wait<R - 1>();
      const float4* weights = ring + stage * (S::kStage / 16);
#pragma unroll
      for (int s = 0; s < 4; ++s)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const float4 v = weights[(s * 2 + r) * 32];
          split2(v.x, v.y, w[0][s][r], w[1][s][r], w[2][s][r]);
          split2(v.z, v.w, w[0][s][2 + r], w[1][s][2 + r], w[2][s][2 + r]);
        }
    }
    stage = stage + 1 == R ? 0 : stage + 1;
    ask_chunk();
  };
  Walk at{(int)blockIdx.x, warp, total_rounds};
  if (a.early) pdl_wait();

  // Rows of A: a lane wants k 4t .. 4t + 3 of each sixteen of row g (of each eight rows), fetched one portion of eight rows ahead. Behind the
  // last row that row is read again: its sums are not stored.
  Walk fetched = at;
  int fetched_nb = 0;
  float4 raw[4];
  auto fetch = [&]() {
    if (fetched.left > 0 && fetched.chunk < chunks) {
      const int m = min((m_tiles == 1 ? 0 : fetched.tile % m_tiles * S::kTokens) + 8 * fetched_nb + g, a.M - 1), k0 = fetched.chunk * kF32Chunk + 4 * t;
      const float* x = a.A + (size_t)m * a.lda + k0;
      if (a.vec && fetched.chunk * kF32Chunk + kF32Chunk <= a.K) {
#pragma unroll
        for (int s = 0; s < 4; ++s) raw[s] = *reinterpret_cast<const float4*>(x + 16 * s);
      } else {
#pragma unroll
        for (int s = 0; s < 4; ++s)
          raw[s] = k0 + 16 * s < a.K ? make_float4(x[16 * s], x[16 * s + 1], x[16 * s + 2], x[16 * s + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    if (++fetched_nb == NB) {
      fetched_nb = 0;
      next(fetched);
    }
  };
  fetch();
  if (total_rounds > 0) split_weights(at.chunk < chunks);      // (while the first rows are on their way)

  float total[GATED ? 2 : 1][kOwn], old[kOwn];
  int round = 0, half = 0;
  for (int r = 0; r < total_rounds; ++r) {
    const int m0 = at.tile % m_tiles * S::kTokens, n0 = at.tile / m_tiles * kCols;
    if (round == 0) {
#pragma unroll
      for (int o = 0; o < kOwn; ++o) {
        const int i = tid + o * S::kThreads, m = m0 + i / kCols, n = n0 + i % kCols;
        total[0][o] = total[GATED ? 1 : 0][o] = 0.0f;
        old[o] = !GATED && i < kOut && m < a.M && n < a.N ? f32_old(a, m, n) : 0.0f;
      }
    }
    float* mine = sums + half * S::kSums;
    const bool there = at.chunk < chunks;
    if (there) {
      float* to = mine + warp * (S::kTokens * S::kStride);
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) {
        uint32_t x[3][4][2];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          split2(raw[s].x, raw[s].y, x[0][s][0], x[1][s][0], x[2][s][0]);
          split2(raw[s].z, raw[s].w, x[0][s][1], x[1][s][1], x[2][s][1]);
        }
        fetch();
        float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        auto product = [&](int s, int pw, int px) {
          mma_16816(d[s >> 1], w[pw][s], x[px][s]);
        };
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int p = 0; p < 3; ++p) {
            const int pw = p == 0 ? 2 : p == 1 ? 0 : 1, px = p == 0 ? 0 : p == 1 ? 2 : 1;
            product(s, pw, px);
            product(s + 2, pw, px);
          }
#pragma unroll
        for (int s = 0; s < 2; ++s)
#pragma unroll
          for (int p = 0; p < 2; ++p) {
            product(s, 1 - p, p);
            product(s + 2, 1 - p, p);
          }
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          product(s, 0, 0);
          product(s + 2, 0, 0);
        }
        to[(8 * nb + 2 * t) * S::kStride + g] = d[0][0] + d[1][0];
        to[(8 * nb + 2 * t + 1) * S::kStride + g] = d[0][1] + d[1][1];
        to[(8 * nb + 2 * t) * S::kStride + g + 8] = d[0][2] + d[1][2];
        to[(8 * nb + 2 * t + 1) * S::kStride + g + 8] = d[0][3] + d[1][3];
      }
    } else {
#pragma unroll
      for (int nb = 0; nb < NB; ++nb) fetch();
    }
    const int first = round * WARPS, last = min(WARPS, chunks - first);
    next(at);
    if (at.left > 0) split_weights(at.chunk < chunks);
    __syncthreads();      // (also: the sums two rounds back have been read)
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const int i = tid + o * S::kThreads;
      if (i >= kOut) break;
      const float* part = mine + (i / kCols) * S::kStride + i % kCols;
#pragma unroll
      for (int v = 0; v < WARPS; v += 2) {
        if (v >= last) break;
        const float* p0 = part + v * (S::kTokens * S::kStride);
        const float* p1 = p0 + S::kTokens * S::kStride;
        total[0][o] += v + 1 < last ? p0[0] + p1[0] : p0[0];
        if constexpr (GATED) total[1][o] += v + 1 < last ? p0[kCols] + p1[kCols] : p0[kCols];
      }
    }
    half ^= 1;
    if (++round < rounds) continue;
    round = 0;
#pragma unroll
    for (int o = 0; o < kOwn; ++o) {
      const int i = tid + o * S::kThreads, m = m0 + i / kCols, n = n0 + i % kCols;
      if (i >= kOut || m >= a.M || n >= a.N) continue;
      if constexpr (GATED) {
        const float gate = f32_checked(a, m, n, total[0][o]), up = f32_checked(a, m, a.N + n, total[1][o]);
        a.C[(size_t)m * a.ldc + n] = gated(a.gate, gate, up);
      } else {
        f32_finish(a, m, n, f32_checked(a, m, n, total[0][o]), old[o]);
      }
    }
  }
}

template <int NB, int WARPS, bool GATED>
static int launch_fr(const F32Args& a, cudaStream_t s) {
  using S = FrShape<NB, WARPS>;
  const auto kernel = gemm_f32_split_rows_kernel<NB, WARPS, GATED>;
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, S::kSmem, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32_rows: cannot reserve %d bytes of shared memory: %s", S::kSmem, cudaGetErrorString(e));
  constexpr int kCols = GATED ? kFrRows / 2 : kFrRows;
  const int m_tiles = (a.M + S::kTokens - 1) / S::kTokens, tiles = (a.N + kCols - 1) / kCols * m_tiles, room = (WARPS == 8 ? 2 : 1) * sm_count();
  const bool early = a.early ? pdl_mode() != 0 : pdl_mode() == 1;
  launch_with(early, kernel, dim3((unsigned)(tiles < room ? tiles : room)), dim3(S::kThreads), (size_t)S::kSmem, s, a, m_tiles);
  return check_launch("gemm_f32_rows");
}

// A block of sixteen warps an SM, or two of eight: in rounds of a chunk a warp, which cost the same with sixteen warps an SM either way; one
// block's rounds are a little dearer (no other block works while it stands at a barrier), half an SM's a little cheaper. Fitted to products of 1 to 64
// rows by 512 to 151,936 x 1,024 to 9,728.
struct FrPlan {
  bool wide;
  double rounds;
};
static FrPlan fr_plan(int M, long long w_rows, int K) {
  const long long tokens = M <= 8 ? 8 : M <= 16 ? 16 : 32, tiles = (w_rows + kFrRows - 1) / kFrRows * ((M + tokens - 1) / tokens);
  const long long chunks = (K + kF32Chunk - 1) / kF32Chunk, sms = sm_count();
  const double narrow = (double)((tiles + 2 * sms - 1) / (2 * sms) * ((chunks + 7) / 8)) * (tiles <= sms ? 0.8 : 1.0);
  const double wide = (double)((tiles + sms - 1) / sms * ((chunks + 15) / 16)) * (tokens == 8 ? 1.34 : 1.08);
  return wide < narrow ? FrPlan{true, wide} : FrPlan{false, narrow};
}

double f32_rows_cost(int M, int N, int K) { return 1200.0 + fr_plan(M, N, K).rounds * (M <= 8 ? 1600.0 : M <= 16 ? 2650.0 : 4500.0); }

template <int NB, bool GATED>
static int launch_fr_tokens(const F32Args& a, cudaStream_t s) {
  return fr_plan(a.M, GATED ? 2ll * a.N : a.N, a.K).wide ? launch_fr<NB, 16, GATED>(a, s) : launch_fr<NB, 8, GATED>(a, s);
}

template <bool GATED>
static int launch_fr_all(const F32Args& a, cudaStream_t s) {
  return a.M <= 8 ? launch_fr_tokens<1, GATED>(a, s) : a.M <= 16 ? launch_fr_tokens<2, GATED>(a, s) : launch_fr_tokens<4, GATED>(a, s);
}

int launch_f32_rows(const F32Args& a, bool gated, cudaStream_t s) { return gated ? launch_fr_all<true>(a, s) : launch_fr_all<false>(a, s); }

}  // namespace slb
