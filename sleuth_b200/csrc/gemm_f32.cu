// The true 32-bit matrix product: C[M, N] (+)= A[M, K] * W[N, K]^T (+ bias[N]), float32 in, float32 out,
// plain FMA on the CUDA cores. No tensor-core mode of any kind is involved, so nothing is rounded below float32.
// It serves matrices with an inner dimension below 1,024 or less than 512 features and those whose rows no 16-byte reads take; the others go to the
// tensor cores (gemm_f32_tc.cu, gemm_f32_rows.cu).
//
// The order of every sum depends on K alone. K is cut into at most eight segments (segment_length); a segment is one
// chain acc = fmaf(a[k], w[k], acc) with k ascending, and the segments' sums are added in ascending order. Both kernels
// below do exactly this, whatever tile they take and whatever M is. A row's result therefore does not depend on how many
// rows run together, which is what lets the 32-bit path give the same logits for a whole prompt, for single tokens and
// for any batch. With few rows the segments are the only parallelism a narrow matrix has; shorter chains also round less.
// (The reference has no such path on the GPU: its float32 models run under bfloat16 autocast there,
// sleuth/forge/infer/generate.py:76-77.)
#include "gemm_f32_split.cuh"

namespace slb {

// Tiles that a block of the streaming kernel takes side by side, with `room` blocks for `tiles` tiles: no more than its warps have
// segments for, and none while blocks are to be had, where joining the tiles' sums takes as long as forming them (K below 64) or
// where three and more segments keep the block busy (8 rows x 12,288 x 384: 14.3 us, two side by side 16.4).
static int groups_of(int K, int tiles, int room) {
  const int segments = (K + segment_length(K) - 1) / segment_length(K), most = kMaxSegments / segments, want = (tiles + room - 1) / room;
  return K < 64 || segments > 2 ? 1 : want < most ? want : most;
}

struct GemmF32Args {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int M, N, K, lda, ldw, ldc, accumulate;
  int early;             // W is fetched before the wait for the kernel in front: only where no kernel writes it
};

// ---- few rows -------------------------------------------------------------------------------------------------
// Up to MP rows (and tiles of MP rows beyond). What bounds it is the weight stream and, from some 8 rows on, what shared memory
// can deliver (a lane's 16-byte read costs its full 16 bytes of 128 a cycle, broadcast or not). So warp w of a block owns segment
// w of K, and streams its part of the block's weight rows (NT features), with the token rows' values for the same k, through a
// ring of its own: CH k values a stage, D stages, 16-byte asynchronous copies, no barrier between warps until a tile's sums are
// joined. With one or two segments (K up to 256) and more tiles than blocks a block takes several tiles side by side (SIDE), group
// g of its warps tile base + g (16 rows x 32,768 x 96: 22.5 us one at a time, 16.4 side by side). A block goes from tile to tile with the ring running on, so its copies never drain. Where the
// caller says that no kernel writes W, the first stages' weights are asked for before the wait for the kernel in front. LM lanes along the rows and 32 / LM along the features
// make each lane's block R x CN as square as the tile allows. 0.6B sizes, 8 rows, us before (one chain per output over all of K, slices of
// 32 k values behind barriers) / now: q/k/v 25.1 / 5.9, o 50.2 / 7.6, gate and up 34.9 / 9.1, down 74.5 / 10.8, head 479 / 145; 64 rows:
// q/k/v 238 / 22.9, o 456 / 17.8.
template <int MP, int NT, int CH, int D, bool VEC>
struct RowsShape {
  static constexpr int LM = MP >= 64 ? 8 : (MP < 4 ? MP : 4);       // lanes along the rows
  static constexpr int LN = NT < 32 / LM ? NT : 32 / LM;           // lanes along the features
  static constexpr int R = MP / LM, CN = NT / LN;
  static constexpr int kRow = CH + 4;                              // floats: 16-byte reads of 8 rows hit 8 different bank groups
  static constexpr int kStage = (NT + MP) * kRow;
  static constexpr int kJoinBuffers = MP * NT >= 512 ? 1 : 2;
  static constexpr int kSmem = (kMaxSegments * D * kStage + kJoinBuffers * kMaxSegments * MP * NT) * 4;
  static constexpr int kBlocksPerSm = kSmem <= 113 * 1024 ? 2 : 1;
};

template <int MP, int NT, int CH, int D, bool VEC, bool SIDE>
__global__ void __launch_bounds__(256, (RowsShape<MP, NT, CH, D, VEC>::kBlocksPerSm))
gemm_f32_rows_kernel(GemmF32Args a, int seg, int tiles, int groups) {
  using S = RowsShape<MP, NT, CH, D, VEC>;
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lm = lane % S::LM, ln = (lane / S::LM) % S::LN;
  float* ring = smem + warp * (D * S::kStage);
  float* join = smem + kMaxSegments * D * S::kStage;
  const int m0 = blockIdx.y * MP, rows = min(MP, a.M - m0);
  const int segments = (a.K + seg - 1) / seg, group = SIDE ? warp / segments : 0, stride = SIDE ? gridDim.x * groups : gridDim.x;
  const int k_begin = (SIDE ? warp % segments : warp) * seg, k_len = SIDE && group >= groups ? 0 : max(0, min(seg, a.K - k_begin));
  const int chunks = (k_len + CH - 1) / CH;

  // A copy brings kCopy k values of one row; a warp's copy instruction kRowsPer rows (or 1 / kTurns of one). Lane: row lr, k value lk.
  constexpr int kCopy = VEC ? 4 : 1, kPerRow = CH / kCopy;
  constexpr int kRowsPer = kPerRow < 32 ? 32 / kPerRow : 1, kTurns = kPerRow < 32 ? 1 : kPerRow / 32;
  const int lr = kPerRow < 32 ? lane / kPerRow : 0, lk = (lane % kPerRow) * kCopy;
  const float* a_lane = a.A + (size_t)(m0 + min(lr, rows - 1)) * a.lda + k_begin + lk;
  auto copy_rows = [&](float* dst, const float* src, size_t ld, int count, int most, int k0) {      // src: this lane's row lr, chunk 0
    float* d = dst + lr * S::kRow + lk;
#pragma unroll
    for (int turn = 0; turn < kTurns; ++turn) {
      const int k = k0 + lk + 32 * turn;
      const int bytes = k < k_len ? 4 * kCopy : 0;
      const float* p = bytes ? src + k0 + 32 * turn : src - lk;      // (nothing is read there)
#pragma unroll
      for (int r = 0; r < most; r += kRowsPer) {
        if (r + lr < count) copy_async<VEC>(d + r * S::kRow + 32 * turn, p, bytes);
        p += kRowsPer * ld;
      }
    }
  };
  // the stage after the last one asked for: its tile and its chunk
  int ask_tile = SIDE ? blockIdx.x * groups + group : blockIdx.x, ask_chunk = 0, ask_slot = 0;
  auto ask_weights = [&]() {
    const int n0 = ask_tile * NT;
    copy_rows(ring + ask_slot * S::kStage, a.W + (size_t)(n0 + lr) * a.ldw + k_begin + lk, a.ldw, a.N - n0, NT, ask_chunk * CH);
  };
  auto ask_tokens = [&](int chunk, int slot) {
    copy_rows(ring + slot * S::kStage + NT * S::kRow, a_lane, a.lda, rows, MP, chunk * CH);
  };
  auto advance = [&]() {
    if (++ask_chunk == chunks) { ask_chunk = 0; ask_tile += stride; }
    if (++ask_slot == D) ask_slot = 0;
  };

  pdl_launch_dependents();
  if (!a.early) pdl_wait();
  if (chunks) {
    for (int s = 0; s < D - 1; ++s) {
      if (ask_tile < tiles) ask_weights();
      advance();
    }
  }
  if (a.early) pdl_wait();
  if (chunks) {
    for (int s = 0, c = 0; s < D - 1; ++s) {
      ask_tokens(c, s);       // (beyond the last tile: copied and not used)
      if (++c == chunks) c = 0;
      copies_commit();
    }
  }

  constexpr int kOut = (MP * NT + 255) / 256;
  int slot = 0, buffer = 0;
  for (int base = SIDE ? blockIdx.x * groups : blockIdx.x; base < tiles; base += stride) {
    const int n0 = base * NT;
    float old[kOut];      // (of the first tile; the others' are read when they are needed)
#pragma unroll
    for (int i = 0; i < kOut; ++i) {
      const int idx = tid + 256 * i, r = idx / NT, n = n0 + idx % NT;
      old[i] = (a.accumulate && idx < MP * NT && r < rows && n < a.N) ? a.C[(size_t)(m0 + r) * a.ldc + n] : 0.0f;
    }
    float acc[S::R][S::CN];
#pragma unroll
    for (int i = 0; i < S::R; ++i)
#pragma unroll
      for (int j = 0; j < S::CN; ++j) acc[i][j] = 0.0f;
    for (int c = 0; c < chunks; ++c) {
      copies_wait<D - 2>();
      __syncwarp();
      const float* ws = ring + slot * S::kStage + ln * S::kRow;
      const float* as = ring + slot * S::kStage + (NT + lm) * S::kRow;
      if (++slot == D) slot = 0;
      if (ask_tile < tiles) {
        ask_weights();
        ask_tokens(ask_chunk, ask_slot);
      }
      advance();
      copies_commit();
      auto quad = [&](int k) {
        float4 av[S::R];
#pragma unroll
        for (int i = 0; i < S::R; ++i) av[i] = *reinterpret_cast<const float4*>(as + i * S::LM * S::kRow + k);
#pragma unroll
        for (int j = 0; j < S::CN; ++j) {
          const float4 wv = *reinterpret_cast<const float4*>(ws + j * S::LN * S::kRow + k);
#pragma unroll
          for (int i = 0; i < S::R; ++i) acc[i][j] = fmaf(av[i].x, wv.x, acc[i][j]);
#pragma unroll
          for (int i = 0; i < S::R; ++i) acc[i][j] = fmaf(av[i].y, wv.y, acc[i][j]);
#pragma unroll
          for (int i = 0; i < S::R; ++i) acc[i][j] = fmaf(av[i].z, wv.z, acc[i][j]);
#pragma unroll
          for (int i = 0; i < S::R; ++i) acc[i][j] = fmaf(av[i].w, wv.w, acc[i][j]);
        }
      };
      const int kn = k_len - c * CH;
      if (kn >= CH) {
#pragma unroll
        for (int k = 0; k < CH; k += 4) quad(k);
      } else {
        for (int k = 0; k < kn; k += 4) quad(k);
      }
    }
    // the segments' sums, joined in ascending order
    float* mine = join + (buffer * kMaxSegments + warp) * (MP * NT);
    if (lane < S::LM * S::LN) {
#pragma unroll
      for (int i = 0; i < S::R; ++i)
#pragma unroll
        for (int j = 0; j < S::CN; ++j) mine[(lm + i * S::LM) * NT + ln + j * S::LN] = acc[i][j];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kOut; ++i) {
      const int idx = tid + 256 * i, r = idx / NT, n = n0 + idx % NT;
      if (idx >= MP * NT || r >= rows || n >= a.N) continue;
      const float* p = join + buffer * kMaxSegments * (MP * NT) + idx;
      float v = p[0];
#pragma unroll
      for (int s = 1; s < kMaxSegments; ++s)
        if (s < segments) v += p[s * (MP * NT)];
      if (a.bias) v += a.bias[n];
      a.C[(size_t)(m0 + r) * a.ldc + n] = a.accumulate ? old[i] + v : v;
    }
    for (int idx = MP * NT + tid; SIDE && idx < groups * (MP * NT); idx += 256) {
      const int g = idx / (MP * NT), e = idx % (MP * NT), r = e / NT, n = n0 + g * NT + e % NT;
      if (r >= rows || n >= a.N) continue;
      const float* p = join + (buffer * kMaxSegments + g * segments) * (MP * NT) + e;
      float v = p[0];
      for (int s = 1; s < segments; ++s) v += p[s * (MP * NT)];
      if (a.bias) v += a.bias[n];
      float* c = a.C + (size_t)(m0 + r) * a.ldc + n;
      *c = a.accumulate ? *c + v : v;
    }
    if (S::kJoinBuffers == 2) buffer ^= 1;      // two buffers: the next tile's barrier stands between these reads and the next writes
    else __syncthreads();
  }
  copies_wait<0>();
}

// ---- many rows ------------------------------------------------------------------------------------------------
// A tile of 16 * RT rows by 128 features per block of 256 threads, RT x 8 outputs per thread, two blocks an SM where there are tiles
// enough. What bounds it is the FMA pipe and, level with it, what shared memory delivers (a k value is RT + 8 floats read per thread
// for 8 * RT FMAs). Operands go through registers into shared memory k-major, kTileK k values at a time, two buffers: a warp's
// reads are then float4 of four rows or features; the FMAs go in packed pairs of neighbouring features. The sums of finished
// segments wait in shared memory, each thread its own (SINGLE: K is one segment, and they stay in registers). 3,000 rows x 6,144 x 1,024: 784 us, 48 TFLOP/s, as without packing and
// segments before; measured and left: tiles of 64 x 128 with 8 x 16 outputs a thread and transposing 4-byte copies (856 us: a
// quarter less to read from shared memory, but two warps a scheduler do not cover its latency), row-major operands with pairs
// along k (910 us).
constexpr int kTileK = 16, kTileN = 128, kTileWRow = kTileN + 4;
constexpr int tile_smem(int rt) { return (2 * kTileK * (16 * rt + 4 + kTileWRow) + 256 * rt * 8) * 4; }

template <int RT, bool VEC, bool SINGLE>
__global__ void __launch_bounds__(256, 2) gemm_f32_tile_kernel(GemmF32Args a, int seg) {
  extern __shared__ __align__(16) float smem[];
  constexpr int BM = 16 * RT, kARow = BM + 4, kBuffer = kTileK * (kARow + kTileWRow);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * kTileN;
  // this thread's rows: 4 * ty + 0..3, then 64 + (RT - 4) * ty + 0..RT - 5; its features: 4 * tx + 0..3 and 64 + 4 * tx + 0..3
  float4* totals = reinterpret_cast<float4*>(smem + 2 * kBuffer) + tid;       // [2 * RT][256]
  // its share of a slice: k values lk .. lk + 3 of rows and features lr, lr + 64
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  const float* ap[2];
  const float* wp[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    ap[h] = a.A + (size_t)min(m0 + lr + 64 * h, a.M - 1) * a.lda + lk;       // beyond the matrix: its last row, whose results are not stored
    wp[h] = a.W + (size_t)min(n0 + lr + 64 * h, a.N - 1) * a.ldw + lk;
  }
  float4 pa[2], pw[2];
  auto four = [&](const float* src, int k0) {
    if (VEC) return k0 + lk < a.K ? *reinterpret_cast<const float4*>(src + k0) : make_float4(0.f, 0.f, 0.f, 0.f);      // K is a multiple of 4
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k0 + lk < a.K) v.x = src[k0];
    if (k0 + lk + 1 < a.K) v.y = src[k0 + 1];
    if (k0 + lk + 2 < a.K) v.z = src[k0 + 2];
    if (k0 + lk + 3 < a.K) v.w = src[k0 + 3];
    return v;
  };
  constexpr bool kTwo = RT > 4;
  const bool second = RT == 8 || lr < BM - 64;
  auto fetch_weights = [&](int k0) { pw[0] = four(wp[0], k0); pw[1] = four(wp[1], k0); };
  auto fetch_tokens = [&](int k0) { pa[0] = four(ap[0], k0); if (kTwo && second) pa[1] = four(ap[1], k0); };
  auto put = [&](int buffer) {
    float* as = smem + buffer * kBuffer + lk * kARow + lr;
    float* ws = smem + buffer * kBuffer + kTileK * kARow + lk * kTileWRow + lr;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h == 0 || (kTwo && second)) {
        as[64 * h] = pa[h].x; as[kARow + 64 * h] = pa[h].y; as[2 * kARow + 64 * h] = pa[h].z; as[3 * kARow + 64 * h] = pa[h].w;
      }
      ws[64 * h] = pw[h].x; ws[kTileWRow + 64 * h] = pw[h].y; ws[2 * kTileWRow + 64 * h] = pw[h].z; ws[3 * kTileWRow + 64 * h] = pw[h].w;
    }
  };
  pdl_launch_dependents();
  if (!a.early) pdl_wait();
  fetch_weights(0);
  if (a.early) pdl_wait();
  fetch_tokens(0);

  f32x2 acc[RT][4];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0;
  if (!SINGLE)
#pragma unroll
    for (int e = 0; e < 2 * RT; ++e) totals[e * 256] = make_float4(0.f, 0.f, 0.f, 0.f);
  put(0);
  __syncthreads();

  int buffer = 0, left = seg;
  for (int k0 = 0; k0 < a.K; k0 += kTileK) {
    const bool more = k0 + kTileK < a.K;
    if (more) { fetch_weights(k0 + kTileK); fetch_tokens(k0 + kTileK); }
    const float* as = smem + buffer * kBuffer + 4 * ty;
    const float* as2 = smem + buffer * kBuffer + 64 + (RT - 4) * ty;
    const float* ws = smem + buffer * kBuffer + kTileK * kARow + 4 * tx;
    auto one = [&](int k) {
      float av[RT];
      *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(as + k * kARow);
      if (RT == 8) *reinterpret_cast<float4*>(av + 4) = *reinterpret_cast<const float4*>(as2 + k * kARow);
      if (RT == 6) *reinterpret_cast<float2*>(av + 4) = *reinterpret_cast<const float2*>(as2 + k * kARow);
      ulonglong2 wv[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(ws + k * kTileWRow + 64 * j);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const f32x2 v = both(av[i]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          acc[i][2 * j] = fma2(v, wv[j].x, acc[i][2 * j]);
          acc[i][2 * j + 1] = fma2(v, wv[j].y, acc[i][2 * j + 1]);
        }
      }
    };
    const int kn = a.K - k0;
    if (kn >= kTileK) {
#pragma unroll
      for (int k = 0; k < kTileK; ++k) one(k);
    } else {
      for (int k = 0; k < kn; ++k) one(k);
    }
    left -= kTileK;
    if (!SINGLE && (left == 0 || !more)) {      // a segment is done (segments are whole multiples of 64)
      left = seg;
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float4 t = totals[(2 * i + j) * 256];
          t.x += low_half(acc[i][2 * j]);
          t.y += high_half(acc[i][2 * j]);
          t.z += low_half(acc[i][2 * j + 1]);
          t.w += high_half(acc[i][2 * j + 1]);
          totals[(2 * i + j) * 256] = t;
          acc[i][2 * j] = acc[i][2 * j + 1] = 0;
        }
    }
    if (more) {
      buffer ^= 1;
      put(buffer);
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    const int gm = m0 + (i < 4 ? 4 * ty + i : 64 + (RT - 4) * ty + i - 4);
    if (gm >= a.M) continue;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float4 t = SINGLE ? make_float4(low_half(acc[i][2 * j]), high_half(acc[i][2 * j]), low_half(acc[i][2 * j + 1]), high_half(acc[i][2 * j + 1]))
                              : totals[(2 * i + j) * 256];
      const float tv[4] = {t.x, t.y, t.z, t.w};
      float* c = a.C + (size_t)gm * a.ldc + n0 + 4 * tx + 64 * j;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int gn = n0 + 4 * tx + 64 * j + e;
        if (gn >= a.N) continue;
        float v = tv[e];
        if (a.bias) v += a.bias[gn];
        c[e] = a.accumulate ? c[e] + v : v;
      }
    }
  }
}

template <int MP, int NT, int CH, int D, bool VEC, bool SIDE>
static int launch_rows_form(const GemmF32Args& a, int tiles, int row_tiles, int room, int groups, cudaStream_t s) {
  using S = RowsShape<MP, NT, CH, D, VEC>;
  static_assert(S::kSmem <= 227 * 1024, "the ring must fit shared memory");
  const auto kernel = gemm_f32_rows_kernel<MP, NT, CH, D, VEC, SIDE>;
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, S::kSmem, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32: cannot reserve %d bytes of shared memory: %s", S::kSmem, cudaGetErrorString(e));
  const int shares = (tiles + groups - 1) / groups;
  launch_with(a.early ? pdl_mode() != 0 : pdl_mode() == 1, kernel, dim3(shares < room ? shares : room, row_tiles), dim3(256), S::kSmem, s, a, segment_length(a.K), tiles, groups);
  return check_launch("gemm_f32 (few rows)");
}
template <int MP, int NT, int CH, int D, bool VEC>
static int launch_rows(const GemmF32Args& a, cudaStream_t s) {
  using S = RowsShape<MP, NT, CH, D, VEC>;
  const int tiles = (a.N + NT - 1) / NT, row_tiles = (a.M + MP - 1) / MP;
  SLB_REQUIRE(row_tiles < 65536, "gemm_f32: M=%d needs more than 65535 row tiles", a.M);
  const int room = S::kBlocksPerSm * sm_count() / row_tiles > 1 ? S::kBlocksPerSm * sm_count() / row_tiles : 1;
  const int groups = groups_of(a.K, tiles, room);
  return groups > 1 ? launch_rows_form<MP, NT, CH, D, VEC, true>(a, tiles, row_tiles, room, groups, s)
                    : launch_rows_form<MP, NT, CH, D, VEC, false>(a, tiles, row_tiles, room, 1, s);
}

// Which kernel and tile a product takes: the sum of its rounds over the SMs, in nanoseconds, fitted to 2,239 products of 32 to 4,099
// by 130 to 32,768 with 1 to 3,000 rows on a B200 (the sums meet the times above a launch's 7 us within 4 to 7 % rms, 20 % at worst). A round
// costs a fixed part, which decides where K is small, and a part per k value; tiles of several rounds run two a SM. us, streaming / tiles:
// 600 rows x 1,024 x 77 43 / 18; 128 x 6,144 x 160 41 / 18; 48 x 32,768 x 160 87 / 29; 300 x 1,024 x 2,048 84 / 142.
struct TileCost {
  double alone, alone_k, two, two_k;      // a round with one tile an SM; with two
};
constexpr TileCost kTile8{830, 104, 2490, 193}, kTile6{850, 82.6, 1720, 155.6}, kTile4{140, 66, 1110, 121}, kTile8Odd{1650, 105.4, 2910, 199};

static long long tiles_of(int M, int N, int rt) { return (long long)((N + kTileN - 1) / kTileN) * ((M + 16 * rt - 1) / (16 * rt)); }
static double tile_cost(int M, int N, int K, int rt, const TileCost& c, long long sms) {
  const long long tiles = tiles_of(M, N, rt), rest = tiles % (2 * sms);
  const double alone = c.alone + c.alone_k * K, two = c.two + c.two_k * K;
  return (double)(tiles / (2 * sms)) * two + (rest == 0 ? 0.0 : rest <= sms ? alone : two);
}

// The streaming kernel's tiles of mp rows by nt features, one block an SM: per tile of a round, per k value of it, per k value of a chain;
// one tile a block at a time, and several side by side.
struct RowsCost {
  int mp, nt;
  double tile, k, chain, side_tile, side_k, side_chain;
};
constexpr RowsCost kRows64{64, 32, 3880, 11.8, 42, 1190, 12.2, 81}, kRows32{32, 32, 1030, 5.8, 26, 960, 5.6, 39}, kRowsOdd{64, 8, 430, 3.8, 37, 670, 0, 76};

static double rows_cost(int M, int N, int K, const RowsCost& c, long long sms) {
  const long long down = (M + c.mp - 1) / c.mp, tiles = (N + c.nt - 1) / c.nt, room = sms / down > 1 ? sms / down : 1;
  const long long groups = groups_of(K, (int)tiles, (int)room), shares = (tiles + groups - 1) / groups, blocks = shares < room ? shares : room;
  const long long rounds = (shares + blocks - 1) / blocks * ((blocks * down + sms - 1) / sms);
  const int chain = K < segment_length(K) ? K : segment_length(K);
  return rounds * (groups == 1 ? c.tile + c.k * K + c.chain * chain : groups * (c.side_tile + c.side_k * K) + c.side_chain * chain);
}

// 0: the streaming kernel; 8, 6 or 4: tiles with so many rows a thread. Up to 16 rows, and up to 64 where the features give the
// streaming kernel's narrow tiles a round to themselves, nothing else comes near it.
static int choose_f32(int M, int N, int K, bool vec) {
  if (M <= 16 || (vec && M <= 64 && N < (M <= 32 ? 4096 : 2048))) return 0;
  const int sms = sm_count();
  if (!vec) return rows_cost(M, N, K, kRowsOdd, sms) <= tile_cost(M, N, K, 8, kTile8Odd, sms) ? 0 : 8;
  const double t8 = tile_cost(M, N, K, 8, kTile8, sms), t6 = tile_cost(M, N, K, 6, kTile6, sms), t4 = tile_cost(M, N, K, 4, kTile4, sms);
  const int rt = t8 <= t6 ? (t8 <= t4 ? 8 : 4) : (t6 <= t4 ? 6 : 4);
  return rows_cost(M, N, K, M <= 32 ? kRows32 : kRows64, sms) <= (rt == 8 ? t8 : rt == 6 ? t6 : t4) ? 0 : rt;
}

template <int RT, bool VEC, bool SINGLE>
static int launch_tile_form(const GemmF32Args& a, cudaStream_t s) {
  const auto kernel = gemm_f32_tile_kernel<RT, VEC, SINGLE>;
  // One block an SM is asked for (by its shared memory) where every tile gets an SM of its own: left to itself a kernel that
  // starts while the one before still runs finds half-empty SMs and doubles up there (1,500 x 1,024 x 2,048: 276 instead of 176 us).
  constexpr int kAlone = 116 * 1024;
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)kernel, kAlone, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_f32: cannot reserve %d bytes of shared memory: %s", kAlone, cudaGetErrorString(e));
  const dim3 grid((a.N + kTileN - 1) / kTileN, (a.M + 16 * RT - 1) / (16 * RT));
  SLB_REQUIRE(grid.y < 65536, "gemm_f32: M=%d needs more than 65535 row tiles", a.M);
  const int smem = tiles_of(a.M, a.N, RT) <= sm_count() ? kAlone : tile_smem(RT);
  launch_with(a.early ? pdl_mode() != 0 : pdl_mode() == 1, kernel, grid, dim3(256), smem, s, a, segment_length(a.K));
  return check_launch("gemm_f32 (tiles)");
}
template <int RT, bool VEC>
static int launch_tile(const GemmF32Args& a, cudaStream_t s) {
  return a.K <= segment_length(a.K) ? launch_tile_form<RT, VEC, true>(a, s) : launch_tile_form<RT, VEC, false>(a, s);
}

}  // namespace slb

using namespace slb;

// What slb_gemm_f32 takes: 0 the streaming kernel, 8, 6 or 4 tiles with so many rows a thread (vec: operands that 16-byte reads can take).
extern "C" int slb_gemm_f32_choice(int M, int N, int K, int vec) { return choose_f32(M, N, K, vec != 0); }

// static_weight: no kernel writes W (a loaded matrix), so that it may be read while the kernel in front of this one still runs.
extern "C" int slb_gemm_f32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, int lda,
                            int ldw, int ldc, int accumulate, int static_weight, void* stream) {
  SLB_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: M=%d N=%d K=%d", M, N, K);
  SLB_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: leading dimensions lda=%d ldw=%d ldc=%d for K=%d N=%d", lda,
              ldw, ldc, K, N);
  if (M == 0) return 0;
  cudaStream_t s = (cudaStream_t)stream;
  const GemmF32Args a{A, W, bias, C, M, N, K, lda, ldw, ldc, accumulate, static_weight};
  const bool vec = (K % 4 == 0) && (lda % 4 == 0) && (ldw % 4 == 0) && ((uintptr_t)A % 16 == 0) && ((uintptr_t)W % 16 == 0);
  const int rt = choose_f32(M, N, K, vec);
  if (rt == 0 && !vec) {      // no 16-byte reads: copies of four bytes
    if (M <= 16) return launch_rows<16, 8, 32, 2, false>(a, s);
    return launch_rows<64, 8, 32, 2, false>(a, s);
  }
  if (rt == 0) {
    // 32 features a tile where that still gives every SM one, else 16 or 8
    const int nt = N >= 4096 ? 32 : (N >= 2048 ? 16 : 8);
    if (M <= 1) return nt >= 16 ? launch_rows<1, 16, 64, 4, true>(a, s) : launch_rows<1, 8, 64, 4, true>(a, s);
    if (M <= 2) return nt >= 16 ? launch_rows<2, 16, 64, 3, true>(a, s) : launch_rows<2, 8, 64, 4, true>(a, s);
    if (M <= 4) return nt == 32 ? launch_rows<4, 32, 32, 4, true>(a, s) : nt == 16 ? launch_rows<4, 16, 64, 2, true>(a, s) : launch_rows<4, 8, 64, 3, true>(a, s);
    if (M <= 8) return nt == 32 ? launch_rows<8, 32, 32, 4, true>(a, s) : nt == 16 ? launch_rows<8, 16, 64, 2, true>(a, s) : launch_rows<8, 8, 64, 3, true>(a, s);
    if (M <= 16) return nt == 32 ? launch_rows<16, 32, 32, 3, true>(a, s) : nt == 16 ? launch_rows<16, 16, 32, 2, true>(a, s) : launch_rows<16, 8, 32, 3, true>(a, s);
    if (M <= 32) return nt == 32 ? launch_rows<32, 32, 32, 2, true>(a, s) : nt == 16 ? launch_rows<32, 16, 32, 3, true>(a, s) : launch_rows<32, 8, 32, 2, true>(a, s);
    if (M <= 64 && nt == 8) return launch_rows<64, 8, 32, 2, true>(a, s);
    return launch_rows<64, 32, 16, 2, true>(a, s);
  }
  if (!vec) return launch_tile<8, false>(a, s);
  if (rt == 8) return launch_tile<8, true>(a, s);
  if (rt == 6) return launch_tile<6, true>(a, s);
  return launch_tile<4, true>(a, s);
}
