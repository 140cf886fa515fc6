// What the forms of the 32-bit product on the tensor cores share (gemm_f32_tc.cu for many rows, gemm_f32_rows.cu for few): the operands, the split
// of a float32 value into bfloat16 parts, the order of the sums, and how a result is stored.
#pragma once

#include "packed_f32.cuh"

namespace slb {

// The FMA kernels' segments of K (gemm_f32.cu).
constexpr int kMaxSegments = 8;
// k values in a segment: an eighth of K in whole 64s, at least 128.
__host__ __device__ inline int segment_length(int K) {
  const int len = ((K + kMaxSegments * 64 - 1) / (kMaxSegments * 64)) * 64;
  return len < 128 ? 128 : len;
}

// Order of the sums: K in chunks of 64; a chunk is two chains of kF32Steps products of 16 values each, the small partial products of a chain
// first, and its sum is chain 0 + chain 1; the chunks' sums are added two by two, and these pairs in ascending order:
//     C = ((pair 0 + pair 1) + pair 2) + ...,  pair p = chunk 2p + chunk 2p + 1
constexpr int kF32Chunk = 64, kF32Steps = 2, kF32Partial = 2;

// Both operands are split after multiplication by 2^24: the last bit of a float32 value, 2^-149 at least, is then a normal bfloat16 value, and the
// three parts add up to the value exactly however small it is. Results are divided by 2^48. From 2^104 (operands) or 2^80 (results) on a sum is not
// finite and is formed again, by FMA.
constexpr float kF32Scale = 16777216.0f, kF32Unscale = 1.0f / (16777216.0f * 16777216.0f);

struct F32Args {
  const float* A;
  const float* W;
  const float* bias;
  float* C;
  int M, N, K, lda, ldw, ldc, accumulate;
  int early;             // no kernel writes W: it is fetched before the wait for the kernel in front
  int vec;               // A's rows can be read 16 bytes at a time
  GateAct gate;          // gated forms: W holds N gate rows, then N up rows; C = act(gate) * up
  int* status;
  NextRead next;         // what the kernel after this one reads, or nothing (the form for few rows asks L2 for it)
};

// Two values into their three parts, packed as the tensor core reads them (the first in the low half).
__device__ __forceinline__ void split2(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  f32x2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(x), "f"(y));
  v = mul2(v, both(kF32Scale));
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

// The result of one output as the FMA kernels form it (gemm_f32.cu), for results that are not finite.
// (Not a call: what a call saves would be spilled around the products.)
__device__ __forceinline__ float f32_plain_dot(const F32Args& a, int m, int n) {
  const float *x = a.A + (size_t)m * a.lda, *w = a.W + (size_t)n * a.ldw;
  const int len = segment_length(a.K);
  float sum = 0.0f;
#pragma unroll 1
  for (int k0 = 0; k0 < a.K; k0 += len) {
    float v = 0.0f;
    const int end = min(a.K, k0 + len);
#pragma unroll 1
    for (int k = k0; k < end; ++k) v = fmaf(x[k], w[k], v);
    sum = k0 ? sum + v : v;
  }
  return sum;
}
__device__ __forceinline__ float f32_checked(const F32Args& a, int m, int n, float v) { return isfinite(v) ? v * kF32Unscale : f32_plain_dot(a, m, n); }
__device__ __forceinline__ float f32_old(const F32Args& a, int m, int n) { return a.accumulate ? a.C[(size_t)m * a.ldc + n] : 0.0f; }
__device__ __forceinline__ void f32_finish(const F32Args& a, int m, int n, float v, float old) {
  if (a.bias) v += a.bias[n];
  a.C[(size_t)m * a.ldc + n] = a.accumulate ? old + v : v;
}

// The form for few rows (gemm_f32_rows.cu); gated: with the activation of a.gate.
int launch_f32_rows(const F32Args& a, bool gated, cudaStream_t s);
double f32_rows_cost(int M, int N, int K);      // about what it takes, in ns

}  // namespace slb
