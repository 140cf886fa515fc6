// bfloat16 matrix product for a few to 64 rows on the fifth-generation tensor cores: C[M, N] = X[M, K] * W[N, K]^T, float32 sums.
//
// What bounds such a product is the stream of the weights. So the weights are the instruction's rows (128 features of a tile, however few
// tokens there are) and the tokens its columns (NT = 16 to 64); K is shared out over a cluster of 1 to 8 blocks, so that narrow
// matrices too keep most SMs loading. A block has a ring of 64-wide slices, about 100 KB, in half an SM's shared memory, and where no
// kernel writes W it asks for the ring's weights before the kernel in front has finished. Per slice one lane issues four tcgen05.mma; the
// sums leave tensor memory through shared memory ([token][feature], in the ring's place), and each block of the cluster adds up the partial
// sums of its share of the tokens, in the order of the blocks, through distributed shared memory, and stores whole lines.
//
// Epilogues: store bfloat16, store float32, add into a float32 matrix, or act(gate) * up for a W that holds the gate rows followed
// by the up rows (a tile is then 64 gate rows and the 64 up rows that match them).
#include "tcgen05.cuh"

namespace slb {

constexpr int kGsK = 64, kGsFeatures = 128, kGsThreads = 192, kGsW = kGsFeatures * kGsK * 2;

enum GsMode : int { kGsBf16 = 0, kGsF32 = 1, kGsAddF32 = 2, kGsGated = 3 };

struct GsArgs {
  void* C;
  int M, N, K, ldc, mode;
  int up_row0;          // kGsGated: first up row of W
  int early;            // no kernel writes W: it is fetched before the wait for the kernel in front
  int splits;           // blocks of a cluster
  int four;             // C's rows take four values at a time (16 bytes of float32, 8 of bfloat16); else one by one
  GateAct gate;
  int* status;
};

template <int NT>
struct GsShape {
  static constexpr int kStage = kGsW + NT * kGsK * 2;
  static constexpr int kStages = 98304 / kStage;
  static constexpr int kSums = NT * kGsFeatures * 4;
  static constexpr int kBody = kStages * kStage > kSums ? kStages * kStage : kSums;
  static constexpr int kSmem = kBody + (2 * kStages + 1) * 8 + 16 + 1024;
  static constexpr int kColumns = NT < 32 ? 32 : NT;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}

template <int NT>
__global__ void __launch_bounds__(kGsThreads, 2)
gemm_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, GsArgs a) {
  using S = GsShape<NT>;
  constexpr int R = S::kStages;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBody);      // full[R], empty[R], done
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * R + 1);
  float* sums = reinterpret_cast<float*>(smem);                       // [token][feature], once every slice has been multiplied
  const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * R, done = empty0 + 8 * R, ring = smem_addr(smem);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool gated_mode = a.mode == kGsGated;
  const int cols = gated_mode ? kGsFeatures / 2 : kGsFeatures;        // of C in a tile
  const int rank = (int)blockIdx.x % a.splits, n0 = (int)blockIdx.x / a.splits * cols;
  const int slices_all = (a.K + kGsK - 1) / kGsK;
  const int s_first = (int)((long long)slices_all * rank / a.splits), slices = (int)((long long)slices_all * (rank + 1) / a.splits) - s_first;

  if (tid == 0) {
    for (int s = 0; s < R; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(S::kColumns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  pdl_launch_dependents();

  // The outputs of this block: its tokens are rank, rank + splits, ...; a group of 32 lanes (16 where gate and up values join) a token,
  // four features a lane; warps 2 to 5. The old values of the first items are on their way while the products run.
  const int per = gated_mode ? 16 : 32, items = (a.M - rank + a.splits - 1) / a.splits * per, first = tid - 64;
  constexpr int kAhead = 4;
  float4 old[kAhead];
  auto place = [&](int i, int& t, int& f, bool& four) {
    t = rank + i / per * a.splits;
    f = i % per * 4;
    four = a.four && n0 + f + 4 <= a.N;
    return i < items && n0 + f < a.N;
  };
  auto old_values = [&](int i) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    int t, f;
    bool four;
    if (a.mode != kGsAddF32 || !place(i, t, f, four)) return v;
    const float* c = reinterpret_cast<const float*>(a.C) + (size_t)t * a.ldc + n0 + f;
    if (four) return *reinterpret_cast<const float4*>(c);
    v.x = c[0];
    if (n0 + f + 1 < a.N) v.y = c[1];
    if (n0 + f + 2 < a.N) v.z = c[2];
    if (n0 + f + 3 < a.N) v.w = c[3];
    return v;
  };

  if (warp == 0) {
    if (elect_one()) {
      auto load_w = [&](int i) {
        const uint32_t bar = full0 + 8 * (i % R), dst = ring + (i % R) * S::kStage;
        const int k0 = (s_first + i) * kGsK;
        mbar_expect_tx(bar, S::kStage);
        tma_load_2d(dst, &map_w, k0, n0, bar);
        tma_load_2d(dst + kGsW / 2, &map_w, k0, gated_mode ? a.up_row0 + n0 : n0 + 64, bar);
      };
      auto load_x = [&](int i) { tma_load_2d(ring + (i % R) * S::kStage + kGsW, &map_x, (s_first + i) * kGsK, 0, full0 + 8 * (i % R)); };
      const int ahead = min(R, slices);
      if (!a.early) pdl_wait();
      for (int i = 0; i < ahead; ++i) load_w(i);
      if (a.early) pdl_wait();
      for (int i = 0; i < ahead; ++i) load_x(i);
      for (int i = ahead; i < slices; ++i) {
        if (!mbar_wait(empty0 + 8 * (i % R), ((i / R) - 1) & 1)) { atomicExch(a.status, 71); break; }
        load_w(i);
        load_x(i);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = instr_desc(kGsFeatures, NT);
      bool ok = true;
      for (int i = 0; i < slices; ++i) {
        if (!mbar_wait(full0 + 8 * (i % R), (i / R) & 1)) { atomicExch(a.status, 72); ok = false; break; }
        tc_fence_after();
        const uint64_t dw = smem_desc(ring + (i % R) * S::kStage), dx = smem_desc(ring + (i % R) * S::kStage + kGsW);
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) mma_bf16_ss(tmem, dw + (uint64_t)(k4 * 2), dx + (uint64_t)(k4 * 2), idesc, (i > 0 || k4 > 0) ? 1u : 0u);
        mma_commit(empty0 + 8 * (i % R));
      }
      if (ok) mma_commit(done);
    }
  } else {
    pdl_wait();        // C may be what kernels in front still use
#pragma unroll
    for (int j = 0; j < kAhead; ++j) old[j] = old_values(first + 128 * j);
    // the sums of lanes 32 * (warp % 4) .. + 31 into shared memory (all slices have been read by then)
    const int quad = warp & 3;
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0));
    if (!ok) {
      if (lane == 0) atomicExch(a.status, 73);
    } else {
      tc_fence_after();
      const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16);
      float* dst = sums + quad * 32 + lane;
#pragma unroll
      for (int c = 0; c < NT; c += 16) {
        if (c >= a.M) break;
        uint32_t r[16];
        tmem_ld16(at + c, r);
#pragma unroll
        for (int j = 0; j < 16; ++j) dst[(c + j) * kGsFeatures] = __uint_as_float(r[j]);
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  if (a.splits > 1) cluster_sync_all();
  else __syncthreads();
  auto finish = [&](int i, float4 before) {
    int t, f;
    bool four;
    if (!place(i, t, f, four)) return;
    const int n = n0 + f;
    const uint32_t at = smem_addr(sums) + (uint32_t)(t * kGsFeatures + f) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f), u = v;
    if (a.splits == 1) {
      v = *reinterpret_cast<const float4*>(sums + t * kGsFeatures + f);
      if (gated_mode) u = *reinterpret_cast<const float4*>(sums + t * kGsFeatures + 64 + f);
    } else {
      float4 p[8], q[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r >= a.splits) break;
        const uint32_t peer = cluster_map(at, (uint32_t)r);
        p[r] = ld_cluster_f4(peer);
        if (gated_mode) q[r] = ld_cluster_f4(peer + 256);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (r >= a.splits) break;
        v.x += p[r].x; v.y += p[r].y; v.z += p[r].z; v.w += p[r].w;
        if (gated_mode) { u.x += q[r].x; u.y += q[r].y; u.z += q[r].z; u.w += q[r].w; }
      }
    }
    if (gated_mode) {
      v.x = gated(a.gate, v.x, u.x);
      v.y = gated(a.gate, v.y, u.y);
      v.z = gated(a.gate, v.z, u.z);
      v.w = gated(a.gate, v.w, u.w);
    }
    if (a.mode == kGsF32 || a.mode == kGsAddF32) {
      v.x += before.x; v.y += before.y; v.z += before.z; v.w += before.w;
      float* c = reinterpret_cast<float*>(a.C) + (size_t)t * a.ldc + n;
      if (four) {
        *reinterpret_cast<float4*>(c) = v;
      } else {
        c[0] = v.x;
        if (n + 1 < a.N) c[1] = v.y;
        if (n + 2 < a.N) c[2] = v.z;
        if (n + 3 < a.N) c[3] = v.w;
      }
    } else {
      __nv_bfloat16* c = reinterpret_cast<__nv_bfloat16*>(a.C) + (size_t)t * a.ldc + n;
      const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
      if (four) {
        uint2 o;
        o.x = *reinterpret_cast<const uint32_t*>(&lo);
        o.y = *reinterpret_cast<const uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(c) = o;
      } else {
        c[0] = lo.x;
        if (n + 1 < a.N) c[1] = lo.y;
        if (n + 2 < a.N) c[2] = hi.x;
        if (n + 3 < a.N) c[3] = hi.y;
      }
    }
  };
  if (warp >= 2) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) finish(first + 128 * j, old[j]);
    for (int i = first + 128 * kAhead; i < items; i += 128) finish(i, old_values(i));
  }
  __syncwarp();
  if (a.splits > 1) cluster_sync_all();      // no block leaves while another still reads its sums
  if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::kColumns) : "memory");
}

// A [rows, K] bfloat16 row-major matrix seen through boxes of box_rows x 64 elements, 128-byte swizzle.
static int gs_map(CUtensorMap* map, const void* base, long long rows, long long K, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(2, "gemm_stream: the driver does not offer cuTensorMapEncodeTiled");
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K * 2};
  cuuint32_t box[2] = {(cuuint32_t)kGsK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(2, "gemm_stream: cuTensorMapEncodeTiled failed with code %d", (int)r);
  return 0;
}

template <int NT>
static int launch_gs(const CUtensorMap& mw, const CUtensorMap& mx, const GsArgs& a, int tiles, cudaStream_t s) {
  using S = GsShape<NT>;
  static std::atomic<unsigned long long> allowed;
  const cudaError_t e = allow_shared((const void*)gemm_stream_kernel<NT>, S::kSmem, allowed);
  if (e != cudaSuccess) return fail(2, "gemm_stream: cannot reserve %d bytes of shared memory: %s", S::kSmem, cudaGetErrorString(e));
  const bool early = a.early ? pdl_mode() != 0 : pdl_mode() == 1;
  launch_clusters(early, (unsigned)a.splits, gemm_stream_kernel<NT>, dim3((unsigned)(tiles * a.splits)), dim3(kGsThreads), (size_t)S::kSmem, s, mw, mx, a);
  return check_launch("gemm_stream");
}

// Blocks that share a tile's K: about 190 blocks in all (measured best of 1 to 8 with 8 to 192 tiles: 32 tiles 6, 48 tiles 4, 96 tiles 2, from
// 152 tiles on 1; 64 rows x 4,096 x 4,096 in 1 / 4 / 6 blocks 31.6 / 20.4 / 18.3 us, 12,288 gated x 4,096 in 1 / 2 / 4 53.1 / 57.3 / 61.3).
static int gs_splits(int tiles, int K) {
  const int slices = (K + kGsK - 1) / kGsK, most = slices < 8 ? slices : 8, want = (190 + tiles / 2) / tiles;
  return want < 1 ? 1 : want > most ? most : want;
}

}  // namespace slb

using namespace slb;

// Whether the kernel takes the problem (rows of 16-byte multiples, whole gate and up tiles need nothing).
extern "C" int slb_gemm_stream_supported(int M, int N, int K) { return M >= 1 && M <= 64 && N >= 1 && K >= 64 && K % 8 == 0; }

// mode: 0 store bfloat16, 1 store float32, 2 add into float32, 3 gated activation (W: N gate rows, then N up rows). splits: 0 for the
// rule's choice, else blocks that share K (1 to 8, at most the 64-wide slices of K). static_weight: no kernel writes W. `status`: a device
// int that the caller zeroed; a bounded wait that gave up writes its code there.
extern "C" int slb_gemm_stream(const void* X, const void* W, void* C, int M, int N, int K, int ldc, int mode, int kind, float limit, float alpha,
                               int static_weight, int splits, int* status, void* stream) {
  SLB_REQUIRE(slb_gemm_stream_supported(M, N, K), "gemm_stream: M=%d N=%d K=%d is not taken (1 to 64 rows, K a multiple of 8 and at least 64)", M, N, K);
  SLB_REQUIRE(mode >= 0 && mode <= 3 && ldc >= N && status != nullptr && kind >= kGateSilu && kind <= kGateLast, "gemm_stream: mode=%d ldc=%d N=%d kind=%d", mode, ldc, N, kind);
  SLB_REQUIRE(((uintptr_t)X % 16 == 0) && ((uintptr_t)W % 16 == 0), "gemm_stream: X and W must be 16-byte aligned");
  SLB_REQUIRE(splits >= 0 && splits <= 8 && splits <= (K + kGsK - 1) / kGsK, "gemm_stream: %d blocks for K=%d", splits, K);
  const bool gated_mode = mode == kGsGated;
  const int cols = gated_mode ? kGsFeatures / 2 : kGsFeatures, tiles = (N + cols - 1) / cols;
  const int nt = M <= 16 ? 16 : M <= 32 ? 32 : 64;
  CUtensorMap mw, mx;
  int rc = gs_map(&mw, W, gated_mode ? 2ll * N : N, K, 64);
  if (rc) return rc;
  rc = gs_map(&mx, X, M, K, nt);
  if (rc) return rc;
  const int width = mode == kGsF32 || mode == kGsAddF32 ? 4 : 2;
  const GsArgs a{C, M, N, K, ldc, mode, N, static_weight, splits ? splits : gs_splits(tiles, K), ldc % 4 == 0 && (uintptr_t)C % (4 * width) == 0,
                 GateAct{kind, limit, alpha}, status};
  cudaStream_t s = (cudaStream_t)stream;
  switch (nt) {
    case 16: return launch_gs<16>(mw, mx, a, tiles, s);
    case 32: return launch_gs<32>(mw, mx, a, tiles, s);
    default: return launch_gs<64>(mw, mx, a, tiles, s);
  }
}
