// Whole prompts of heads whose keys and values have different widths, or whose keys have a rotated part, on the tcgen05 attention, which
// takes keys and values of one width W (64 or 128) in pages: the step's per-head keys, values and queries are laid out in rows of W with
// zeros at their ends (scores and outputs are the same numbers), and the outputs are taken out of such rows, gated, for the output
// product. Pieces of 16 bytes a thread. 2,048 tokens, 16 heads of 64 + 32 key and 64 value channels, us a layer:
// 141 with the attention on mma.sync; 20 + 31 (tcgen05 attention) + 5 now. The layout's 40 MB would take 6 us and the outputs' 13 MB 2 us at the rate of
// a copy: what bounds the layout is each piece's index arithmetic (divisions by run-time sizes) and the rotated pieces' single loads.
#include "common.cuh"

namespace slb {

struct HeadPagesArgs {
  const __nv_bfloat16* q;        // [T, H, dn + P] rotated part not yet turned
  const __nv_bfloat16* kv;       // [T, H * dn + H * dv]: every head's unrotated key values, then every head's values
  const __nv_bfloat16* k_rot;    // [T, P] the shared key part, turned
  __nv_bfloat16* q_out;          // [T, H, W]
  __nv_bfloat16* k_pages;        // [pages, H, 64, W]; sequence i's pages begin at seq_start[i] / 64 + i
  __nv_bfloat16* v_pages;
  const float* cos_t;            // [positions, rot / 2]
  const float* sin_t;
  const int* tok_seq;
  const int* tok_pos;
  const int* seq_start;
  int T, H, dn, P, dv, rot, W;
};

// A block a token; a thread one 16-byte piece of a head's query, key or value row after the other.
__global__ void __launch_bounds__(256) head_pages_kernel(HeadPagesArgs a) {
  pdl_enter();
  const int t = blockIdx.x, seq = a.tok_seq[t], pos = a.tok_pos[t];
  const int page = a.seq_start[seq] / kPageTokens + seq + pos / kPageTokens, row = pos % kPageTokens;
  const int pieces = a.W / 8, per_head = 3 * pieces, dk = a.dn + a.P, half = a.rot / 2;
  const __nv_bfloat16* kv = a.kv + (size_t)t * a.H * (a.dn + a.dv);
  for (int i = threadIdx.x; i < a.H * per_head; i += blockDim.x) {
    const int h = i / per_head, rest = i - h * per_head, what = rest / pieces, c = (rest - what * pieces) * 8;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (what == 0) {
      const __nv_bfloat16* q = a.q + ((size_t)t * a.H + h) * dk;
      if (c < a.dn || (c < dk && c - a.dn >= a.rot)) {
        v = *reinterpret_cast<const uint4*>(q + c);
      } else if (c < dk) {
        __nv_bfloat16 o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int j = c - a.dn + e;
          float x = __bfloat162float(q[a.dn + j]);
          if (j < a.rot) {
            const int f = j < half ? j : j - half;
            const float cs = a.cos_t[(size_t)pos * half + f], sn = a.sin_t[(size_t)pos * half + f];
            x = j < half ? x * cs - __bfloat162float(q[a.dn + j + half]) * sn : x * cs + __bfloat162float(q[a.dn + j - half]) * sn;
          }
          o[e] = __float2bfloat16_rn(x);
        }
        v = *reinterpret_cast<const uint4*>(o);
      }
      *reinterpret_cast<uint4*>(a.q_out + ((size_t)t * a.H + h) * a.W + c) = v;
    } else {
      if (what == 1) {
        if (c < a.dn) v = *reinterpret_cast<const uint4*>(kv + h * a.dn + c);
        else if (c < dk) v = *reinterpret_cast<const uint4*>(a.k_rot + (size_t)t * a.P + c - a.dn);
      } else if (c < a.dv) {
        v = *reinterpret_cast<const uint4*>(kv + a.H * a.dn + h * a.dv + c);
      }
      *reinterpret_cast<uint4*>((what == 1 ? a.k_pages : a.v_pages) + (((size_t)page * a.H + h) * kPageTokens + row) * a.W + c) = v;
    }
  }
}

// y[t, h, :] = rows[t, h, 0 : dv] * sigmoid(gate), the gate a value a channel (gate), a value a head (head_gate), or none.
__global__ void __launch_bounds__(256)
head_rows_kernel(const __nv_bfloat16* rows, const __nv_bfloat16* gate, const float* head_gate, long long head_gate_stride, __nv_bfloat16* y,
                 long long total8, int H, int dv8, int w8) {
  pdl_enter();
  const long long step = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total8; i += step) {
    const long long th = i / dv8, t = th / H;
    const int c = (int)(i - th * dv8), h = (int)(th - t * H);
    Bf16x8 v = reinterpret_cast<const Bf16x8*>(rows)[th * w8 + c];
    if (gate != nullptr || head_gate != nullptr) {
      float f[8], z[8];
      unpack8(v, f);
      if (gate != nullptr) {
        unpack8(reinterpret_cast<const Bf16x8*>(gate)[i], z);
      } else {
        const float one = head_gate[t * head_gate_stride + h];
#pragma unroll
        for (int e = 0; e < 8; ++e) z[e] = one;
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] *= 1.0f / (1.0f + expf(-z[e]));
#pragma unroll
      for (int e = 0; e < 4; ++e) v.v[e] = __floats2bfloat162_rn(f[2 * e], f[2 * e + 1]);
    }
    reinterpret_cast<Bf16x8*>(y)[i] = v;
  }
}

}  // namespace slb

using namespace slb;

// Rows of `width` (64 or 128) from q [T, H, dn + P], kv [T, H (dn + dv)] and k_rot [T, P] of a step whose sequences all start at position 0: queries
// turned into q_out, keys and values into pages (the value rows behind a sequence's last token are not written).
extern "C" int slb_head_pages(const void* q, const void* kv, const void* k_rot, void* q_out, void* k_pages, void* v_pages, const float* cos_t,
                              const float* sin_t, const int* tok_seq, const int* tok_pos, const int* seq_start, int T, int H, int dn, int P,
                              int dv, int rot, int width, void* stream) {
  SLB_REQUIRE((width == 64 || width == 128) && dn > 0 && dn % 8 == 0 && P >= 0 && P % 8 == 0 && dv > 0 && dv % 8 == 0 && dn + P <= width && dv <= width,
              "head_pages: heads of %d + %d and %d channels in rows of %d", dn, P, dv, width);
  SLB_REQUIRE(T >= 0 && H > 0 && rot >= 0 && rot <= P && rot % 2 == 0 && (rot == 0 || (cos_t && sin_t)), "head_pages: tokens=%d heads=%d rot=%d", T, H, rot);
  SLB_REQUIRE((uintptr_t)q % 16 == 0 && (uintptr_t)kv % 16 == 0 && (uintptr_t)k_rot % 16 == 0 && (uintptr_t)q_out % 16 == 0 &&
              (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0, "head_pages: 16-byte alignment");
  if (T == 0) return 0;
  const HeadPagesArgs a{(const __nv_bfloat16*)q, (const __nv_bfloat16*)kv, (const __nv_bfloat16*)k_rot, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pages,
                        (__nv_bfloat16*)v_pages, cos_t, sin_t, tok_seq, tok_pos, seq_start, T, H, dn, P, dv, rot, width};
  launch(head_pages_kernel, dim3(T), dim3(256), 0, (cudaStream_t)stream, a);
  return check_launch("head_pages");
}

// y [T, H * dv] from rows [T, H, width]; gate: bfloat16 [T, H * dv] or null; head_gate: float32, a value per (token, head), rows
// head_gate_stride apart, or null.
extern "C" int slb_head_rows(const void* rows, const void* gate, const float* head_gate, long long head_gate_stride, void* y, int T, int H,
                             int dv, int width, void* stream) {
  SLB_REQUIRE(T >= 0 && H > 0 && dv > 0 && dv % 8 == 0 && width % 8 == 0 && dv <= width && (gate == nullptr || head_gate == nullptr),
              "head_rows: tokens=%d heads=%d width=%d of %d", T, H, dv, width);
  SLB_REQUIRE((uintptr_t)rows % 16 == 0 && (uintptr_t)gate % 16 == 0 && (uintptr_t)y % 16 == 0, "head_rows: 16-byte alignment");
  if (T == 0) return 0;
  const long long total8 = (long long)T * H * (dv / 8);
  long long blocks = (total8 + 255) / 256;
  if (blocks > (long long)sm_count() * 16) blocks = (long long)sm_count() * 16;
  launch(head_rows_kernel, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, (const __nv_bfloat16*)rows, (const __nv_bfloat16*)gate,
         head_gate, head_gate_stride, (__nv_bfloat16*)y, total8, H, dv / 8, width / 8);
  return check_launch("head_rows");
}
