// One warp's share of the attention of one query token: groups of 16 keys of one KV head against all query heads of it,
// online softmax in registers.  Used by the split-K decode kernel (attn_decode.cu) and the token kernel (token.cu).
//
//   * Every K and V byte goes from global memory straight into the registers of the thread that needs it as an
//     mma.sync operand — sixteen 16-byte loads per thread and group, all issued before the first is used, each warp
//     instruction covering whole 64- or 128-byte runs of a row.  The tensor-core fragments do not care in which
//     order the head dimension is summed, nor which output column stands for which dimension, so the loads can be
//     laid out for the memory system and the fragments follow (the permutation is the same for Q and K, and undone
//     when O is written);
//   * S = Q K^T as m16n8k16 products with the group's query heads as rows (rows past the group size are zero), the
//     softmax of the group in registers, then O^T += V^T P^T with the head dimension as rows and the query heads as
//     columns, whose A operand pairs the same dimension of two consecutive keys with one byte permute each.
#pragma once
#include "mma_common.cuh"

namespace infllm {

constexpr int kMaxGroup = 8;     // query heads per KV head
constexpr int kDecodeRow = 132;  // floats of a head's outputs in shared memory, padded
// the dimension that lies at a place of such a row
__device__ __forceinline__ int decode_dim(int place) { return (place & 64) | ((place & 7) << 3) | ((place >> 3) & 7); }

__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 r;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "l"(p));
  return r;
}

template <typename T>
struct DecodeWarp {
  uint4 qf[4];     // Q of this thread's row g: elements j*32 + t*8 .. +7 for j = 0..3 (zero for rows past the group)
  float ot[8][4];  // O^T tile i: [0],[1] = dim g*8+i of heads 2t, 2t+1; [2],[3] = dim 64+g*8+i
  float m, l;      // running maximum of head g; this thread's share of its row sum

  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i) ot[i][0] = ot[i][1] = ot[i][2] = ot[i][3] = 0.f;
    m = -INFINITY;
    l = 0.f;
  }

  // Keys j0 .. j0 + nk - 1 (nk <= 16) of rows row_bytes apart.  deposit != null: what was read also goes to that K block
  // (V block v_off behind it).  logits != null: the scaled log2-domain logits of this thread's head, from key j0 on.
  __device__ __forceinline__ void group(const char* kbase, const char* vbase, int64_t row_bytes, int j0, int nk, bool qrow,
                                        float scale_log2, char* deposit, int64_t v_off, float* logits) {
    using namespace mma;
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // ---- every load of the group.  K: keys j0 + nt*8 + g (this thread's B-fragment column), 64 bytes of the row in
    //      four pieces j*64 + t*16; V: keys j0 + {2t, 2t+1, 2t+8, 2t+9}, 32 bytes in two pieces p*128 + g*16.
    //      Rows past the end of the segment are read from its last row and masked below.
    uint4 kr[2][4], vr[4][2];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      const int r = nt * 8 + g;
      const char* rp = kbase + (int64_t)(j0 + (r < nk ? r : nk - 1)) * row_bytes + t * 16;
#pragma unroll
      for (int j = 0; j < 4; ++j) kr[nt][j] = ld_stream16(rp + j * 64);
    }
#pragma unroll
    for (int ki = 0; ki < 4; ++ki) {
      const int r = 2 * t + (ki & 1) + (ki >> 1) * 8;
      const char* rp = vbase + (int64_t)(j0 + (r < nk ? r : nk - 1)) * row_bytes + g * 16;
      vr[ki][0] = ld_stream16(rp);
      vr[ki][1] = ld_stream16(rp + 128);
    }
    if (deposit) {  // what was just read, to the same place of the landing slot (K block, then V block)
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const int r = nt * 8 + g;
        if (r < nk) {
          char* wp = deposit + (int64_t)(j0 + r) * row_bytes + t * 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(wp + j * 64) = kr[nt][j];
        }
      }
#pragma unroll
      for (int ki = 0; ki < 4; ++ki) {
        const int r = 2 * t + (ki & 1) + (ki >> 1) * 8;
        if (r < nk) {
          char* wp = deposit + v_off + (int64_t)(j0 + r) * row_bytes + g * 16;
          *reinterpret_cast<uint4*>(wp) = vr[ki][0];
          *reinterpret_cast<uint4*>(wp + 128) = vr[ki][1];
        }
      }
    }
    // ---- S = Q K^T: rows = query heads, columns = the 16 keys (two n-tiles), 8 k-steps of 16 elements
    float sacc[2][4];
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
      sacc[nt][0] = sacc[nt][1] = sacc[nt][2] = sacc[nt][3] = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t a0[4] = {qf[j].x, 0u, qf[j].y, 0u};
        mma16816<T>(sacc[nt], a0, kr[nt][j].x, kr[nt][j].y);
        const uint32_t a1[4] = {qf[j].z, 0u, qf[j].w, 0u};
        mma16816<T>(sacc[nt], a1, kr[nt][j].z, kr[nt][j].w);
      }
    }
    // ---- softmax of the group against the running maximum: this thread holds keys nt*8 + 2t + e of head g
    float sv[4];
    float mx = -INFINITY;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int key = nt * 8 + 2 * t + e;
        const float v = (qrow && key < nk) ? sacc[nt][e] * scale_log2 : -INFINITY;
        sv[nt * 2 + e] = v;
        mx = fmaxf(mx, v);
        if (logits && qrow && key < nk) logits[j0 + key] = v;
      }
    }
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
    const float mn = fmaxf(m, mx);
    const float ms = mn == -INFINITY ? 0.f : mn;
    const float al = exp2f(m - ms);  // 0 for the first group of a row
    m = mn;
    float p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = exp2f(sv[i] - ms);
    l = l * al + (p[0] + p[1]) + (p[2] + p[3]);
    // the O^T columns of this thread are heads 2t and 2t+1: their factors come from the lanes that own those rows
    const float a0 = __shfl_sync(0xffffffffu, al, (2 * t) * 4), a1 = __shfl_sync(0xffffffffu, al, (2 * t + 1) * 4);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      ot[i][0] *= a0;
      ot[i][1] *= a1;
      ot[i][2] *= a0;
      ot[i][3] *= a1;
    }
    // ---- O^T += V^T P^T: B = P^T (this thread: head g, keys 2t, 2t+1 | 2t+8, 2t+9), A = V^T built by byte permutes
    const uint32_t b0 = pack2<T>(p[0], p[1]), b1 = pack2<T>(p[2], p[3]);
    const uint32_t* v00 = reinterpret_cast<const uint32_t*>(&vr[0][0]);
    const uint32_t* v10 = reinterpret_cast<const uint32_t*>(&vr[1][0]);
    const uint32_t* v20 = reinterpret_cast<const uint32_t*>(&vr[2][0]);
    const uint32_t* v30 = reinterpret_cast<const uint32_t*>(&vr[3][0]);
    const uint32_t* v01 = reinterpret_cast<const uint32_t*>(&vr[0][1]);
    const uint32_t* v11 = reinterpret_cast<const uint32_t*>(&vr[1][1]);
    const uint32_t* v21 = reinterpret_cast<const uint32_t*>(&vr[2][1]);
    const uint32_t* v31 = reinterpret_cast<const uint32_t*>(&vr[3][1]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = i >> 1;
      const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;  // the high or the low 16 bits of both words
      uint32_t a[4];
      a[0] = __byte_perm(v00[r], v10[r], sel);  // dim g*8+i of keys 2t, 2t+1
      a[1] = __byte_perm(v01[r], v11[r], sel);  // dim 64+g*8+i
      a[2] = __byte_perm(v20[r], v30[r], sel);  // keys 2t+8, 2t+9
      a[3] = __byte_perm(v21[r], v31[r], sel);
      mma16816<T>(ot[i], a, b0, b1);
    }
  }

  // The warp's result into its slots of shared memory: sm_m[head], sm_l[head], and the outputs at sm_o[head][place].
  // Dimension half*64 + g*8 + i lies at place half*64 + i*8 + g, and a head's row is kDecodeRow floats long: the 32 lanes of
  // a store then hit 32 banks (in plain order eight lanes shared each of four).
  __device__ __forceinline__ void store(float (*sm_o)[kDecodeRow], float* sm_m, float* sm_l, int n_heads_of_group) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (g < n_heads_of_group && t == 0) {
      sm_m[g] = m;
      sm_l[g] = l;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int head = 2 * t + e;
        if (head < n_heads_of_group) {
          sm_o[head][i * 8 + g] = ot[i][e];
          sm_o[head][64 + i * 8 + g] = ot[i][2 + e];
        }
      }
    }
  }
};

}  // namespace infllm
