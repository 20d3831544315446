// One decode token of a context memory as ONE launch: ingestion, unit scoring, top-k, attention over window, sink and the
// retrieved units, and the merge with the accumulation of the local scores.
//
// As separate kernels a token is five launches (ingest, scoring + top-k, table update, split-K attention, merge) whose
// boundaries cost more than their work at ordinary context lengths: 160 units are 28 MB, 4.4 us of HBM, in 27 us.  Here one
// CTA per SM stays for the whole token:
//   rows       the query mean is rotated into shared memory by every CTA for itself; warps stream the representative keys
//              (one row per warp and turn, eight 16-byte loads per lane in flight, rows interleaved over the SMs)
//   ranking    one CTA has nothing else to do: it collects the scores as they appear and ranks them
//   window     meanwhile the others take their share of the keys that need no retrieval (window, sink, overflow)
//   units      then their share of the retrieved units, each read wherever the table of unit addresses says (a unit
//              that lives in the store is also written to its landing slot)
//   merge      the CTAs of a KV head exchange their partial results, each merges a share of the outputs and adds its own
//              window columns to the accumulated scores
// CTA (run r, KV head h) works for one KV head throughout, so that a warp's running softmax lives in registers across the
// phases.  Scores, ids and partials travel between CTAs as 8-byte words {value, token number} that carry their own
// arrival: the reader polls the words it needs.  (With a ticket counter, the last CTA ranking, and counters that the CTAs
// meet at, each exchange is a fence, an atomic, a poll and a load one after another.)  The CTAs wait for one another, hence
// a cooperative launch (all of them are resident), and every wait is bounded: one that runs out leaves the error record
// (device and pinned host copy), and the outputs that it was for are not written.
//
// Several contexts' tokens share a launch: the y index of a CTA is its context, whose runs are what its share of the SMs
// gives.  More rounds per warp, but the latencies of the chain are paid once: four contexts of 28/4 heads take 27.9 us
// side by side and 18.7 us each one after another.
//
// Bound: HBM (representative keys + K/V); at small sizes the chain prologue - rows - ranking - units - merge.  160 units of
// 32/8 heads: 14.4 us inside the kernel (prologue 1.9, rows 1.6, window 2 beside the ranking, ids at 7.1, units at 9.5,
// partials at 10.3, log-sum-exps at 12.5) where the five launches took 27; 8192 units: 24 us, of which 10 stream
// 64 MiB of representative keys at 6.4 TB/s.
#include <algorithm>

#include "attn_common.cuh"
#include "decode_warp.cuh"
#include "token.cuh"

namespace infllm {

constexpr int kTokWarps = 12;  // 168 registers a thread: what the attention of a warp takes
constexpr int kTokThreads = kTokWarps * 32;
constexpr int kTokMaxRuns = 160;
constexpr int kTokMaxK = 64;
constexpr int kTokMaxUnits = 16384;
constexpr int kTokScan = 22;    // scores a ranking thread keeps in registers: 8448 of them in one round

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_word_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, uint32_t value, uint32_t seq) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(((unsigned long long)seq << 32) | value) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {  // 16-byte multiples
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t order_bits(float f) {  // larger float <-> larger word; NaN ranks with -inf
  if (!(f == f)) f = -INFINITY;
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __noinline__ void token_gave_up(int32_t* err, int32_t* err_host, int where) {
  if (atomicCAS(&err[0], 0, kTokErrTimeout) == 0) {
    err[1] = where;
    err[2] = blockIdx.x;
    err[3] = 0;
    volatile int32_t* h = err_host;
    h[1] = where, h[2] = blockIdx.x, h[3] = 0;
    __threadfence_system();
    h[0] = kTokErrTimeout;
  }
}
// a word once it carries this token's number (v: what was read of it already); false: the bound ran out
__device__ __forceinline__ bool poll_word(const unsigned long long* p, unsigned long long& v, const TokenParams& P, int where) {
  for (uint32_t i = 0; (uint32_t)(v >> 32) != P.seq; v = ld_word(p)) {
    if (++i > P.spin) {
      token_gave_up(P.err, P.err_host, where);
      return false;
    }
    if (i > 64) __nanosleep(i > 4096 ? 256 : 20);
  }
  return true;
}

// The ranking CTA: the k best of the scores, published in order; ties to the lower id.
__device__ __forceinline__ void token_rank(const TokenParams& P, unsigned long long* cand) {
  constexpr int kGroups = kTokThreads / 4;  // groups of four threads' scores
  __shared__ __align__(16) uint32_t s_gm[kGroups];
  __shared__ uint32_t s_tau;
  __shared__ int s_cnt;
  const int tid = threadIdx.x;
  // the table of unit addresses learns what the host changed since the last token.  The fence here, while there is time, is
  // what lets the ids be published later by plain stores.
  if (tid < P.n_upd) P.ptrs[P.upd_id[tid]] = P.upd_val[tid];
  if (tid == 0) s_tau = 0u, s_cnt = 0;
  __syncthreads();
  __threadfence();
  uint32_t best = 0u, kept[kTokScan];
  bool ok = true;
  // thread t collects the scores t, t + kTokThreads, ...; eleven words on their way at a time
#pragma unroll
  for (int c = 0; c < kTokScan; c += 11) {
    unsigned long long w[11];
#pragma unroll
    for (int u = 0; u < 11; ++u) {
      const int i = (c + u) * kTokThreads + tid;
      w[u] = i < P.n ? ld_word(P.score_words + i) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < 11; ++u) {
      const int i = (c + u) * kTokThreads + tid;
      kept[c + u] = 0u;
      if (i < P.n && ok) {
        ok = poll_word(P.score_words + i, w[u], P, 702);
        kept[c + u] = order_bits(__uint_as_float((uint32_t)w[u]));
        best = max(best, kept[c + u]);
      }
    }
  }
  for (int i = kTokScan * kTokThreads + tid; i < P.n && ok; i += kTokThreads) {
    unsigned long long w = ld_word(P.score_words + i);
    ok = poll_word(P.score_words + i, w, P, 702);
    best = max(best, order_bits(__uint_as_float((uint32_t)w)));
  }
  if (__syncthreads_or(!ok)) return;
  int nc;
  if (P.n <= kTokThreads) {  // one score per thread: all of them are candidates
    nc = P.n;
    if (tid < nc) cand[tid] = ((unsigned long long)kept[0] << 32) | (uint32_t)(~(uint32_t)tid);
    __syncthreads();
  } else {
    best = max(best, __shfl_xor_sync(0xffffffffu, best, 1));
    best = max(best, __shfl_xor_sync(0xffffffffu, best, 2));
    if ((tid & 3) == 0) s_gm[tid >> 2] = best;
    __syncthreads();
    // tau = the k-th largest of the groups' best scores (0 when fewer than k groups hold any: then everything is a
    // candidate): at least k scores reach it
    if (tid < kGroups) {
      const uint32_t x = s_gm[tid];
      int reach = 0;
#pragma unroll 8
      for (int j = 0; j < kGroups; j += 4) {
        const uint4 y = *reinterpret_cast<const uint4*>(s_gm + j);
        reach += (y.x >= x) + (y.y >= x) + (y.z >= x) + (y.w >= x);
      }
      if (x != 0u && reach >= P.k_top) atomicMax(&s_tau, x);
    }
    __syncthreads();
    const unsigned long long tau = (unsigned long long)s_tau << 32;
    auto consider = [&](uint32_t bits, int i) {
      const unsigned long long key = ((unsigned long long)bits << 32) | (uint32_t)(~(uint32_t)i);
      if (key >= tau) {
        cand[atomicAdd(&s_cnt, 1)] = key;  // room for all n: scores may all be equal
      }
    };
#pragma unroll
    for (int c = 0; c < kTokScan; ++c)
      if (c * kTokThreads + tid < P.n) consider(kept[c], c * kTokThreads + tid);
    for (int i = kTokScan * kTokThreads + tid; i < P.n; i += kTokThreads)
      consider(order_bits(__uint_as_float((uint32_t)ld_word(P.score_words + i))), i);
    __syncthreads();
    nc = s_cnt;
  }
  for (int c = tid; c < nc; c += kTokThreads) {
    const unsigned long long mine = cand[c];
    int rank = 0;
#pragma unroll 8
    for (int j = 0; j < nc; ++j) rank += cand[j] > mine;
    if (rank < P.k_top) {
      const uint32_t id = ~(uint32_t)(mine & 0xffffffffu);
      st_word(P.id_words + rank, id, P.seq);
      // the host's copy, which it may read while this kernel is still running
      *(volatile unsigned long long*)(P.ids_host + rank) = ((unsigned long long)P.seq << 32) | id;
    }
  }
}

template <int NB>
struct TokenBatch {
  TokenParams p[NB];
};

template <typename T, int NB>
__global__ void __launch_bounds__(kTokThreads, 1) token_kernel(const __grid_constant__ TokenBatch<NB> B) {
  const TokenParams& P = B.p[NB == 1 ? 0 : blockIdx.y];
  extern __shared__ __align__(16) unsigned char dyn[];
  // [0, width) fp32 query mean, then the warps' attention results; the ranking CTA keeps its candidates here
  float* sq = reinterpret_cast<float*>(dyn);
  float(*sm_o)[kMaxGroup][kDecodeRow] = reinterpret_cast<float(*)[kMaxGroup][kDecodeRow]>(dyn + P.width * 4);
  __shared__ __align__(16) T s_q[2][kMaxGroup][128];  // the KV head's queries: window-relative, one-angle
  __shared__ T s_new[2][128];                         // the new token's rotated key and its value
  __shared__ float sm_m[kTokWarps + 1][kMaxGroup], sm_l[kTokWarps][kMaxGroup], s_lse[kMaxGroup], s_w[kMaxGroup][kTokMaxRuns],
      s_res[kTokWarps + 1][kMaxGroup];

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int cta = blockIdx.x, n_cta = P.n_runs * P.n_kv, hkv = cta % P.n_kv, run = cta / P.n_kv;
  if (cta == n_cta) {
    token_rank(P, reinterpret_cast<unsigned long long*>(dyn));
    return;
  }
  if (cta > n_cta) return;  // (a context of the batch with fewer CTAs than another)
  const int group = P.group;
  const bool qrow = g < group;
  const T* bk = (const T*)P.bk;

  // ---------------------------------------------------------------------------------------------------- rows
  // (the order of a row's sum is that of block_score_topk_kernel: equal scores bit for bit)
  const int stride_rows = n_cta * kTokWarps, pieces = (P.width + 2047) / 2048;
  int row = warp * n_cta + cta, piece = 0;
  uint4 raw[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const int c = (u * 32 + lane) * 8;
    raw[u] = (row < P.n && c < P.width) ? __ldcs(reinterpret_cast<const uint4*>(bk + (int64_t)row * P.width + c)) : make_uint4(0, 0, 0, 0);
  }
  // this CTA's share of the keys that need no retrieval comes into L2 meanwhile: HBM does not wait for the phases before
  const int n_rest = P.rest_begin[3];
  const int lo = (int)((int64_t)run * n_rest / P.n_runs), hi = (int)((int64_t)(run + 1) * n_rest / P.n_runs);
  if (warp == kTokWarps - 1) {
    const int end = std::min(hi, P.rest_begin[1]) * 16;  // the window's part: contiguous rows
    for (int r = lo * 16 + lane * 32; r < end; r += 32 * 32) {
      const int rows = std::min(std::min(32, end - r), P.rest[0].len - r);
      if (rows <= 0) break;
      const int64_t off = ((int64_t)hkv * P.rest[0].hs + (int64_t)r * 128) * 2;
      prefetch_l2((const char*)P.rest[0].k + off, rows * 256);
      prefetch_l2((const char*)P.rest[0].v + off, rows * 256);
    }
  }
  {
    const T* q = (const T*)P.q;
    constexpr int kHeadsAtOnce = kTokThreads / 64;  // thread tid owns the pair (i, i + 64) of every sixth head
    const int i = tid & 63;
    const float cg = P.cos_t[P.pos_glb * 64 + i], sg = P.sin_t[P.pos_glb * 64 + i], cl = P.cos_t[P.pos_loc * 64 + i],
                sl = P.sin_t[P.pos_loc * 64 + i];
    for (int h0 = tid >> 6; h0 < P.n_heads; h0 += 6 * kHeadsAtOnce) {
      T x[6][2];
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const int h = std::min(h0 + e * kHeadsAtOnce, P.n_heads - 1);
        x[e][0] = q[h * P.q_hs + i], x[e][1] = q[h * P.q_hs + i + 64];
      }
#pragma unroll
      for (int e = 0; e < 6; ++e) {
        const int h = h0 + e * kHeadsAtOnce, hg = h - hkv * group;
        if (h >= P.n_heads) break;
        const float x1 = Act<T>::to_f(x[e][0]), x2 = Act<T>::to_f(x[e][1]);
        const T g1 = Act<T>::from_f(__fadd_rn(__fmul_rn(x1, cg), __fmul_rn(-x2, sg)));
        const T g2 = Act<T>::from_f(__fadd_rn(__fmul_rn(x2, cg), __fmul_rn(x1, sg)));
        sq[h * 128 + i] = Act<T>::to_f(g1);
        sq[h * 128 + i + 64] = Act<T>::to_f(g2);
        if (hg >= 0 && hg < group) {
          s_q[1][hg][i] = g1, s_q[1][hg][i + 64] = g2;
          s_q[0][hg][i] = Act<T>::from_f(__fadd_rn(__fmul_rn(x1, cl), __fmul_rn(-x2, sl)));
          s_q[0][hg][i + 64] = Act<T>::from_f(__fadd_rn(__fmul_rn(x2, cl), __fmul_rn(x1, sl)));
        }
      }
    }
    if (run == 0 && tid < 64) {  // the new token's rows of this KV head
      const T r1 = ((const T*)P.k)[hkv * P.k_hs + tid], r2 = ((const T*)P.k)[hkv * P.k_hs + tid + 64];
      const T v1 = ((const T*)P.v)[hkv * P.v_hs + tid], v2 = ((const T*)P.v)[hkv * P.v_hs + tid + 64];
      const float x1 = Act<T>::to_f(r1), x2 = Act<T>::to_f(r2);
      const T k1 = Act<T>::from_f(__fadd_rn(__fmul_rn(x1, cl), __fmul_rn(-x2, sl)));
      const T k2 = Act<T>::from_f(__fadd_rn(__fmul_rn(x2, cl), __fmul_rn(x1, sl)));
      T *kr = (T*)P.k_raw + hkv * P.kv_hs, *ko = (T*)P.k_rot + hkv * P.kv_hs, *vo = (T*)P.v_out + hkv * P.kv_hs;
      kr[tid] = r1, kr[tid + 64] = r2;
      ko[tid] = k1, ko[tid + 64] = k2;
      vo[tid] = v1, vo[tid + 64] = v2;
      s_new[0][tid] = k1, s_new[0][tid + 64] = k2;
      s_new[1][tid] = v1, s_new[1][tid + 64] = v2;
    }
  }
  __syncthreads();
  {
    float acc = 0.f;
    while (row < P.n) {
      int nrow = row, npiece = piece + 1;
      if (npiece == pieces) {
        npiece = 0;
        nrow = row + stride_rows;
      }
      const bool more = nrow < P.n;
      const T* np = bk + (int64_t)(more ? nrow : 0) * P.width + npiece * 2048 + lane * 8;
      const int c0 = piece * 2048 + lane * 8, cn0 = npiece * 2048 + lane * 8;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int c = c0 + u * 256;
        const typename Act<T>::T2* v2 = reinterpret_cast<const typename Act<T>::T2*>(&raw[u]);
        const float2 f0 = Act<T>::to_f2(v2[0]), f1 = Act<T>::to_f2(v2[1]), f2 = Act<T>::to_f2(v2[2]),
                     f3 = Act<T>::to_f2(v2[3]);
        // the slot is free: the matching piece of what comes next is requested before this one is summed
        raw[u] = (more && cn0 + u * 256 < P.width) ? __ldcs(reinterpret_cast<const uint4*>(np + u * 256)) : make_uint4(0, 0, 0, 0);
        if (c < P.width) {
          const float4 qa = *reinterpret_cast<const float4*>(sq + c);
          const float4 qb = *reinterpret_cast<const float4*>(sq + c + 4);
          acc = fmaf(f0.x, qa.x, acc);
          acc = fmaf(f0.y, qa.y, acc);
          acc = fmaf(f1.x, qa.z, acc);
          acc = fmaf(f1.y, qa.w, acc);
          acc = fmaf(f2.x, qb.x, acc);
          acc = fmaf(f2.y, qb.y, acc);
          acc = fmaf(f3.x, qb.z, acc);
          acc = fmaf(f3.y, qb.w, acc);
        }
      }
      if (npiece == 0) {  // the row is complete
        acc = warp_sum(acc);
        if (lane == 0) st_word(P.score_words + row, __float_as_uint(acc), P.seq);
        acc = 0.f;
      }
      row = nrow;
      piece = npiece;
    }
  }

  // -------------------------------------------------------------------------------------- window, sink, overflow
  DecodeWarp<T> W;
  W.clear();
  auto load_q = [&](int which) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      W.qf[j] = qrow ? *reinterpret_cast<const uint4*>(&s_q[which][g][j * 32 + t * 8]) : make_uint4(0, 0, 0, 0);
  };
  const int hq = hkv * group + (qrow ? g : 0);
  {
    int cur = -1, sgm = 0;
#pragma unroll 1
    for (int it = lo + warp; it < hi; it += kTokWarps) {
      while (it >= P.rest_begin[sgm + 1]) ++sgm;
      const TokenParams::Seg& S = P.rest[sgm];
      if (cur != (sgm > 0)) {
        cur = sgm > 0;
        load_q(cur);
      }
      const int j0 = (it - P.rest_begin[sgm]) * 16;
      const int64_t off = (int64_t)hkv * S.hs * 2;
      W.group((const char*)S.k + off, (const char*)S.v + off, 256, j0, S.len - j0 < 16 ? S.len - j0 : 16, qrow, P.scale_log2, nullptr, 0,
              sgm == 0 ? P.logits + (int64_t)hq * P.logit_hs : nullptr);
    }
  }

  // --------------------------------------------------------------------------------------------- retrieved units
  // every warp waits for the ids it needs; the warps take their groups in reverse order, so that those with one group more of
  // the window have one less here
  bool ok = true;
  {
    load_q(1);
    const int per = (P.unit_len + 15) / 16, n_unit = P.k_top * per;
    const int ulo = (int)((int64_t)run * n_unit / P.n_runs), uhi = (int)((int64_t)(run + 1) * n_unit / P.n_runs);
    int cur = -1;
    const char *kb = nullptr, *vb = nullptr;
    char* dep = nullptr;
#pragma unroll 1
    for (int it = ulo + kTokWarps - 1 - warp; it < uhi; it += kTokWarps) {
      const int u = it / per, j0 = (it - u * per) * 16;
      if (u != cur) {
        cur = u;
        unsigned long long w = ld_word_acquire(P.id_words + u);
        for (uint32_t i = 0; (uint32_t)(w >> 32) != P.seq; w = ld_word_acquire(P.id_words + u)) {
          if (++i > P.spin) {
            ok = false;
            break;
          }
          if (i > 64) __nanosleep(i > 4096 ? 256 : 20);
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
          if (lane == 0) token_gave_up(P.err, P.err_host, 700);
          break;
        }
        const unsigned long long a = __ldcg(P.ptrs + (uint32_t)w);
        const int64_t off = (int64_t)hkv * P.unit_len * 256;
        kb = reinterpret_cast<const char*>(a & ~1ull) + off;
        vb = kb + P.unit_bytes / 2;
        dep = nullptr;
        if (a & 1ull) {  // the unit's place in the store, not a cache slot
          const unsigned long long la = __ldcg(P.ptrs + P.landing_at + u);
          if (la) dep = reinterpret_cast<char*>(la) + off;
        }
      }
      W.group(kb, vb, 256, j0, P.unit_len - j0 < 16 ? P.unit_len - j0 : 16, qrow, P.scale_log2, dep, P.unit_bytes / 2, nullptr);
    }
  }

  // ----------------------------------------------------------------------------------------- the CTA's partial
  W.store(sm_o[warp], sm_m[warp], sm_l[warp], group);
  if (run == 0 && warp < group) {  // the new token's own key: one more result, with weight 1 and output v
    float d = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) d = fmaf(Act<T>::to_f(s_q[0][warp][lane * 4 + e]), Act<T>::to_f(s_new[0][lane * 4 + e]), d);
    d = warp_sum(d) * P.scale_log2;
    if (lane == 0) sm_m[kTokWarps][warp] = d;
  }
  if (__syncthreads_or(!ok)) return;
  unsigned long long* pw = P.part_words + ((int64_t)run * P.n_heads + hkv * group) * 129;
  // weights of the warps' results, per head
  for (int h = warp; h < group; h += kTokWarps) {
    const float mv = lane < kTokWarps || (lane == kTokWarps && run == 0) ? sm_m[lane][h] : -INFINITY;
    const float mx = warp_max(mv), w = mx == -INFINITY ? 0.f : exp2f(mv - mx);
    const float den = warp_sum(w * (lane < kTokWarps ? sm_l[lane][h] : 1.f)), inv = den > 0.f ? 1.f / den : 0.f;
    if (lane <= kTokWarps) s_res[lane][h] = w * inv;
    if (lane == 0) st_word(pw + h * 129 + 128, __float_as_uint(den > 0.f ? mx + log2f(den) : -INFINITY), P.seq);
  }
  __syncthreads();
  for (int idx = tid; idx < group * 128; idx += kTokThreads) {
    const int h = idx >> 7, d = idx & 127;
    float num = run == 0 ? s_res[kTokWarps][h] * Act<T>::to_f(s_new[1][decode_dim(d)]) : 0.f;
#pragma unroll
    for (int w = 0; w < kTokWarps; ++w) num = fmaf(s_res[w][h], sm_o[w][h][d], num);
    st_word(pw + h * 129 + d, __float_as_uint(num), P.seq);  // in the order of sm_o: undone when the outputs leave
  }
  // --------------------------------------------------------------------------------------------------- merge
  // What the last step adds to is on its way before the partials have arrived: the token's attention row joins the accumulated
  // local scores (context_manager.py:488, 623-625), each CTA adds the window columns whose logits it computed itself.
  const int c_lo = std::min(lo, P.rest_begin[1]) * 16, c_hi = std::min(std::min(hi, P.rest_begin[1]) * 16, P.rest[0].len);
  const int n_cols = c_hi > c_lo ? c_hi - c_lo : 0, n_add = n_cols * group;
  auto column = [&](int i, const float** lg, float** sc, int* h) {
    *h = i / n_cols;
    const int c = c_lo + i - *h * n_cols;
    *lg = P.logits + (int64_t)(hkv * group + *h) * P.logit_hs + c;
    *sc = P.win_score + (int64_t)(hkv * group + *h) * P.score_hs + c;
  };
  float pre_l[4], pre_s[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int i = tid + e * kTokThreads;
    if (i < n_add) {
      const float* lg;
      float* sc;
      int h;
      column(i, &lg, &sc, &h);
      pre_l[e] = __ldcg(lg);
      pre_s[e] = *sc;
    }
  }
  // this CTA's share of the KV head's outputs, eight threads to each
  const int total = group * 128, o_lo = (int)((int64_t)run * total / P.n_runs), o_hi = (int)((int64_t)(run + 1) * total / P.n_runs);
  const int sub = tid & 7;
  auto part_at = [&](int o, int p) {
    return P.part_words + ((int64_t)p * P.n_heads + hkv * group + (o >> 7)) * 129 + (o & 127);
  };
  unsigned long long pre_o[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int o = o_lo + (tid >> 3), p = sub + 8 * e;
    pre_o[e] = o < o_hi && p < P.n_runs ? ld_word(part_at(o, p)) : 0ull;
  }
  for (int h = warp; h < group; h += kTokWarps) {  // every head's log-sum-exp and the runs' weights
    float v[kTokMaxRuns / 32], mx = -INFINITY;
    unsigned long long lw[kTokMaxRuns / 32];
#pragma unroll
    for (int e = 0; e < kTokMaxRuns / 32; ++e)
      if (lane + 32 * e < P.n_runs) lw[e] = ld_word(part_at(h * 128, lane + 32 * e) + 128);
#pragma unroll
    for (int e = 0; e < kTokMaxRuns / 32; ++e) {
      v[e] = -INFINITY;
      if (lane + 32 * e < P.n_runs && ok) {
        ok = poll_word(part_at(h * 128, lane + 32 * e) + 128, lw[e], P, 701);
        v[e] = __uint_as_float((uint32_t)lw[e]);
      }
      mx = fmaxf(mx, v[e]);
    }
    mx = warp_max(mx);
    float den = 0.f;
#pragma unroll
    for (int e = 0; e < kTokMaxRuns / 32; ++e) {
      v[e] = mx == -INFINITY ? 0.f : exp2f(v[e] - mx);
      den += v[e];
    }
    den = warp_sum(den);
    const float inv = den > 0.f ? 1.f / den : 0.f;
#pragma unroll
    for (int e = 0; e < kTokMaxRuns / 32; ++e)
      if (lane + 32 * e < P.n_runs) s_w[h][lane + 32 * e] = v[e] * inv;
    if (lane == 0) s_lse[h] = den > 0.f ? mx + log2f(den) : -INFINITY;
  }
  if (__syncthreads_or(!ok)) return;
  for (int o0 = o_lo; o0 < o_hi; o0 += kTokThreads / 8) {
    const int o = o0 + (tid >> 3), h = o >> 7;
    float num = 0.f;
    if (o < o_hi) {
      for (int p0 = sub; p0 < P.n_runs; p0 += 32) {  // four words on their way at a time
        unsigned long long w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (p0 + 8 * e < P.n_runs) w[e] = o0 == o_lo && p0 == sub ? pre_o[e] : ld_word(part_at(o, p0 + 8 * e));
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (p0 + 8 * e < P.n_runs && ok) {
            ok = poll_word(part_at(o, p0 + 8 * e), w[e], P, 701);
            num = fmaf(s_w[h][p0 + 8 * e], __uint_as_float((uint32_t)w[e]), num);
          }
      }
    }
    num += __shfl_xor_sync(0xffffffffu, num, 1);
    num += __shfl_xor_sync(0xffffffffu, num, 2);
    num += __shfl_xor_sync(0xffffffffu, num, 4);
    if (__all_sync(0xffffffffu, ok) && o < o_hi && sub == 0) ((T*)P.out)[(int64_t)(hkv * group + h) * P.o_hs + decode_dim(o & 127)] = Act<T>::from_f(num);
  }
#pragma unroll 1
  for (int i0 = tid; i0 < n_add; i0 += 4 * kTokThreads) {
    if (i0 != tid) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = i0 + e * kTokThreads;
        if (i < n_add) {
          const float* lg;
          float* sc;
          int h;
          column(i, &lg, &sc, &h);
          pre_l[e] = __ldcg(lg);
          pre_s[e] = *sc;
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + e * kTokThreads;
      if (i < n_add) {
        const float* lg;
        float* sc;
        int h;
        column(i, &lg, &sc, &h);
        *sc = pre_s[e] + exp2f(pre_l[e] - s_lse[h]);
      }
    }
  }
  if (run == 0 && tid < group)  // the new token's column starts here
    P.win_score[(int64_t)(hkv * group + tid) * P.score_hs + P.rest[0].len] = exp2f(sm_m[kTokWarps][tid] - s_lse[tid]);
}

static size_t token_smem(int width, int n) {
  return std::max(sizeof(unsigned long long) * n, (size_t)width * 4 + sizeof(float) * kTokWarps * kMaxGroup * kDecodeRow);
}

// One CTA per SM, one of them for the ranking.  The sizes: what a CTA's shared memory holds (width), the ranking's limits
// (64 of 16384 units, as in block_score_topk_kernel), 8 query heads per KV head.
int token_runs(int n_heads, int n_kv_heads, int head_dim, int64_t n_units, int topk, int block_size, int sms) {
  const int width = n_heads * head_dim;
  if (sms <= n_kv_heads || head_dim != 128 || n_heads / n_kv_heads > kMaxGroup || width > 12288 || n_units > kTokMaxUnits || topk > kTokMaxK || block_size % 8)
    return 0;
  return std::min((sms - 1) / n_kv_heads, kTokMaxRuns);
}

// Two runs per KV head at least: below that the CTAs' rounds of window and units are long enough for a launch of their own.
int token_batch_max(int n_kv_heads, int sms) { return std::max(1, std::min(kTokMaxBatch, sms / (2 * n_kv_heads + 1))); }

template <typename T, int NB>
static int token_launch_batch(const TokenParams* P, int n, cudaLaunchConfig_t& cfg) {
  TokenBatch<NB> B;
  std::copy(P, P + n, B.p);
  auto kern = token_kernel<T, NB>;
  // (the opt-in holds for the current device only: asked for at every launch)
  INFLLM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cfg.dynamicSmemBytes));
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, B);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return fail(INFLLM_E_UNSUPPORTED, "token: a grid of %u x %u CTAs that is not resident at once", cfg.gridDim.x, cfg.gridDim.y);
  }
  INFLLM_CUDA_OK(e);
  return INFLLM_OK;
}

int token_launch(const TokenParams* P, int n, int dtype, cudaStream_t s) {
  size_t smem = 0;
  int ctas = 0;
  for (int i = 0; i < n; ++i) {
    if (P[i].n_upd > kTokMaxUpdates || P[i].n_runs < 1 || P[i].n_runs > kTokMaxRuns) return fail(INFLLM_E_BADARG, "token: bad argument");
    smem = std::max(smem, token_smem(P[i].width, P[i].n));
    ctas = std::max(ctas, P[i].n_runs * P[i].n_kv + 1 + (P[i].too_large ? 4096 : 0));
  }
  if (n < 1 || n > kTokMaxBatch) return fail(INFLLM_E_BADARG, "token: %d contexts", n);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ctas, n);
  cfg.blockDim = dim3(kTokThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  INFLLM_DISPATCH_DTYPE(dtype, T, {
    if (n == 1) {
      INFLLM_TRY((token_launch_batch<T, 1>(P, n, cfg)));
    } else if (n <= 4) {
      INFLLM_TRY((token_launch_batch<T, 4>(P, n, cfg)));
    } else {
      INFLLM_TRY((token_launch_batch<T, kTokMaxBatch>(P, n, cfg)));
    }
  });
  INFLLM_LAUNCH_OK("token_kernel");
  return INFLLM_OK;
}

}  // namespace infllm
