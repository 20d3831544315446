// One call of the sink + window attention types ("infinite-lm", "stream-llm"; inf_llm/attention/infinite_lm.py:6-100,
// stream_llm.py:6-111) over the cache the previous call returned and the call's new tokens.
//
// sink_prepare_kernel goes once over the rows of [cache | new tokens] and over the queries and leaves everything the
// attention reads and the caller keeps: the window's keys rotated to their window positions (they move with every
// call, so they are rotated with every call), its values where they do not lie in one piece already, the sink, both
// rotations of the queries, and the new cache.  It is bound by those bytes: as separate copies, concatenations and
// rotations the same work took 250 us of a 4096-token call and 60 us of a token.  The attention itself is the two
// stages, jointly normalised, as one launch of the tcgen05 kernel, or, for one token, of the split-K kernel.
#include <algorithm>

#include "attn_common.cuh"
#include "attn_tc.cuh"

namespace infllm {

constexpr int kSinkThreads = 256;

struct SinkPrepare {
  const char *q, *k, *v, *past_k, *past_v;  // new tokens, cache of the previous call
  char *cache_k, *cache_v;                  // new cache (may be null), rows contiguous
  char *k_rot, *v_win;                      // (n_kv, rows_w, 128): window rows from `win0` on; v_win may be null
  char *snk_k, *snk_v;                      // (n_kv, n_snk, 128)
  char *q_loc, *q_snk;                      // (n_heads, len_q, 128)
  int64_t q_hs, q_ts, k_hs, k_ts, p_hs, p_ts;  // elements
  const float *cos_t, *sin_t;
  int32_t n_heads, n_kv, len_q, past_len, total, win0, rows_w, n_snk, cache_head, cache_rows, pos_w0, pos_q0, pos_snk,
      rotate_snk;
};

template <typename T>
__device__ __forceinline__ void rotate16(const uint4& lo, const uint4& hi, const float* cs, const float* sn, uint4* olo,
                                         uint4* ohi) {
  const T *a = reinterpret_cast<const T*>(&lo), *b = reinterpret_cast<const T*>(&hi);
  T *oa = reinterpret_cast<T*>(olo), *ob = reinterpret_cast<T*>(ohi);
#pragma unroll
  for (int i = 0; i < 8; ++i) {  // the arithmetic of rope_apply_kernel: fp32 products, one rounding at the end
    const float x1 = Act<T>::to_f(a[i]), x2 = Act<T>::to_f(b[i]), cv = cs[i], sv = sn[i];
    oa[i] = Act<T>::from_f(__fadd_rn(__fmul_rn(x1, cv), __fmul_rn(-x2, sv)));
    ob[i] = Act<T>::from_f(__fadd_rn(__fmul_rn(x2, cv), __fmul_rn(x1, sv)));
  }
}

// eight threads per row: thread c owns the elements c*8..+7 of both halves, the pairs that rotate together
template <typename T>
__global__ void __launch_bounds__(kSinkThreads) sink_prepare_kernel(const __grid_constant__ SinkPrepare P) {
  chain_enter();
  const int64_t idx = (int64_t)blockIdx.x * kSinkThreads + threadIdx.x;
  const int c = (int)(idx & 7);
  const int64_t r = idx >> 3;
  const int64_t n_key = (int64_t)P.n_kv * P.total;
  auto put = [&](char* base, int64_t row, const uint4& lo, const uint4& hi) {
    *reinterpret_cast<uint4*>(base + row * 256 + c * 16) = lo;
    *reinterpret_cast<uint4*>(base + row * 256 + 128 + c * 16) = hi;
  };
  if (r < n_key) {
    const int h = (int)(r / P.total), row = (int)(r - (int64_t)h * P.total);
    const int tail = P.cache_rows - P.cache_head;  // rows of the new cache that come from the end
    const int crow = row < P.cache_head ? row : (row >= P.total - tail ? P.cache_head + row - (P.total - tail) : -1);
    const bool keep = P.cache_k && crow >= 0, snk = row < P.n_snk, win = row >= P.win0;
    if (!keep && !snk && !win) return;
    const bool old = row < P.past_len;
    const int64_t off = (old ? h * P.p_hs + (int64_t)row * P.p_ts : h * P.k_hs + (int64_t)(row - P.past_len) * P.k_ts) * 2 + c * 16;
    const char *ks = (old ? P.past_k : P.k) + off, *vs = (old ? P.past_v : P.v) + off;
    const uint4 k0 = *reinterpret_cast<const uint4*>(ks), k1 = *reinterpret_cast<const uint4*>(ks + 128);
    const uint4 v0 = *reinterpret_cast<const uint4*>(vs), v1 = *reinterpret_cast<const uint4*>(vs + 128);
    if (keep) {
      put(P.cache_k, (int64_t)h * P.cache_rows + crow, k0, k1);
      put(P.cache_v, (int64_t)h * P.cache_rows + crow, v0, v1);
    }
    uint4 a, b;
    if (win) {
      const int j = row - P.win0, pos = (P.pos_w0 + j) * 64 + c * 8;
      rotate16<T>(k0, k1, P.cos_t + pos, P.sin_t + pos, &a, &b);
      put(P.k_rot, (int64_t)h * P.rows_w + j, a, b);
      if (P.v_win) put(P.v_win, (int64_t)h * P.rows_w + j, v0, v1);
    }
    if (snk) {
      if (P.rotate_snk) {
        rotate16<T>(k0, k1, P.cos_t + row * 64 + c * 8, P.sin_t + row * 64 + c * 8, &a, &b);
        put(P.snk_k, (int64_t)h * P.n_snk + row, a, b);
      } else {
        put(P.snk_k, (int64_t)h * P.n_snk + row, k0, k1);
      }
      put(P.snk_v, (int64_t)h * P.n_snk + row, v0, v1);
    }
  } else {
    const int64_t rq = r - n_key;
    if (rq >= (int64_t)P.n_heads * P.len_q) return;
    const int h = (int)(rq / P.len_q), i = (int)(rq - (int64_t)h * P.len_q);
    const char* qs = P.q + (h * P.q_hs + (int64_t)i * P.q_ts) * 2 + c * 16;
    const uint4 q0 = *reinterpret_cast<const uint4*>(qs), q1 = *reinterpret_cast<const uint4*>(qs + 128);
    uint4 a, b;
    const int pos = (P.pos_q0 + i) * 64 + c * 8;
    rotate16<T>(q0, q1, P.cos_t + pos, P.sin_t + pos, &a, &b);
    put(P.q_loc, rq, a, b);
    if (P.n_snk > 0) {
      rotate16<T>(q0, q1, P.cos_t + P.pos_snk * 64 + c * 8, P.sin_t + P.pos_snk * 64 + c * 8, &a, &b);
      put(P.q_snk, rq, a, b);
    }
  }
}

// where everything lies in the caller's scratch, and the sizes of the call
struct SinkPlan {
  int64_t total, lw, w0, n_snk, rows_w, win0;
  bool one, v_from_cache;
  int n_split, max_parts;
  size_t k_rot, v_win, snk_k, snk_v, q_loc, q_snk, part, bytes;
};

static SinkPlan sink_plan(const infllm_sink_window* a) {
  SinkPlan p{};
  p.total = a->past_len + a->len_q;
  p.lw = std::min<int64_t>(p.total, a->len_q + (int64_t)a->n_local);
  p.w0 = p.total - p.lw;
  p.n_snk = a->seen > a->n_local ? std::min<int64_t>(a->n_init, p.total) : 0;
  p.one = a->len_q == 1 && a->n_heads / a->n_kv_heads <= 8;
  // one query sees at most n_local keys: the row that has just left its window is not prepared
  p.rows_w = p.one ? std::min<int64_t>(p.lw, a->n_local) : p.lw;
  p.win0 = p.total - p.rows_w;
  p.v_from_cache = p.one && a->d_cache_v && (a->cache_head == p.total || a->cache_rows - a->cache_head >= p.rows_w);
  p.n_split = p.one ? 1 : attn_tc3_splits(a->len_q, a->n_heads, std::min<int64_t>(p.lw, a->n_local + 128) + p.n_snk);
  p.max_parts = p.one ? (int)infllm_attn_decode_max_parts(2, p.rows_w + p.n_snk) : p.n_split;
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t r = at;
    at += (bytes + 1023) / 1024 * 1024;
    return r;
  };
  p.k_rot = take((size_t)a->n_kv_heads * p.rows_w * 256);
  p.v_win = p.v_from_cache ? 0 : take((size_t)a->n_kv_heads * p.rows_w * 256);
  p.snk_k = take((size_t)a->n_kv_heads * p.n_snk * 256);
  p.snk_v = take((size_t)a->n_kv_heads * p.n_snk * 256);
  p.q_loc = take((size_t)a->n_heads * a->len_q * 256);
  p.q_snk = take((size_t)a->n_heads * a->len_q * 256);
  p.part = p.max_parts > 1 || p.one ? take((size_t)p.max_parts * a->n_heads * a->len_q * 130 * sizeof(float)) : 0;
  p.bytes = at;
  return p;
}

static int sink_check(const infllm_sink_window* a) {
  if (!a || a->n_heads <= 0 || a->n_kv_heads <= 0 || a->n_heads % a->n_kv_heads || a->len_q <= 0 || a->past_len < 0 ||
      a->n_local <= 0 || a->n_init < 0 || a->seen < a->len_q)
    return fail(INFLLM_E_BADARG, "sink_window: bad sizes");
  if (a->head_dim != 128) return fail(INFLLM_E_UNSUPPORTED, "sink_window: head_dim %d (128 is built)", a->head_dim);
  if (a->past_len + a->len_q > (1ll << 30)) return fail(INFLLM_E_UNSUPPORTED, "sink_window: too many tokens");
  const int64_t total = a->past_len + a->len_q;
  if (a->d_cache_k && (!a->d_cache_v || a->cache_head < 0 || a->cache_rows < a->cache_head || a->cache_rows > total))
    return fail(INFLLM_E_BADARG, "sink_window: a cache of %lld + %lld rows of %lld", (long long)a->cache_head,
                (long long)(a->cache_rows - a->cache_head), (long long)total);
  return INFLLM_OK;
}

}  // namespace infllm

extern "C" int64_t infllm_sink_window_scratch(const infllm_sink_window* args) {
  using namespace infllm;
  if (sink_check(args) != INFLLM_OK) return -1;
  return (int64_t)sink_plan(args).bytes;
}

extern "C" int infllm_sink_window_run(const infllm_sink_window* args, void* stream) {
  using namespace infllm;
  INFLLM_TRY(sink_check(args));
  const infllm_sink_window& a = *args;
  const SinkPlan p = sink_plan(args);
  cudaStream_t s = (cudaStream_t)stream;
  if (!a.d_q || !a.d_k || !a.d_v || !a.d_out || !a.d_scratch || !a.d_cos || !a.d_sin || (a.past_len > 0 && (!a.d_past_k || !a.d_past_v)))
    return fail(INFLLM_E_BADARG, "sink_window: null pointer");
  if ((a.q_hs | a.q_ts | a.k_hs | a.k_ts | a.past_hs | a.past_ts | a.o_hs | a.o_ts) % 8 ||
      ((uintptr_t)a.d_q | (uintptr_t)a.d_k | (uintptr_t)a.d_v | (uintptr_t)a.d_past_k | (uintptr_t)a.d_past_v | (uintptr_t)a.d_out |
       (uintptr_t)a.d_cache_k | (uintptr_t)a.d_cache_v | (uintptr_t)a.d_scratch) % 16)
    return fail(INFLLM_E_BADARG, "sink_window: rows must be 16-byte aligned");
  if (a.scratch_bytes < (int64_t)p.bytes) return fail(INFLLM_E_BADARG, "sink_window: %lld bytes of scratch, %zu needed", (long long)a.scratch_bytes, p.bytes);
  const int64_t pos_snk = a.stream_positions ? a.n_local + (int64_t)a.n_init - 1 : a.n_local - 1;
  if (p.lw > a.table_len || (p.n_snk > 0 && pos_snk >= a.table_len))
    return fail(INFLLM_E_BADARG, "sink_window: a rotary table of %lld rows", (long long)a.table_len);
  char* w = (char*)a.d_scratch;
  SinkPrepare P{};
  P.q = (const char*)a.d_q; P.k = (const char*)a.d_k; P.v = (const char*)a.d_v;
  P.past_k = (const char*)a.d_past_k; P.past_v = (const char*)a.d_past_v;
  P.cache_k = (char*)a.d_cache_k; P.cache_v = (char*)a.d_cache_v;
  P.k_rot = w + p.k_rot; P.v_win = p.v_from_cache ? nullptr : w + p.v_win;
  P.snk_k = w + p.snk_k; P.snk_v = w + p.snk_v; P.q_loc = w + p.q_loc; P.q_snk = w + p.q_snk;
  P.q_hs = a.q_hs; P.q_ts = a.q_ts; P.k_hs = a.k_hs; P.k_ts = a.k_ts; P.p_hs = a.past_hs; P.p_ts = a.past_ts;
  P.cos_t = a.d_cos; P.sin_t = a.d_sin;
  P.n_heads = a.n_heads; P.n_kv = a.n_kv_heads; P.len_q = (int)a.len_q; P.past_len = (int)a.past_len; P.total = (int)p.total;
  P.win0 = (int)p.win0; P.rows_w = (int)p.rows_w; P.n_snk = (int)p.n_snk;
  P.cache_head = (int)a.cache_head; P.cache_rows = (int)a.cache_rows;
  P.pos_w0 = (int)(p.win0 - p.w0); P.pos_q0 = (int)(p.lw - a.len_q); P.pos_snk = (int)pos_snk;
  P.rotate_snk = a.stream_positions;
  const int64_t rows = (int64_t)a.n_kv_heads * p.total + (int64_t)a.n_heads * a.len_q;
  INFLLM_DISPATCH_DTYPE(a.dtype, T, {
    launch_chained(sink_prepare_kernel<T>, dim3((unsigned)ceil_div(rows * 8, kSinkThreads)), dim3(kSinkThreads), 0, s, P);
  });
  INFLLM_LAUNCH_OK("sink_prepare_kernel");
  const char* v_base = p.v_from_cache ? (const char*)a.d_cache_v + (a.cache_rows - p.rows_w) * 256 : w + p.v_win;
  const int64_t v_hs = (p.v_from_cache ? a.cache_rows : p.rows_w) * 128;
  const int64_t snk_off = a.seen - a.len_q;  // query i is token snk_off + i of the sequence: it sees sink key j when
                                             // i - j + snk_off >= n_local
  if (p.one) {
    const int64_t snk_vis = std::max<int64_t>(0, std::min<int64_t>(p.n_snk, snk_off - a.n_local + 1));
    KvSeg segs[2];
    const int32_t qsel[2] = {0, 1};
    segs[0] = {P.k_rot, v_base, p.rows_w * 128, 128, (int32_t)p.rows_w, v_hs};
    segs[1] = {P.snk_k, P.snk_v, p.n_snk * 128, 128, (int32_t)snk_vis};
    float *part = (float*)(w + p.part), *plse = part + (size_t)p.max_parts * a.n_heads * 128;
    int n = 0;
    INFLLM_TRY(attn_decode_launch(P.q_loc, P.q_snk, 128, a.n_heads, a.n_kv_heads, 128, 2, segs, qsel, part, plse, p.max_parts, &n,
                                  -1, nullptr, a.dtype, s, nullptr));
    return lse_merge_launch(part, plse, n, a.n_heads, 128, a.d_out, a.o_hs, nullptr, a.dtype, s, nullptr, 0, nullptr, 0, nullptr);
  }
  AttnTcParams A{};
  const bool pair = attn_tc3_pairs(a.len_q, a.n_heads, a.n_kv_heads);
  INFLLM_TRY(encode_rows_map(&A.maps[0], a.dtype, P.q_loc, a.len_q, a.n_heads, a.len_q * 128, 128, kBoxTile));
  INFLLM_TRY(encode_rows_map(&A.maps[1], a.dtype, P.k_rot, p.rows_w, a.n_kv_heads, p.rows_w * 128, 128, box_k(pair)));
  INFLLM_TRY(encode_rows_map(&A.maps[2], a.dtype, v_base, p.rows_w, a.n_kv_heads, v_hs, 128, box_v(pair)));
  INFLLM_TRY(tc_get_error_ptr(&A.err));
  A.exact = 1;
  A.n_stage = 1; A.n_heads = a.n_heads; A.n_kv_heads = a.n_kv_heads; A.lq = a.len_q;
  A.out = a.d_out; A.o_hs = a.o_hs; A.o_ts = a.o_ts; A.scale_log2 = kLog2e / sqrtf(128.f);
  A.stage[0] = {0, 0, INFLLM_MASK_WINDOW, 0, 1, 0, p.lw - a.len_q, a.n_local, p.lw};
  A.seg[0] = {1, 2, 0, -1, -1, (int32_t)p.lw};
  if (p.n_snk > 0) {
    INFLLM_TRY(encode_rows_map(&A.maps[3], a.dtype, P.q_snk, a.len_q, a.n_heads, a.len_q * 128, 128, kBoxTile));
    INFLLM_TRY(encode_rows_map(&A.maps[4], a.dtype, P.snk_k, p.n_snk, a.n_kv_heads, p.n_snk * 128, 128, box_k(pair)));
    INFLLM_TRY(encode_rows_map(&A.maps[5], a.dtype, P.snk_v, p.n_snk, a.n_kv_heads, p.n_snk * 128, 128, box_v(pair)));
    A.stage[1] = {3, 0, INFLLM_MASK_COMPLEMENT, 1, 2, 0, snk_off, a.n_local, p.n_snk};
    A.seg[1] = {4, 5, 0, -1, -1, (int32_t)p.n_snk};
    A.n_stage = 2;
  }
  A.n_split = p.n_split;
  if (p.n_split == 1) return attn_tc3_launch(A, a.dtype, s);
  const int64_t q_rows = (int64_t)a.n_heads * a.len_q;
  A.part_acc = (float*)(w + p.part);
  A.part_m = A.part_acc + p.n_split * q_rows * 128;
  A.part_l = A.part_m + p.n_split * q_rows;
  INFLLM_TRY(attn_tc3_launch(A, a.dtype, s));
  return attn_tc_combine_launch(A.part_acc, A.part_m, A.part_l, p.n_split, a.n_heads, a.len_q, a.d_out, a.o_hs, a.o_ts, nullptr,
                                nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, a.dtype, s);
}
