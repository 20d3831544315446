// Parameters of the one-launch decode token (token.cu), of one context memory or of several at once.
#pragma once
#include "common.cuh"

namespace infllm {

constexpr int kTokMaxUpdates = 96;  // changes of the table of unit addresses that travel with a token
constexpr uint32_t kTokSpin = 1u << 22;  // polls after which a wait gives up: a second or two
constexpr int kTokErrTimeout = 1;   // code of the error record: a bounded wait ran out (700 ids, 701 partials, 702 scores)

struct TokenParams {
  struct Seg {
    const void *k, *v;
    int64_t hs;  // head stride, elements; rows of 128 elements, contiguous
    int32_t len, pad;
  };
  // the token
  const void *q, *k, *v;
  int64_t q_hs, k_hs, v_hs;
  void *k_raw, *k_rot, *v_out;  // its row in the token buffers (KV head 0), heads kv_hs elements apart
  int64_t kv_hs;
  const float *cos_t, *sin_t;
  int64_t pos_loc, pos_glb;
  // retrieval.  A "word" is {value, token number} in 8 bytes.
  const void* bk;
  unsigned long long* score_words;  // (n)
  unsigned long long* id_words;     // (k_top)
  unsigned long long* ids_host;     // pinned: the same words
  int32_t n, width, k_top, n_upd;
  // attention: [0] the window without the new token (window-relative queries), [1] sink, [2] overflow (one-angle queries)
  Seg rest[3];
  int32_t rest_begin[4];  // first 16-key group of each
  unsigned long long* ptrs;  // table of unit addresses; the landing slots of the k_top positions from landing_at on
  int64_t landing_at, unit_bytes;
  int32_t unit_len, n_heads, n_kv, group, n_runs;
  uint32_t spin;  // kTokSpin
  float scale_log2;
  unsigned long long* part_words;  // (n_runs, n_heads, 129): a run's normalised outputs and their log-sum-exp
  float* logits;                   // (n_heads, logit_hs)
  int64_t logit_hs;
  float* win_score;  // accumulated scores from the window's first key on, heads score_hs apart
  int64_t score_hs;
  void* out;
  int64_t o_hs;
  int32_t too_large;  // (for tests) a grid that no device can hold: the launch is refused
  uint32_t seq;  // number of this token among those that have used these words; never 0
  int32_t *err, *err_host;
  int32_t upd_id[kTokMaxUpdates];
  unsigned long long upd_val[kTokMaxUpdates];
};

constexpr int kTokMaxBatch = 8;  // contexts of one launch: their parameters are 14 KB

// runs per KV head over `sms` SMs (0: these sizes are not for token_kernel)
int token_runs(int n_heads, int n_kv_heads, int head_dim, int64_t n_units, int topk, int block_size, int sms);
// how many contexts with that many KV heads share a launch on a device of `sms` SMs
int token_batch_max(int n_kv_heads, int sms);
// n contexts' tokens, each with the n_runs its share of the SMs gives it; INFLLM_E_UNSUPPORTED: the CTAs cannot all be
// resident where this process runs
int token_launch(const TokenParams* P, int n, int dtype, cudaStream_t s);

}  // namespace infllm
