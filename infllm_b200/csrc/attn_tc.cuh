// Parameter blocks and host entry points of the tensor-core attention kernels (attn_tc.cu).
#pragma once
#include "attn_common.cuh"
#include "tc_common.cuh"

namespace infllm {

constexpr int kTcMaxMaps = 12;
constexpr int kTile = 128;
// boxes of the tensor maps: rows, and halves of the 128 dimensions
struct TcBox {
  uint32_t rows, halves;
};
constexpr TcBox kBoxTile = {kTile, 2};  // a whole tile: queries, and keys and values of a CTA that works alone
constexpr TcBox kBoxPairK = {kTile / 2, 2}, kBoxPairV = {kTile, 1};  // a CTA's share of a pair's keys and values
constexpr TcBox box_k(bool pair) { return pair ? kBoxPairK : kBoxTile; }
constexpr TcBox box_v(bool pair) { return pair ? kBoxPairV : kBoxTile; }
// Exec blocks of up to one tile of queries are attended to in fp32's precision throughout, like every stage of the
// multi-stage class and the sink + window types.  Up to 64 queries they used to be the shape-generic kernel's, which does;
// up to 128 their key tiles are cut into runs, and where a row is one key's for the most part it matters which tiles share
// a reference maximum (an 8192-token prompt in exec blocks of 128: largest error 2.6e-2 instead of 2.0e-2, 1.2 % more in
// the 2-norm).  It costs them 3 % (128 queries by 1152 + 700 keys, merge included: 15.2 us instead of 14.8) to 9 % (128 by 4224 + 2304:
// 24.5, 22.6; 37 by 4133 + 2200: 22.5, 20.7).  Larger exec blocks, which it would cost 7 to 10 % (256 of 32/32 heads in two runs: 40.0,
// 37.3; 512 by 4608 + 2688: 60.3, 54.7), have had the cubic and the lazy maximum all along.
constexpr int kExactQueries = kTile;

struct TcSeg {
  int16_t map_k, map_v;  // indices into AttnTcParams::maps
  int32_t tok0;          // token coordinate of the segment's first key
  int32_t c3_k, c3_v;    // 5th coordinate for rank-5 maps (cache slots), -1 for rank-4 maps
  int32_t len;
};

struct TcStage {
  int32_t map_q, q_row0;
  int32_t mask_mode, seg_begin, seg_end, pad;
  int64_t mask_offset, mask_size, lk;
};

struct AttnTcParams {
  alignas(64) CUtensorMap maps[kTcMaxMaps];
  TcStage stage[kMaxStage];
  TcSeg seg[kMaxSeg];
  int32_t n_stage, n_heads, n_kv_heads, pad;
  int64_t lq;
  void* out;
  int64_t o_hs, o_ts;
  float* lse;
  float scale_log2;
  int* err;
  // The key tiles of a work item are cut into n_split runs; with n_split > 1 every run writes an un-normalised
  // partial (acc, m, l) and attn_tc_combine merges them.  With n_split == 1 the kernel writes its state here
  // instead of out / lse when part_acc is set, and folds in the state st_* when that is set (it may be the same memory).
  int32_t n_split;
  int32_t exact;    // exponentials to fp32's precision throughout (see kExactQueries)
  float* part_acc;  // (n_split, H, lq, 128)
  float* part_m;    // (n_split, H, lq)
  float* part_l;    // (n_split, H, lq)
  const float *st_acc, *st_m, *st_l;
};

constexpr int kNoBound = -(1 << 30);
struct ColsumTcParams {
  alignas(64) CUtensorMap map_q, map_k;
  int32_t q_row0, k_tok0, n_heads, group;
  int64_t lq, lk;
  int32_t accumulate, tiles_per_cta;
  int32_t late_wait;  // nothing is read that the kernel before on the stream writes: it is waited for at the end only
  int32_t lo_add, hi_add;  // queries [j + lo_add, j + hi_add] see key j; kNoBound: no bound on that side
  const float* lse;
  float* score;
  int64_t score_hs;
  float scale_log2;
  int* err;
};


int encode_rows_map(CUtensorMap* map, int dtype, const void* base, int64_t rows, int64_t heads, int64_t hs, int64_t ts,
                    TcBox box);
bool tc_rows_ok(const void* base, int64_t hs, int64_t ts);
int tc_get_error_ptr(int** p);
// one CTA per (128-query tile, head)
int attn_tc3_launch(const AttnTcParams& P, int dtype, cudaStream_t s);
int attn_tc3_splits(int64_t lq, int n_heads, int64_t keys);
// whether a launch of these sizes runs in pairs of CTAs: its maps of keys and values have the boxes of one
bool attn_tc3_pairs(int64_t lq, int n_heads, int n_kv_heads);
int attn_tc_combine_launch(const float* acc, const float* m, const float* l, int n_split, int n_heads, int64_t lq, void* out,
                           int64_t o_hs, int64_t o_ts, float* lse, const float* st_acc, const float* st_m,
                           const float* st_l, float* new_acc, float* new_m, float* new_l, int dtype, cudaStream_t s);
int colsum_tc_launch_maps(const CUtensorMap& map_q, const CUtensorMap& map_k, int q_row0, int k_tok0, int n_heads,
                          int n_kv_heads, int64_t lq, int64_t lk, int mask_mode, int64_t mask_offset,
                          int64_t mask_size, const float* lse, float* score, int64_t score_hs, int accumulate,
                          bool late_wait, int dtype, cudaStream_t s);
int colsum_tc_launch(const void* q, int64_t q_hs, int64_t q_ts, const void* k, int64_t k_hs, int64_t k_ts, int n_heads,
                     int n_kv_heads, int64_t lq, int64_t lk, int mask_mode, int64_t mask_offset, int64_t mask_size,
                     const float* lse, float* score, int64_t score_hs, int accumulate, int dtype, cudaStream_t s);

}  // namespace infllm
