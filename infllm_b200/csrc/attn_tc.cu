// Tensor-core (tcgen05 + TMEM + TMA) attention kernels for head_dim 128.
//
// attn_tc3_kernel   one 128-query tile of one head per CTA, all stages of an exec block fused:
//                   local window stage (window-relative rotated q/k, causal window mask) and global
//                   stage (one-angle q; retrieved units in their cache slots, init sink, overflow),
//                   jointly normalised.  Two CTAs of a cluster share the key tiles (cta_group::2).  Warp-specialised: two
//                   teams of four softmax warps (a thread per query row, key tiles in turn), 1 TMA producer warp, two
//                   issuing warps (S = Q K^T and O += P V).  S accumulates in TMEM (three buffers), P is written back over
//                   its S columns and feeds the P V product from TMEM, O stays in TMEM for the whole tile with lazy
//                   rescaling.  Where the grid leaves SMs idle the key tiles are cut into runs.
// colsum_tc_kernel  per-key score pass: S^T = K Q^T with keys as TMEM lanes; a CTA keeps one head's query tiles
//                   resident and streams a run of key tiles through a TMA ring and four TMEM buffers; four
//                   threads per key sum exp2(s - lse) over the queries that see it.
// Every mbarrier wait is bounded; a wait that runs out records an error code and the CTA unwinds.
#include <algorithm>
#include <type_traits>

#include "attn_common.cuh"
#include "tc_common.cuh"
#include "ring.cuh"
#include "attn_tc.cuh"

namespace infllm {

using namespace tc;

__device__ int g_tc_error[4];  // [0] code, [1] where, [2] blockIdx.x, [3] blockIdx.y

__device__ __forceinline__ void record_error(int* err, int code, int where) {
  if (atomicCAS(&err[0], 0, code) == 0) {
    err[1] = where;
    err[2] = blockIdx.x;
    err[3] = blockIdx.y;
  }
}

// wait that also gives up when another role of the CTA has already failed
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err,
                                              int where) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    if (i > 64) __nanosleep(i > 4096 ? 256 : 32);
  }
  *abort_flag = 1;
  record_error(err, kErrWaitTimeout, where);
  return false;
}

// the same for a whole (converged) warp, whose lanes go on or give up together.  Nearly always the phase has passed or is about
// to: one look, in straight code, before the loop, in which lanes could part (75 cycles a wait instead of 110; four such waits are in
// the way of a key tile: 512 queries by 4608 + 2688 keys 5 % less)
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err, int where) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return __all_sync(0xffffffffu, wait_or_abort(bar, parity, abort_flag, err, where));
}

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Blackwell's packed fp32 pairs and three-input maximum: half the instructions of the scalar forms
__device__ __forceinline__ float fmax3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float2 ffma2(float a0, float a1, float2 b, float2 c) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rc, rd; mov.b64 ra, {%2,%3}; mov.b64 rb, {%4,%5}; mov.b64 rc, {%6,%7}; "
      "fma.rn.f32x2 rd, ra, rb, rc; mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y) : "f"(a0), "f"(a1), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rd; mov.b64 ra, {%2,%3}; mov.b64 rb, {%4,%5}; mul.rn.f32x2 rd, ra, rb; mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
  float2 d;
  asm("{ .reg .b64 ra, rb, rd; mov.b64 ra, {%2,%3}; mov.b64 rb, {%4,%5}; add.rn.f32x2 rd, ra, rb; mov.b64 {%0,%1}, rd; }"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return d;
}

// exp2 of a pair on the FMA and integer pipes (the special-function unit does 16 per clock per SM, which bounds the
// softmax when every exponential goes there): x = n + f with n the nearest integer (magic-number rounding) and f in
// [-0.5, 0.5], 2^f by a polynomial whose relative error was minimised over that interval (least squares on Chebyshev
// points), times 2^n.  A NaN stays one; arguments below -126, those of masked keys too, give 2^-126.
//   cubic    7.5e-5: a twentieth of the rounding of a bf16 P, a third to a sixth of that of an fp16 P
//   quartic  2.6e-6
//   quintic  2e-7 as evaluated in fp32, which is what ex2.approx has: where exp2f was
__device__ __forceinline__ float max_nan(float a, float b) {
  float d;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(d) : "f"(a), "f"(b));
  return d;
}
template <int kDegree>
__device__ __forceinline__ float2 ex2_poly2(float2 x) {
  static_assert(kDegree >= 3 && kDegree <= 5, "");
  x.x = max_nan(x.x, -126.f);
  x.y = max_nan(x.y, -126.f);
  const float2 magic = make_float2(12582912.f, 12582912.f), neg_magic = make_float2(-12582912.f, -12582912.f);
  const float2 t = fadd2(x, magic);
  const float2 n = fadd2(t, neg_magic);
  const float2 f = fadd2(x, make_float2(-n.x, -n.y));
  auto c2 = [](float c) { return make_float2(c, c); };
  float2 p;
  if (kDegree == 3) {
    p = ffma2(f.x, f.y, c2(0.05517167f), c2(0.24261113f));
    p = ffma2(p.x, p.y, f, c2(0.69326097f));
    p = ffma2(p.x, p.y, f, c2(0.99992806f));
  } else if (kDegree == 4) {
    p = ffma2(f.x, f.y, c2(0.0095701022f), c2(0.055917859f));
    p = ffma2(p.x, p.y, f, c2(0.24024744f));
    p = ffma2(p.x, p.y, f, c2(0.69312179f));
    p = ffma2(p.x, p.y, f, c2(0.99999928f));
  } else {
    p = ffma2(f.x, f.y, c2(0.00132669706f), c2(0.00967545994f));
    p = ffma2(p.x, p.y, f, c2(0.0555074252f));
    p = ffma2(p.x, p.y, f, c2(0.240221217f));
    p = ffma2(p.x, p.y, f, c2(0.693146944f));
    p = ffma2(p.x, p.y, f, c2(1.00000012f));
  }
  // a product, not an addition to the exponent's bits: that would make a number of a NaN
  return fmul2(p, make_float2(__int_as_float((__float_as_int(t.x) << 23) + 0x3f800000),
                              __int_as_float((__float_as_int(t.y) << 23) + 0x3f800000)));
}

// tiles [first, last] of a segment that intersect the visible key range [vis_lo, vis_hi] of the stage
__device__ __forceinline__ bool seg_tiles(int64_t vis_lo, int64_t vis_hi, int64_t seg_j0, int seg_len, int* first,
                                          int* last) {
  int64_t a = vis_lo - seg_j0, b = vis_hi - seg_j0;
  if (a < 0) a = 0;
  if (b > seg_len - 1) b = seg_len - 1;
  if (a > b) return false;
  *first = (int)(a / kTile);
  *last = (int)(b / kTile);
  return true;
}

// ------------------------------------------------------------------------------------------------
// attn_tc3_kernel: one 128-query tile of one head per CTA; P never touches shared memory.  P = exp2(S - m) goes back
// into the TMEM columns of its S buffer as packed 16-bit pairs and is the A operand of the P V product from there, and there are
// three S/P buffers in TMEM.
// Pairs of CTAs (attn_tc3_pairs: where a KV head's query tiles, over all its query heads, come out even): the products are
// cta_group::2, 256 rows of two CTAs by 128 keys, and a CTA fetches and holds half of every K and V tile.  That halves the
// bytes from L2 to shared memory (a lone CTA's 64 KB a tile take 1600 cycles at 40 bytes per clock and SM) and leaves room for
// four tiles in flight.  Alone (12/12 heads by 3 tiles: 384 queries by 4480 + 2688 keys) the same code takes 51.3 us, 55.5
// with the waits that are named below.  Two query heads of a KV head make a pair, so that both see the same keys; two tiles of one head where there is only one.
// The softmax is two teams of four warps with the key tiles in turn, a thread per query row: no exchange within a row, and one
// team's maximum and waits under the other's exponentials.  One pair of exponentials in eight is a polynomial on the FMA pipe (none:
// 3 % more time; a quarter: 1 % less, kExact 1 % more).
// Issuers and producer are whole warps of which one lane issues: eight products in 120 cycles instead of 600, and one load per
// tile and operand (both 64-dimension halves in one box) instead of four at about 390 cycles each, which was 1570 per tile
// whatever their size.  The producer asks for K one tile ahead of V.
// kExact (see kExactQueries): that polynomial is as good as exp2f, and the reference
// maximum of a row follows its maximum, so that the largest probabilities have no rounding (2 to 6 % less error of an
// output against 64 bits); whenever a row's maximum grows, O is scaled.
// What bounds it (clock stamps, cycles): a key tile every 1420, of which the tensor pipe needs 1024.  Two ways round are equally long:
// that of a team, two tiles in 2840 - exponentials 1500, maximum 400, the other team's 230, the rest waits and hand-overs that are
// there already and cost 75 to 100 each - and that of an S/P buffer, three tiles: product 700, softmax 2300, to the issuer 250, P V and
// back 850.  Set-up and first loads take 6000 and the end 4500.
// 32/8 heads, 512 queries by 4608 + 2688 keys, twenty launches in a row: 54.7 us, with each wait through a loop, a barrier for every
// maximum and ordering cluster barriers 60.6 (kExact: 60.3, 65.1; on another B200 52.7 and 58.2, 57.5 and 62.3); 256 queries of 32/32
// heads in two runs, merge included, 37.3, 41.2; 128 queries by 1152 + 700 in four 15.2, 16.3; 4096 queries by 8192 keys, kExact, 264, 286.
namespace tc3 {
constexpr int kBufs = 3;                         // S/P buffers in TMEM
constexpr int kQ = 0;                            // a tile for each of the two stages
constexpr int kK = kQ + 4 * kSubTileBytes;       // two stages of a tile, or four of a CTA's half of one
constexpr int kV = kK + 4 * kSubTileBytes;       // the same
constexpr int kBar = kV + 4 * kSubTileBytes;
constexpr int kTmax = kBar + 512;                // the rows' maxima in the last four tiles, each with its tile's number
constexpr int kXmax = kTmax + 4 * 1024;          // per team: the reference its row sums stand at
constexpr int kXsum = kXmax + 2 * 512;           // per team: row sums
constexpr int kPlan = kXsum + 2 * 512;
constexpr int kTotal = kPlan + 32 + kMaxSeg * 32;
constexpr int kPolyEvery = 8;
enum { T3_Q_FULL0 = 0, T3_K_FULL0 = 2, T3_K_EMPTY0 = 6, T3_V_FULL0 = 10, T3_V_EMPTY0 = 14, T3_S_FULL0 = 18,
       T3_P_FULL0 = 21, T3_PV_DONE0 = 24, T3_O_FULL = 27, T3_N_BARS };
constexpr int kWarpTma = 8, kWarpPv = 9, kWarpQk = 10;  // behind the eight softmax warps
constexpr int kThreads = 11 * 32;
// What a CTA does, worked out once, by one warp: the segments of its run that have tiles, in order.  Left to every role's own
// loop over stages and segments, the 64-bit arithmetic for 20 segments took 8400 cycles before the first product of a run
// and 6000 behind its last one, of 46000 for 12 tiles.
struct Part {
  int32_t n;           // key tiles
  int32_t tok;         // token coordinate of the first
  int32_t c3_k, c3_v;
  int16_t map_k, map_v;
  int32_t stage;       // bit 8: the stage's last part of this run
  int32_t j;           // the first tile's first key within the stage
  int32_t lim;         // the segment's last key within the stage
};
static_assert(sizeof(Part) == 32, "");
struct Plan {
  int32_t n_parts, n_tiles, pad[6];
  Part part[kMaxSeg];
};
__device__ __forceinline__ int warp_scan(int v) {  // inclusive
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}
// one warp; queries [i0, i1], run `split` of n_split.  kPer segments per lane: one for the usual numbers.
template <int kPer>
__device__ __forceinline__ void make_plan(const AttnTcParams& P, int64_t i0, int64_t i1, int split, Plan* plan) {
  static_assert(kMaxStage == 2, "");
  const int lane = threadIdx.x & 31, n_stage = P.n_stage, n_seg = P.stage[n_stage - 1].seg_end;
  const int seg1 = n_stage > 1 ? P.stage[1].seg_begin : n_seg;  // the second stage's first
  int64_t vlo[2] = {0, 0}, vhi[2] = {-1, -1};
  visible_key_range(P.stage[0].mask_mode, P.stage[0].mask_offset, P.stage[0].mask_size, i0, i1, P.stage[0].lk, &vlo[0], &vhi[0]);
  if (n_stage > 1)
    visible_key_range(P.stage[1].mask_mode, P.stage[1].mask_offset, P.stage[1].mask_size, i0, i1, P.stage[1].lk, &vlo[1], &vhi[1]);
  int len[kPer], j0[kPer], tf[kPer], n[kPer], first[kPer];
  int keys = 0, base = 0, tiles = 0;  // keys of the segments before, of the first stage's; tiles
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int sg = e * 32 + lane;
    len[e] = sg < n_seg ? P.seg[sg].len : 0;
    const int inc = warp_scan(len[e]);
    j0[e] = keys + inc - len[e];
    keys += __shfl_sync(0xffffffffu, inc, 31);
    if (seg1 / 32 == e) base = __shfl_sync(0xffffffffu, j0[e], seg1 & 31);
  }
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int sg = e * 32 + lane, st = sg >= seg1;
    if (st) j0[e] -= base;
    const int64_t lo = st ? vlo[1] : vlo[0], hi = st ? vhi[1] : vhi[0];
    int tl;
    n[e] = 0;
    if (sg < n_seg && lo <= hi && seg_tiles(lo, hi, j0[e], len[e], &tf[e], &tl)) n[e] = tl - tf[e] + 1;
    const int inc = warp_scan(n[e]);
    first[e] = tiles + inc - n[e];
    tiles += __shfl_sync(0xffffffffu, inc, 31);
  }
  int g0 = 0, g1 = tiles;
  if (P.n_split > 1) g0 = tiles * split / P.n_split, g1 = tiles * (split + 1) / P.n_split;
  int at = 0, last[2] = {-1, -1};
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int sg = e * 32 + lane, st = sg >= seg1;
    const int a = first[e] > g0 ? first[e] : g0, b = first[e] + n[e] < g1 ? first[e] + n[e] : g1;
    const unsigned has = __ballot_sync(0xffffffffu, a < b), has1 = __ballot_sync(0xffffffffu, a < b && st);
    if (a < b) {
      const TcSeg& G = P.seg[sg];
      Part& R = plan->part[at + __popc(has & ((1u << lane) - 1u))];
      const int t = tf[e] + a - first[e];
      R.n = b - a, R.tok = G.tok0 + t * kTile, R.c3_k = G.c3_k, R.c3_v = G.c3_v, R.map_k = G.map_k, R.map_v = G.map_v;
      R.stage = st, R.j = j0[e] + t * kTile, R.lim = j0[e] + len[e] - 1;
    }
    if (has != has1) last[0] = at + __popc(has & ~has1) - 1;  // (the first stage's parts come before the second's)
    if (has1) last[1] = at + __popc(has) - 1;
    at += __popc(has);
  }
  __syncwarp();
  if (lane == 0) {
    plan->n_parts = at, plan->n_tiles = g1 - g0;
    if (last[0] >= 0) plan->part[last[0]].stage |= 256;
    if (last[1] >= 0) plan->part[last[1]].stage |= 256;
  }
}
// a word of shared memory that another thread of the CTA watches: it is stored and loaded whole
__device__ __forceinline__ uint64_t look_word(uint32_t addr) {
  uint64_t v;
  asm volatile("ld.volatile.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void leave_word(uint32_t addr, uint64_t v) { asm volatile("st.volatile.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory"); }
// exponentials of 32 columns of a row, packed; sums into rs
template <typename T, bool kExact>
__device__ __forceinline__ void exp_chunk(const float2* a, float2* rs, uint32_t* pk) {
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    float2 p;
    if (k % kPolyEvery == kPolyEvery - 1) {
      p = ex2_poly2<kExact ? 5 : 3>(a[k]);  // one pair in kPolyEvery off the special-function unit
    } else {
      p = make_float2(ex2_approx(a[k].x), ex2_approx(a[k].y));
    }
    rs[k & 3] = fadd2(rs[k & 3], p);
    typename Act<T>::T2 v = Act<T>::from_f2(p.x, p.y);
    pk[k] = *reinterpret_cast<uint32_t*>(&v);
  }
}
// 32 columns of scores into exponents; what they were loaded into may be loaded into again behind it
__device__ __forceinline__ void arg_chunk(const float* s, float sc, float neg_m, float2* a) {
  const float2 sc2 = make_float2(sc, sc), nm2 = make_float2(neg_m, neg_m);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    a[k] = ffma2(s[2 * k], s[2 * k + 1], sc2, nm2);
    asm volatile("" : "+f"(a[k].x), "+f"(a[k].y));
  }
}
// a row's reference maximum behind a tile whose maximum is m_tile.  Lazy: it only moves when the maximum grew by more than
// 2^8 - or, kExact, at all, so that the largest probabilities of a row are the ones that a 16-bit P holds without a rounding
template <bool kExact>
__device__ __forceinline__ float next_ref(float m, float m_tile) {
  return m_tile - m > (kExact ? 0.f : 8.f) ? m_tile : m;  // (from -inf: any number)
}
__device__ __forceinline__ void max_chunk(const float* s, float* mx) {
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    mx[0] = fmax3(mx[0], s[i], s[i + 1]);
    mx[1] = fmax3(mx[1], s[i + 2], s[i + 3]);
    mx[2] = fmax3(mx[2], s[i + 4], s[i + 5]);
    mx[3] = fmax3(mx[3], s[i + 6], s[i + 7]);
  }
}
}  // namespace tc3

template <typename T, bool kExact, bool kPair>
__global__ void __launch_bounds__(tc3::kThreads, 1) attn_tc3_kernel(const __grid_constant__ AttnTcParams P) {
  using namespace tc3;
  constexpr int kStages = kPair ? 4 : 2;
  constexpr int kCtas = kPair ? 2 : 1;
  constexpr int kShare = 2 * kSubTileBytes / kCtas;  // bytes of a K or V tile that a CTA holds
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t sQ = s_base + kQ, sK = s_base + kK, sV = s_base + kV;
  const uint32_t bars = s_base + kBar;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBar + T3_N_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kBar + T3_N_BARS * 8 + 8);
  const uint32_t tmax = s_base + kTmax;
  float* xmax = reinterpret_cast<float*>(smem + kXmax);
  float* xsum = reinterpret_cast<float*>(smem + kXsum);
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  const int rank = kPair ? (int)(blockIdx.x & 1) : 0;
  // the barriers that count both CTAs' loads and probabilities are those of the first
  auto lead_bar = [&](int i) { return kPair ? cluster_map(bar(i), 0) : bar(i); };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // work items of a KV head: (query tile, head), the heads of a tile side by side; a pair of CTAs takes two in a row
  const int group = P.n_heads / P.n_kv_heads, hkv = blockIdx.y;
  const int qt = (int)blockIdx.x / group, h = hkv * group + (int)blockIdx.x % group;
  const int64_t i0 = (int64_t)qt * kTile;
  const int rows_q = (int)((P.lq - i0) < kTile ? (P.lq - i0) : kTile);
  const int split = blockIdx.z;

  if (warp == 0) {
    static_assert(T3_N_BARS <= 32, "");
    if (lane < T3_N_BARS) mbar_init(bar(lane), lane >= T3_P_FULL0 && lane < T3_P_FULL0 + kBufs ? 4u * kCtas : 1u);
    if (lane == 0) *abort_flag = 0;
    mbar_fence_init();
  }
  for (int i = threadIdx.x; i < 4 * kTile; i += kThreads) reinterpret_cast<uint64_t*>(smem + kTmax)[i] = ~0ull;  // (no tile's number)
  if (kPair) cluster_arrive();  // (waited for below: the other CTA's barriers stand before anything is signalled on them)
  if (warp == kWarpQk && lane < P.n_stage) {  // the descriptors of the first loads are on their way while the run's parts are worked out
    const TcStage& S = P.stage[lane];
    tma_prefetch_map(&P.maps[S.map_q]);
    if (S.seg_begin < S.seg_end) {
      tma_prefetch_map(&P.maps[P.seg[S.seg_begin].map_k]);
      tma_prefetch_map(&P.maps[P.seg[S.seg_begin].map_v]);
    }
  }
  tc3::Plan* plan = reinterpret_cast<tc3::Plan*>(smem + kPlan);
  if (warp == kWarpTma) {  // the run's parts, of all queries of the pair
    const int64_t u0 = kPair ? (int64_t)((int)(blockIdx.x & ~1u) / group) * kTile : i0;
    const int64_t u1 = kPair ? (int64_t)((int)(blockIdx.x | 1u) / group + 1) * kTile : i0 + kTile;
    const int64_t last = (u1 < P.lq ? u1 : P.lq) - 1;
    if (P.stage[P.n_stage - 1].seg_end <= 32) make_plan<1>(P, u0, last, split, plan);
    else make_plan<(kMaxSeg + 31) / 32>(P, u0, last, split, plan);
  }

  if (warp == kWarpPv) {
    tmem_alloc<kPair>(smem_u32(tmem_slot), 512);
    tmem_relinquish<kPair>();
  }
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_wait();
  tc_fence_after();
  chain_wait();  // up to here nothing has been read or written that the kernel before on the stream has to do with
  const uint32_t tmem = *tmem_slot;
  const uint32_t tO = tmem + 384;  // three S/P buffers at columns [0,128), [128,256), [256,384)
  constexpr bool kBf16 = !std::is_same<T, __half>::value;
  constexpr uint32_t idesc_qk = make_idesc(kBf16, 128 * kCtas, 128, false);
  constexpr uint32_t idesc_pv = make_idesc(kBf16, 128 * kCtas, 128, true);

  if (warp == kWarpTma) {
    // ======================================================================== TMA producer
    // K runs one tile ahead of V: the buffer of K is free as soon as its S has been formed, that of V only
    // when its P V product has run, late in the tile's cycle; asked for in tile order, K queued
    // behind that wait and the next S was not ready when the softmax warps came for it.
    // Of a pair, each CTA fetches its own queries, 64 of a tile's keys and half of the values' dimensions.
    // One load per tile and operand, asked for by one lane of a warp whose lanes stay together: four loads a tile from a
    // thread of its own took 1570 cycles a tile whatever their size, and nothing could be faster than that.
    const bool lead = elect_one();
    int it = 0, sidx = 0, stage = -1;
    bool ok = true;
    struct { int it, tok, c3, map; } pend = {-1, 0, 0, 0};  // the V tile that has not been asked for yet
    auto load_v = [&]() {
      const int b = pend.it % kStages;
      if (pend.it >= kStages) ok = warp_wait(bar(T3_V_EMPTY0 + b), ((pend.it / kStages) - 1) & 1, abort_flag, P.err, 602);
      if (!ok) return;
      if (lead) {
        const uint32_t dv = sV + b * kShare, fb = lead_bar(T3_V_FULL0 + b);
        if (rank == 0) mbar_expect_tx(bar(T3_V_FULL0 + b), 2 * kSubTileBytes);
        if (pend.c3 < 0) tma_load_4d<kPair>(dv, &P.maps[pend.map], fb, 0, pend.tok, rank, hkv);
        else tma_load_5d<kPair>(dv, &P.maps[pend.map], fb, 0, pend.tok, rank, hkv, pend.c3);
      }
      __syncwarp();
      pend.it = -1;
    };
    const int n_parts = plan->n_parts;
    for (int p = 0; p < n_parts && ok; ++p) {
      const Part R = plan->part[p];
      if ((R.stage & 255) != stage) {  // the stage's queries, in a buffer of their own
        stage = R.stage & 255;
        const TcStage& S = P.stage[stage];
        if (lead) {
          const uint32_t dq = sQ + sidx * 2 * kSubTileBytes, fb = lead_bar(T3_Q_FULL0 + sidx);
          if (rank == 0) mbar_expect_tx(bar(T3_Q_FULL0 + sidx), 2 * kSubTileBytes * kCtas);
          tma_load_4d<kPair>(dq, &P.maps[S.map_q], fb, 0, S.q_row0 + (int)i0, 0, h);
        }
        __syncwarp();
        ++sidx;
      }
      for (int t = 0; t < R.n && ok; ++t) {
        const int b = it % kStages, tok = R.tok + t * kTile;
        if (it >= kStages) ok = warp_wait(bar(T3_K_EMPTY0 + b), ((it / kStages) - 1) & 1, abort_flag, P.err, 601);
        if (!ok) break;
        if (lead) {
          const uint32_t dk = sK + b * kShare, fb = lead_bar(T3_K_FULL0 + b);
          if (rank == 0) mbar_expect_tx(bar(T3_K_FULL0 + b), 2 * kSubTileBytes);
          if (R.c3_k < 0) tma_load_4d<kPair>(dk, &P.maps[R.map_k], fb, 0, tok + 64 * rank, 0, hkv);
          else tma_load_5d<kPair>(dk, &P.maps[R.map_k], fb, 0, tok + 64 * rank, 0, hkv, R.c3_k);
        }
        __syncwarp();
        if (pend.it >= 0) load_v();
        if (!ok) {
          ++it;  // its K has been asked for
          break;
        }
        pend.it = it, pend.tok = tok, pend.c3 = R.c3_v, pend.map = R.map_v;
        ++it;
      }
    }
    if (ok && pend.it >= 0) load_v();
    // Nothing is on its way to this CTA any more when it says so (cluster_arrive below).  Of what the products signal, the releases
    // of K and V are waited for above and not signalled behind the last loads, and the P V products before the last are waited for
    // here: the softmax warps do so only where they scale O.  (Waiting for the last releases too cost 0.5 to 1.1 us a launch.)
#pragma unroll 1
    for (int b = 0; b < kBufs && ok; ++b) {
      const int i = ring_last(it - 1, kBufs, b);
      if (i >= 0) ok = warp_wait(bar(T3_PV_DONE0 + b), ring_parity(i, kBufs), abort_flag, P.err, 603);
    }
    // given up: loads that are still in flight get a bounded chance to land before the CTA's memory goes away
    if (!ok && lane == 0) {
      auto land = [&](int first, int asked, int n) {
#pragma unroll 1
        for (int b = 0; b < n; ++b) {
          const int i = ring_last(asked, n, b);
          for (uint32_t w = 0; i >= 0 && w < 4096 && !mbar_try_wait(bar(first + b), ring_parity(i, n)); ++w) __nanosleep(64);
        }
      };
      if (rank == 0) {  // (of a pair, until the other CTA's share of the tile has landed there too)
        land(T3_Q_FULL0, sidx, 2);
        land(T3_K_FULL0, it, kStages);
        land(T3_V_FULL0, pend.it >= 0 ? pend.it : it, kStages);
      } else {  // its loads are counted in the first CTA, which may have given up before it asked for as many: a millisecond
        for (uint32_t w = 0; w < 4096; ++w) __nanosleep(256);
      }
    }
    __syncwarp();
  } else if (warp == kWarpPv || warp == kWarpQk) {
    // ========================================================================== MMA issuers
    // Two warps: one issues S = Q K^T, one O += P V, so that neither's waits hold up the other (one warp for both: 72.3 us
    // instead of 70).  What the tensor pipe would order by itself then - S of tile t+3 may overwrite its buffer only when P V of
    // tile t has read P from it - is the wait for that product's commit.  Of a pair, the first CTA's issue for both.
    if (rank == 0) {
      const bool lead = elect_one();
      const int n = plan->n_tiles;
      bool ok = true;
      if (warp == kWarpQk) {
        const uint64_t qd0[2] = {make_sdesc(sQ, 16, 1024), make_sdesc(sQ + 2 * kSubTileBytes, 16, 1024)};
        const uint64_t kd0 = make_sdesc(sK, 16, 1024);
        const int n_parts = plan->n_parts;
        int iq = 0, sq = 0;
        bool q_due = true;
        for (int p = 0; p < n_parts && ok; ++p) {
          const int np = plan->part[p].n, last = plan->part[p].stage & 256;
          for (int t = 0; t < np && ok; ++t, ++iq) {
            const int b = iq % kStages;
            if (q_due) ok = warp_wait(bar(T3_Q_FULL0 + sq), 0, abort_flag, P.err, 610);
            q_due = false;
            if (ok) ok = warp_wait(bar(T3_K_FULL0 + b), (iq / kStages) & 1, abort_flag, P.err, 611);
            const int b3 = iq % kBufs;  // S/P buffer: free once the P V product of tile iq-3 has read P from it
            if (ok && iq >= kBufs) ok = warp_wait(bar(T3_PV_DONE0 + b3), ((iq / kBufs) - 1) & 1, abort_flag, P.err, 614);
            if (!ok) break;
            tc_fence_after();
            const uint64_t qd = sq & 1 ? qd0[1] : qd0[0], kd = kd0 + (uint64_t)(b * kShare >> 4);
            if (lead) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
              const uint64_t qo = (uint64_t)(((ks >> 2) * kSubTileBytes + (ks & 3) * 32) >> 4);
              const uint64_t ko = (uint64_t)(((ks >> 2) * (kShare / 2) + (ks & 3) * 32) >> 4);
              mma_ss<kPair>(tmem + b3 * 128, qd + qo, kd + ko, idesc_qk, ks > 0);
            }
            tc_commit<kPair>(bar(T3_S_FULL0 + b3));
            if (iq + kStages < n) tc_commit<kPair>(bar(T3_K_EMPTY0 + b));
            }
            if (last && t == np - 1) {
              ++sq;
              q_due = true;
            }
            __syncwarp();
          }
        }
      } else {
        const uint64_t vd0 = make_sdesc(sV, kSubTileBytes, 1024);
        for (int ip = 0; ip < n && ok; ++ip) {
          const int b = ip % kStages, b3 = ip % kBufs;
          ok = warp_wait(bar(T3_V_FULL0 + b), (ip / kStages) & 1, abort_flag, P.err, 613);
          ok = ok && warp_wait(bar(T3_P_FULL0 + b3), (ip / kBufs) & 1, abort_flag, P.err, 612);
          if (!ok) break;
          tc_fence_after();
          const uint64_t vd = vd0 + (uint64_t)(b * kShare >> 4);
          if (lead) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks) {
            // A = P from TMEM, in the buffer's columns [0,64)
            mma_ts<kPair>(tO, tmem + b3 * 128 + 8 * ks, vd + (uint64_t)((ks * 2048) >> 4), idesc_pv, (ip > 0) || (ks > 0));
          }
          if (ip + kStages < n) tc_commit<kPair>(bar(T3_V_EMPTY0 + b));
          if (ip + 1 < n) tc_commit<kPair>(bar(T3_PV_DONE0 + b3));
          }
          __syncwarp();
        }
        // (without a product nobody waits for it, and it would arrive in the other CTA when that one may be gone)
        if (ok && n > 0 && lead) tc_commit<kPair>(bar(T3_O_FULL));
      }
    }
  } else if (warp < 8) {
    // ===================================================================== softmax / epilogue
    // Two teams of four warps take the key tiles in turn: a thread has a query row (its TMEM lane) and all 128 keys of
    // it, so that nothing is exchanged within a row.  What one team waits for - scores from TMEM, the maximum, the way
    // of P into TMEM - is covered by the other's exponentials.  There is one O and so one reference maximum per row; it follows
    // from the tiles' maxima, in order, and every thread works it out for itself from those of its own tiles and those that
    // the other team leaves in shared memory (tmax).
    const int quad = warp & 3, team = warp >> 2, row = quad * 32 + lane;
    const uint32_t lane_base = ((uint32_t)(quad * 32)) << 16;
    const int64_t qi = i0 + row;
    const bool row_valid = qi < P.lq;
    const uint32_t p_full = lead_bar(T3_P_FULL0);
    float m_ref = -INFINITY, l_part = 0.f;  // the reference behind this team's last tile, and its sum relative to it
    int it0 = 0, stage = -1;
    bool ok = true;
    int jlo = 0, jhi = 0, wlo = 0, whi = 0;  // keys of the stage visible to this thread's query row, and to all rows of the warp
    const int n_parts = plan->n_parts, n_tiles = plan->n_tiles;
    for (int p = 0; p < n_parts && ok; ++p) {
      const Part R = plan->part[p];
      if ((R.stage & 255) != stage) {
        stage = R.stage & 255;
        const TcStage& S = P.stage[stage];
        auto clamp = [](int64_t v) { return (int)(v < -(1 << 30) ? -(1 << 30) : v > (1 << 30) ? (1 << 30) : v); };
        int64_t lo = 0, hi = S.lk - 1;
        // rows past the last query are not masked, so that whole tiles stay whole: nothing of them is written
        if (row_valid && S.mask_mode == INFLLM_MASK_WINDOW) {
          lo = qi + S.mask_offset - S.mask_size + 1;
          hi = qi + S.mask_offset;
        } else if (row_valid && S.mask_mode == INFLLM_MASK_COMPLEMENT) {
          hi = qi + S.mask_offset - S.mask_size;
        }
        jlo = clamp(lo), jhi = clamp(hi);
        wlo = __reduce_max_sync(0xffffffffu, jlo), whi = __reduce_min_sync(0xffffffffu, jhi);
      }
      const int j_hi = jhi < R.lim ? jhi : R.lim, w_hi = whi < R.lim ? whi : R.lim;
      for (int t = (team + it0) & 1; t < R.n && ok; t += 2) {
        const int it = it0 + t, b3 = it % kBufs;
        const uint32_t tS = tmem + b3 * 128 + lane_base;
        ok = warp_wait(bar(T3_S_FULL0 + b3), (it / kBufs) & 1, abort_flag, P.err, 620);
        if (!ok) break;
        tc_fence_after();
        const int j0 = R.j + t * kTile;
        if (wlo > j0 || w_hi < j0 + kTile - 1) {
          const int c_lo = jlo - j0, c_hi = j_hi - j0;
          // a tile at an edge: what a row does not see is taken out of the scores where they are
#pragma unroll 1
          for (int c = 0; c < kTile; c += 32) {
            const int lo = c_lo - c, hi = c_hi - c;
            if (__all_sync(0xffffffffu, lo <= 0 && hi >= 31)) continue;
            uint32_t u[32];
            tmem_ld32(tS + c, u);
            tmem_wait_ld32(u);
#pragma unroll
            for (int i = 0; i < 32; ++i) u[i] = i >= lo && i <= hi ? u[i] : 0xff800000u;
            tmem_st32(tS + c, u);
          }
          tmem_wait_st();
        }
        float sa[32], mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        uint32_t* ua = reinterpret_cast<uint32_t*>(sa);
        {
          float b[32];
          uint32_t* ub = reinterpret_cast<uint32_t*>(b);
          tmem_ld32(tS + 32, ub);
          tmem_ld32(tS + 64, ua);
          tmem_wait_ld32(ub);
          tmem_wait_ld32(ua);
          max_chunk(b, mx);
          tmem_ld32(tS + 96, ub);
          max_chunk(sa, mx);
          tmem_ld32(tS, ua);
          tmem_wait_ld32(ub);
          tmem_wait_ld32(ua);
          max_chunk(b, mx);
          max_chunk(sa, mx);
        }
        const float m_tile = fmaxf(fmax3(mx[0], mx[1], mx[2]), mx[3]) * P.scale_log2;
        // What the other team left of the tile before, if it has.  The tile's number comes with the value, in one word, so that there
        // is nothing else to wait for (a barrier per tile and quarter of the rows, a load behind it and two votes: 400 cycles, now 230).
        const uint32_t there = tmax + (uint32_t)(((it - 1) & 3) * kTile + row) * 8;
        uint64_t left = look_word(there);
        float m_prev = it > 0 ? next_ref<kExact>(m_ref, __uint_as_float((uint32_t)left)) : m_ref, m_new = next_ref<kExact>(m_prev, m_tile), alpha = 1.f;
        bool resc = false;
        auto move_ref = [&]() {  // what the row's O and this team's sum are to be scaled by
          resc = __any_sync(0xffffffffu, m_new != m_prev && m_prev != -INFINITY) && it >= 1;
          alpha = m_prev == -INFINITY ? 1.f : ex2_approx(m_prev - m_new);
          if (m_new != m_ref) {
            l_part *= ex2_approx(m_ref - m_new);
            m_ref = m_new;
          }
        };
        // (lazy: nearly always the word is there and no reference moves, which one vote says)
        const bool there_is = it == 0 || (int)(left >> 32) == it - 1;
        if (!__all_sync(0xffffffffu, there_is && (kExact || m_new == m_ref))) {
          for (uint32_t w = 0; it > 0 && (int)(left >> 32) != it - 1; ++w) {
            if (*abort_flag || w >= kSpinLimit) {
              ok = false;
              break;
            }
            if (w > 64) __nanosleep(w > 4096 ? 256 : 32);
            left = look_word(there);
          }
          if (!ok && !*abort_flag) {
            *abort_flag = 1;
            record_error(P.err, kErrWaitTimeout, 621);
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (it > 0) m_prev = next_ref<kExact>(m_ref, __uint_as_float((uint32_t)left));
          m_new = next_ref<kExact>(m_prev, m_tile);
          if (!kExact) move_ref();
        }
        // (left behind the look at the other team's: a place is taken again four tiles later, by the same team, which by then has
        // seen the maximum of the tile before, and the other team left that one behind its own look at this place)
        leave_word(tmax + (uint32_t)((it & 3) * kTile + row) * 8, (uint64_t)(uint32_t)it << 32 | __float_as_uint(m_tile));
        if (kExact) move_ref();
        const float neg_m = m_new == -INFINITY ? 0.f : -m_new;
        float2 rs[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        // P, packed, takes the place of the scores that have been read: 16 columns for 32.  (Rolled: the fetch of code is what
        // unrolled loops wait for.)
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          float2 e[16];
          uint32_t pk[16];
          arg_chunk(sa, P.scale_log2, neg_m, e);
          tmem_ld32_if(c < 3, tS + 32 * c + 32, ua);
          exp_chunk<T, kExact>(e, rs, pk);
          tmem_st16(tS + 16 * c, pk);
          tmem_wait_ld32(ua);
        }
        const float2 r = fadd2(fadd2(rs[0], rs[1]), fadd2(rs[2], rs[3]));
        l_part += r.x + r.y;
        if (resc) {
          // O holds the products up to tile it-1: wait for the last of them, then scale this warp's 32 rows
          ok = warp_wait(bar(T3_PV_DONE0 + ((it - 1) % kBufs)), ((it - 1) / kBufs) & 1, abort_flag, P.err, 622);
          if (!ok) break;
          tc_fence_after();
          // kExact, where most tiles come here: all 128 columns at once (four rounds of 32, one behind the other, took 3 % more: 4096
          // queries by 8192 keys)
          constexpr int kRound = kExact ? 128 : 32;
          const float2 al = make_float2(alpha, alpha);
#pragma unroll 1
          for (int c0 = 0; c0 < 128; c0 += kRound) {
            uint32_t o[kRound];
#pragma unroll
            for (int c = 0; c < kRound; c += 32) tmem_ld32(tO + lane_base + c0 + c, o + c);
#pragma unroll
            for (int c = 0; c < kRound; c += 32) tmem_wait_ld32(o + c);
#pragma unroll
            for (int c = 0; c < kRound; c += 32) {
#pragma unroll
              for (int i = c; i < c + 32; i += 2) {
                const float2 x = fmul2(make_float2(__uint_as_float(o[i]), __uint_as_float(o[i + 1])), al);
                o[i] = __float_as_uint(x.x), o[i + 1] = __float_as_uint(x.y);
              }
              tmem_st32(tO + lane_base + c0 + c, o + c);
            }
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {  // per warp: arrivals on one word take turns
          if (kPair) mbar_arrive_cluster(p_full + 8u * (uint32_t)b3);
          else mbar_arrive(p_full + 8u * (uint32_t)b3);
        }
      }
      it0 += R.n;
    }
    // ---- epilogue: the teams' row sums come together; then every warp writes 64 output columns of
    // 32 rows
    xsum[team * kTile + row] = l_part;
    xmax[team * kTile + row] = m_ref;
    asm volatile("bar.sync 1, 256;" ::: "memory");
    const int half = team, col0 = half * 64;
    const uint32_t row_base = lane_base;
    const int it = n_tiles;
    const float m_row = it >= 1 ? xmax[((it - 1) & 1) * kTile + row] : -INFINITY;
    float l_sum = 0.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const float m = xmax[e * kTile + row], l = xsum[e * kTile + row];
      l_sum += m == m_row ? l : l * ex2_approx(m - m_row);
    }
    // Three ways out: a run of a split work item leaves its un-normalised partial; a stage of a multi-stage attention
    // leaves the state (acc, m, l); everything else is normalised.  A state that came in is folded in first.
    const int64_t srow = (int64_t)h * P.lq + qi;
    // (the polynomial leaves 2^-126 of a masked key: a row that saw no key has the sum 0 by its maximum)
    float ws = 1.f, wp = 0.f, m_out = m_row, l_out = it >= 1 && m_row != -INFINITY ? l_sum : 0.f;
    if (P.st_acc) {
      if (row_valid) {
        const float mp = P.st_m[srow], mm = fmaxf(mp, m_row), ms = mm == -INFINITY ? 0.f : mm;
        ws = exp2f(m_row - ms);
        wp = exp2f(mp - ms);
        l_out = ws * l_out + wp * P.st_l[srow];
        m_out = mm;
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");  // both halves of a row have read (m, l): they may be overwritten
    }
    if (ok && it >= 1) ok = warp_wait(bar(T3_O_FULL), 0, abort_flag, P.err, 624);
    // Nothing more is signalled to or from this CTA, and no data goes with the arrival: O_FULL has said that the products are done, and so
    // that the loads and probabilities that either CTA counted on the other's barriers have been taken; every S_FULL was waited for here, the
    // PV_DONEs and the releases that are signalled at all by the producer.  (The other CTA's arrival is waited for at the end.)
    if (kPair) cluster_arrive();
    if (ok) {
      tc_fence_after();
      const bool raw = P.part_acc != nullptr;
      const int64_t prow = (int64_t)split * P.n_heads * P.lq + srow;
      const float inv = l_out > 0.f ? 1.f / l_out : 0.f;
      // (loops that stay rolled: this runs once, and what it waits for is its instructions)
      if (!P.st_acc && (!raw || rows_q <= 64)) {
        T* orow = raw ? nullptr : (T*)P.out + (int64_t)h * P.o_hs + qi * P.o_ts + col0;
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t o[32];
          if (it >= 1) {
            tmem_ld32(tO + row_base + col0 + c, o);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = 0;
          }
          if (row_valid && raw) {
            uint4* ap = reinterpret_cast<uint4*>(P.part_acc + prow * 128 + col0 + c);
#pragma unroll
            for (int k = 0; k < 32; k += 4) ap[k >> 2] = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
          } else if (row_valid) {
#pragma unroll
            for (int k = 0; k < 32; k += 8) {
              uint4 v;
              uint32_t* pv = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                typename Act<T>::T2 v2 = Act<T>::from_f2(__uint_as_float(o[k + 2 * e]) * inv, __uint_as_float(o[k + 2 * e + 1]) * inv);
                pv[e] = *reinterpret_cast<uint32_t*>(&v2);
              }
              *reinterpret_cast<uint4*>(orow + c + k) = v;
            }
          }
        }
      } else if (i0 + quad * 32 < P.lq) {
        // fp32 in or out, for more than a few rows: the warp's 32 rows by 64 columns go through shared memory (the operand buffers, which nothing reads
        // any more), so that half a warp has 64 columns of a row and touches every 32-byte sector once
        constexpr int kPitch = 68;  // floats; 16-byte pieces of eight neighbouring rows are in 32 different banks
        float* stage = reinterpret_cast<float*>(smem) + warp * 32 * kPitch;
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t o[32];
          if (it >= 1) {
            tmem_ld32(tO + row_base + col0 + c, o);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) o[k] = 0;
          }
          uint4* w = reinterpret_cast<uint4*>(stage + lane * kPitch + c);
#pragma unroll
          for (int k = 0; k < 32; k += 4) w[k >> 2] = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
        }
        __syncwarp();
        const int cl = (lane & 15) * 4;
        const int64_t row0 = i0 + quad * 32, srow0 = (int64_t)h * P.lq + row0, prow0 = (int64_t)split * P.n_heads * P.lq + srow0;
        const float nrm = raw ? 1.f : inv;
        // (a round's loads before its first store, rows past the last query with the last one's; one row after the other took 0.4 us
        // more of 15 for 128 queries in four runs)
        const int n_rows = (int)((P.lq - row0) < 32 ? P.lq - row0 : 32);
#pragma unroll 1
        for (int k0 = 0; k0 < 16; k0 += 8) {
          float4 v[8], x[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int rr = 2 * (k0 + k) + (lane >> 4), ra = rr < n_rows ? rr : n_rows - 1;
            v[k] = *reinterpret_cast<const float4*>(stage + rr * kPitch + cl);
            if (P.st_acc) x[k] = *reinterpret_cast<const float4*>(P.st_acc + (srow0 + ra) * 128 + col0 + cl);
          }
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int rr = 2 * (k0 + k) + (lane >> 4);
            const float f = __shfl_sync(0xffffffffu, ws * nrm, rr), fp = __shfl_sync(0xffffffffu, wp * nrm, rr);
            v[k] = make_float4(v[k].x * f, v[k].y * f, v[k].z * f, v[k].w * f);
            if (P.st_acc) v[k] = make_float4(fmaf(fp, x[k].x, v[k].x), fmaf(fp, x[k].y, v[k].y), fmaf(fp, x[k].z, v[k].z), fmaf(fp, x[k].w, v[k].w));
            if (rr >= n_rows) continue;
            if (raw) {
              *reinterpret_cast<float4*>(P.part_acc + (prow0 + rr) * 128 + col0 + cl) = v[k];
            } else {
              typename Act<T>::T2 v01 = Act<T>::from_f2(v[k].x, v[k].y), v23 = Act<T>::from_f2(v[k].z, v[k].w);
              *reinterpret_cast<uint2*>((T*)P.out + (int64_t)h * P.o_hs + (row0 + rr) * P.o_ts + col0 + cl) =
                  make_uint2(*reinterpret_cast<uint32_t*>(&v01), *reinterpret_cast<uint32_t*>(&v23));
            }
          }
        }
      }
      if (half == 0 && row_valid) {
        if (raw) {
          P.part_m[prow] = m_out;
          P.part_l[prow] = l_out;
        } else if (P.lse) {
          P.lse[srow] = l_out > 0.f ? m_out + log2f(l_out) : -INFINITY;
        }
      }
    }
  }
  if (kPair && warp >= 8) cluster_arrive();
  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (kPair) cluster_wait();  // nothing is signalled in a CTA that has gone
  if (warp == kWarpPv) tmem_dealloc<kPair>(tmem, 512);
}

// Merge of n_split partials (acc, m, l) per row, and of a state that came in (st_*, may be null): the sum of
// acc_s 2^(m_s - m), normalised into out / lse, or, when out is null, left as the new state (which may overwrite the
// old one in place).  l == null: the partials are normalised and m is their log-sum-exp.  One warp per row.
template <typename T>
__global__ void attn_tc_combine_kernel(const float* __restrict__ acc, const float* __restrict__ m,
                                       const float* __restrict__ l, int n_split, int n_heads, int64_t lq,
                                       T* __restrict__ out, int64_t o_hs, int64_t o_ts, float* __restrict__ lse,
                                       const float* st_acc, const float* st_m, const float* st_l, float* new_acc,
                                       float* new_m, float* new_l) {
  chain_enter();
  const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);  // h * lq + i
  if (row >= (int64_t)n_heads * lq) return;
  const int lane = threadIdx.x & 31;
  const int64_t h = row / lq, i = row - h * lq;
  const int64_t stride = (int64_t)n_heads * lq;
  // What bounds it is two loads behind one another and the launch: the first four partials are asked for whole, before their maximum is
  // known (with the attention, 256 queries of 28/4 heads in two runs 31.2 us, behind the maximum 32.5; 37 of 32/8 in four 22.6, 23.2; 16
  // of 16/2 in four 9.2, 10.0; 128 of 32/8 in four no difference)
  constexpr int kAhead = 4;
  float4 pa[kAhead];
  float pm[kAhead], pl[kAhead];
#pragma unroll
  for (int s = 0; s < kAhead; ++s) {
    if (s >= n_split) continue;
    pm[s] = m[s * stride + row], pl[s] = l ? l[s * stride + row] : 1.f;
    pa[s] = *reinterpret_cast<const float4*>(acc + (s * stride + row) * 128 + lane * 4);
  }
  float mx = st_acc ? st_m[row] : -INFINITY;
#pragma unroll
  for (int s = 0; s < kAhead; ++s)
    if (s < n_split) mx = fmaxf(mx, pm[s]);
  for (int s = kAhead; s < n_split; ++s) mx = fmaxf(mx, m[s * stride + row]);
  float den = 0.f;
  float4 num = make_float4(0.f, 0.f, 0.f, 0.f);
  if (mx != -INFINITY) {
    auto add = [&](float ms, float ls, float4 a) {
      if (ms == -INFINITY) return;
      const float w = exp2f(ms - mx);
      den = fmaf(w, ls, den);
      num.x = fmaf(w, a.x, num.x);
      num.y = fmaf(w, a.y, num.y);
      num.z = fmaf(w, a.z, num.z);
      num.w = fmaf(w, a.w, num.w);
    };
    auto fold = [&](float ms, float ls, const float* ap) { add(ms, ls, *reinterpret_cast<const float4*>(ap + row * 128 + lane * 4)); };
    if (st_acc) fold(st_m[row], st_l[row], st_acc);
#pragma unroll
    for (int s = 0; s < kAhead; ++s)
      if (s < n_split) add(pm[s], pl[s], pa[s]);
#pragma unroll 4
    for (int s = kAhead; s < n_split; ++s) fold(m[s * stride + row], l ? l[s * stride + row] : 1.f, acc + s * stride * 128);
  }
  if (out) {
    const float inv = den > 0.f ? 1.f / den : 0.f;
    typename Act<T>::T2 v01 = Act<T>::from_f2(num.x * inv, num.y * inv), v23 = Act<T>::from_f2(num.z * inv, num.w * inv);
    uint2 v = make_uint2(*reinterpret_cast<uint32_t*>(&v01), *reinterpret_cast<uint32_t*>(&v23));
    *reinterpret_cast<uint2*>(out + h * o_hs + i * o_ts + lane * 4) = v;
    if (lane == 0 && lse) lse[row] = den > 0.f ? mx + log2f(den) : -INFINITY;
  } else {
    __syncwarp();  // every lane has read the old state of this row
    *reinterpret_cast<float4*>(new_acc + row * 128 + lane * 4) = num;
    if (lane == 0) new_m[row] = mx, new_l[row] = den;
  }
}

// ------------------------------------------------------------------------------------ column sums
// One CTA owns one query head and a run of 128-key tiles.  The head's query tiles (at most four, 512 queries)
// and their log-sum-exps stay in shared memory for the whole CTA; the key tiles stream through a two-stage TMA
// ring; every (key tile, visible query tile) pair is one S^T = K Q^T into one of four TMEM buffers, and each buffer has
// four of the sixteen compute warps of its own, which turn it into sum_q exp2(s - lse_q).  A key tile is loaded once
// per head and a query tile once per CTA, which keeps the L2 traffic an order of magnitude below one load per pair.
// Bound: 16384 exponentials per pair, 768 cycles of the special-function unit with every fourth pair of them as a
// quartic on the FMA pipe (a quintic, kExact, for exec blocks of one query tile; without any 29.0 us, with an eighth 27.9, three
// eighths 27.0), the product, 514, whose operands want shared memory for all of that time, and 424 more there for the log-sum-exps
// (709 in 16-byte loads); a pair takes 1030.  512 queries x 32 heads over 4608 keys: 26.7 us (28.5 with those loads, a loop at
// every wait and sums cleared beforehand), 37 over 4133: 9.9 (10.7).
namespace colsum_smem {
constexpr int kQTiles = 4;                     // resident query tiles
constexpr int kMaxKeyTiles = 10;               // key tiles per CTA
constexpr int kBufs = 4;                       // TMEM accumulators in flight
constexpr int kIssuers = 2;                    // warps that issue products (a divisor of kBufs)
constexpr int kThreads = (16 + 1 + kIssuers) * 32;
constexpr int kQ = 0;
constexpr int kK = kQ + kQTiles * 2 * kSubTileBytes;   // two stages
constexpr int kLse = kK + 2 * 2 * kSubTileBytes;       // kQTiles x 128 fp32
constexpr int kBar = kLse + kQTiles * 512;
constexpr int kAcc = kBar + 256;               // [key tile][TMEM buffer][key] partial sums
constexpr int kTotal = kAcc + kMaxKeyTiles * 4 * 128 * 4;
}  // namespace colsum_smem

// Queries [lo, hi] that see key j, before clamping to [0, lq): with d = j - mask_offset a window gives
// [d, d + mask_size - 1], a complement [d + mask_size, lq - 1], no mask everything; P.lo_add / hi_add hold the
// constants (clamped to 2^30 on the host, so that 32-bit arithmetic is enough).
__device__ __forceinline__ void colsum_range(const ColsumTcParams& P, int j, int* lo, int* hi) {
  *lo = P.lo_add == kNoBound ? 0 : j + P.lo_add;
  *hi = P.hi_add == kNoBound ? (int)P.lq - 1 : j + P.hi_add;
}
// query tiles [tf, tl] that can see a key of the tile [j0, j0 + keys) (tl < tf: none)
__device__ __forceinline__ void colsum_q_tiles(const ColsumTcParams& P, int j0, int keys, int* tf, int* tl) {
  int lo, hi, x;
  colsum_range(P, j0, &lo, &x);
  colsum_range(P, j0 + keys - 1, &x, &hi);
  lo = lo < 0 ? 0 : lo;
  hi = hi > (int)P.lq - 1 ? (int)P.lq - 1 : hi;
  *tf = lo <= hi ? lo / kTile : 0;
  *tl = lo <= hi ? hi / kTile : -1;
}

// eight bytes of shared memory that all lanes ask for.  (Sixteen at a time took 2.99 million turns of the path into the registers
// for 512 queries x 32 heads over 4608 keys, these take 1.79, beside the operands of the products, which want all of it: 3 % less time)
__device__ __forceinline__ float2 lds8(const float* p) {
  float2 v;
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(smem_u32(p)));
  return v;
}

template <typename T, bool kExact>
__global__ void __launch_bounds__(colsum_smem::kThreads, 1) colsum_tc_kernel(const __grid_constant__ ColsumTcParams P) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t s_base = smem_u32(smem);
  const uint32_t sQ = s_base + colsum_smem::kQ, sK = s_base + colsum_smem::kK;
  float* s_lse = reinterpret_cast<float*>(smem + colsum_smem::kLse);
  float* s_acc = reinterpret_cast<float*>(smem + colsum_smem::kAcc);
  const uint32_t bars = s_base + colsum_smem::kBar;
  constexpr int NB = colsum_smem::kBufs;
  // barriers: k_full[2], k_free[2], s_full[NB], free[NB], q_full[query tile]
  constexpr int KF = 0, KE = 2, SF = 4, FR = 4 + NB, QF = 4 + 2 * NB, N_BARS = QF + colsum_smem::kQTiles;
  auto bar = [&](int i) { return bars + 8u * (uint32_t)i; };
  static_assert(N_BARS * 8 <= 144, "");
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + colsum_smem::kBar + 144);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + colsum_smem::kBar + 152);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int h = blockIdx.y, hkv = h / P.group;
  const int n_key_tiles = (int)((P.lk + kTile - 1) / kTile);
  const int kt0 = blockIdx.x * P.tiles_per_cta;
  const int kt1 = kt0 + P.tiles_per_cta < n_key_tiles ? kt0 + P.tiles_per_cta : n_key_tiles;
  // the query tiles any key tile of this CTA needs: from the first one's first to the last one's last (both only grow with
  // the key tile), of those that are seen at all
  int q_first = 1 << 30, q_last = -1;
  auto tile_q = [&](int kt, int* tf, int* tl) {
    const int j0 = kt * kTile;
    colsum_q_tiles(P, j0, (int)P.lk - j0 < kTile ? (int)P.lk - j0 : kTile, tf, tl);
    return *tl >= *tf;
  };
  for (int kt = kt0, tf, tl; kt < kt1; ++kt)
    if (tile_q(kt, &tf, &tl)) {
      q_first = tf;
      break;
    }
  for (int kt = kt1 - 1, tf, tl; kt >= kt0; --kt)
    if (tile_q(kt, &tf, &tl)) {
      q_last = tl;
      break;
    }
  const bool any = q_last >= q_first;
  auto load_q = [&](int t) {
    mbar_expect_tx(bar(QF + t), 2 * kSubTileBytes);
    tma_load_4d(sQ + t * 2 * kSubTileBytes, &P.map_q, bar(QF + t), 0, P.q_row0 + t * kTile, 0, h);
  };
  auto load_k = [&](int b, int j0) {
    mbar_expect_tx(bar(KF + b), 2 * kSubTileBytes);
    tma_load_4d(sK + b * 2 * kSubTileBytes, &P.map_k, bar(KF + b), 0, P.k_tok0 + j0, 0, hkv);
  };
  if (warp == 16 && lane == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(KF + i), 1);
      mbar_init(bar(KE + i), colsum_smem::kIssuers);
    }
    for (int i = 0; i < NB; ++i) {
      mbar_init(bar(SF + i), 1);
      mbar_init(bar(FR + i), 4);  // the warps of the group that reads the buffer
    }
    for (int i = 0; i < colsum_smem::kQTiles; ++i) mbar_init(bar(QF + i), 1);
    *abort_flag = 0;
    mbar_fence_init();
    if (!P.late_wait) chain_wait();
    // what the first products need is on its way while the CTA sets up; they run as soon as a query tile is there
    if (any) {
      int n = 0;
      for (int kt = kt0; kt < kt1 && n < 2; ++kt) {
        const int j0 = kt * kTile;
        const int keys = (int)P.lk - j0 < kTile ? (int)P.lk - j0 : kTile;
        int tf, tl;
        colsum_q_tiles(P, j0, keys, &tf, &tl);
        if (tl < tf) continue;
        if (n == 0) {
          load_q(tf);
          load_k(0, j0);
          for (int t = q_first; t <= q_last; ++t)
            if (t != tf) load_q(t);
        } else {
          load_k(1, j0);
        }
        ++n;
      }
    }
  }
  if (warp == 17) {
    tmem_alloc(smem_u32(tmem_slot), 128 * NB);
    tmem_relinquish();
  }
  if (!P.late_wait) chain_wait();
  // (past L1: with late_wait this grid may have been launched before the log-sum-exps were written)
  for (int i = threadIdx.x; i < colsum_smem::kQTiles * 128; i += blockDim.x)
    s_lse[i] = i < P.lq ? -__ldcg(P.lse + (int64_t)h * P.lq + i) : -INFINITY;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  constexpr bool kBf16 = !std::is_same<T, __half>::value;
  constexpr uint32_t idesc = make_idesc(kBf16, 128, 128, false);

  if (warp == 16) {
    // ==================================================== producer: the key tiles after the first two
    if (lane == 0 && any) {
      bool ok = true;
      int n = 0;  // key tiles with work, in order
      for (int kt = kt0; kt < kt1 && ok; ++kt) {
        const int j0 = kt * kTile;
        const int keys = (int)P.lk - j0 < kTile ? (int)P.lk - j0 : kTile;
        int tf, tl;
        colsum_q_tiles(P, j0, keys, &tf, &tl);
        if (tl < tf) continue;
        if (n >= 2) {
          ok = wait_or_abort(bar(KE + (n & 1)), ((n >> 1) - 1) & 1, abort_flag, P.err, 410);
          if (!ok) break;
          load_k(n & 1, j0);
        }
        ++n;
      }
      // loads that are still in flight get a bounded chance to land before the CTA's memory goes away, whoever gave up
      for (int b = 0; b < 2; ++b) {
        const int i = ring_last(n, 2, b);
        for (uint32_t w = 0; i >= 0 && w < 4096 && !mbar_try_wait(bar(KF + b), ring_parity(i, 2)); ++w) __nanosleep(64);
      }
      for (int t = q_first; t <= q_last; ++t)
        for (uint32_t w = 0; w < 4096 && !mbar_try_wait(bar(QF + t), 0); ++w) __nanosleep(64);
    }
  } else if (warp > 16) {
    // ====================================================================================== MMA issuers
    // Two warps take the products in turn, one lane of each issues (see attn_tc3_kernel); a thread of its own took 1385 cycles
    // for a product, of which the pipe is busy for 514.  A TMEM buffer always has the same issuer, which therefore never
    // gets a whole turn ahead of the buffer's phases.
    if (any) {
      const int me = warp - 17;
      const bool lead = elect_one();
      const uint64_t kd0 = make_sdesc(sK, 16, 1024), qd0 = make_sdesc(sQ, 16, 1024);
      bool ok = true;
      int n = 0, step = 0, q_there = 0;
      for (int kt = kt0; kt < kt1 && ok; ++kt) {
        const int j0 = kt * kTile;
        const int keys = (int)P.lk - j0 < kTile ? (int)P.lk - j0 : kTile;
        int tf, tl;
        colsum_q_tiles(P, j0, keys, &tf, &tl);
        if (tl < tf) continue;
        const int kb = n & 1;
        ok = warp_wait(bar(KF + kb), (n >> 1) & 1, abort_flag, P.err, 412);
        for (int t = tf; t <= tl && ok; ++t, ++step) {
          const int b = step % NB;
          if (b % colsum_smem::kIssuers != me) continue;
          if (!(q_there >> t & 1)) ok = warp_wait(bar(QF + t), 0, abort_flag, P.err, 411);
          q_there |= 1 << t;
          if (ok && step >= NB) ok = warp_wait(bar(FR + b), ((step / NB) - 1) & 1, abort_flag, P.err, 413);
          if (!ok) break;
          tc_fence_after();
          const uint64_t ad = kd0 + (uint64_t)(kb * 2 * kSubTileBytes >> 4), bd = qd0 + (uint64_t)(t * 2 * kSubTileBytes >> 4);
          if (lead) {
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
              // S^T = K Q^T: keys are the M rows (TMEM lanes), queries the N columns
              const uint64_t off = (uint64_t)(((ks >> 2) * kSubTileBytes + (ks & 3) * 32) >> 4);
              mma_ss(tmem + b * 128, ad + off, bd + off, idesc, ks > 0);
            }
            tc_commit(bar(SF + b));
          }
          __syncwarp();
        }
        if (ok && lead) tc_commit(bar(KE + kb));  // this warp's products with this key tile have been issued
        __syncwarp();
        ++n;
      }
    }
  } else {
    // ========================================================================================== compute
    // Group `part` of four warps takes every fourth product - TMEM buffer `part` - whole: a thread owns one key and all
    // 128 queries of it, in four loads of 32 columns (asking for the next columns ahead costs registers and gained nothing: the
    // other groups' warps fill the wait).
    const int quad = warp & 3, part = warp >> 2;
    const int krow = quad * 32 + lane;
    const uint32_t tS = tmem + part * 128 + (((uint32_t)(quad * 32)) << 16);
    bool ok = true;
    int step = 0;
    for (int kt = kt0; kt < kt1 && ok; ++kt) {
      const int j0 = kt * kTile;
      const int keys = (int)P.lk - j0 < kTile ? (int)P.lk - j0 : kTile;
      int tf, tl;
      colsum_q_tiles(P, j0, keys, &tf, &tl);
      if (tl < tf) {
        s_acc[((kt - kt0) * 4 + part) * 128 + krow] = 0.f;
        continue;
      }
      // queries [vi_lo, vi_hi] see this thread's key
      int vi_lo, vi_hi;
      colsum_range(P, j0 + krow, &vi_lo, &vi_hi);
      if (krow >= keys) vi_hi = -1;
      float total = 0.f;
      for (int t = tf; t <= tl && ok; ++t, ++step) {
        if ((step % NB) != part) continue;
        ok = warp_wait(bar(SF + part), (step / NB) & 1, abort_flag, P.err, 414);
        if (!ok) break;
        tc_fence_after();
        const int q_end = (int)P.lq - 1 - t * kTile, c_lo = vi_lo - t * kTile,
                  c_hi = vi_hi - t * kTile < q_end ? vi_hi - t * kTile : q_end;
        // a query row without any visible key has lse = -inf; it cannot see this key either, so it is masked
        const bool full = __all_sync(0xffffffffu, c_lo <= 0 && c_hi >= kTile - 1);
        const int last = q_end < kTile - 1 ? q_end >> 5 : 3;  // the last 32 columns with queries at all
        const float* ls = s_lse + t * kTile;
        const float2 sc2 = make_float2(P.scale_log2, P.scale_log2);
        float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll 1
        for (int cc = 0; cc <= last; ++cc) {
          float sc[32];
          tmem_ld32(tS + cc * 32, reinterpret_cast<uint32_t*>(sc));
          tmem_wait_ld();
          if (cc == last) {  // everything is in registers: the buffer can be overwritten
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(FR + part));
          }
          if (full || __all_sync(0xffffffffu, c_lo <= cc * 32 && c_hi >= cc * 32 + 31)) {
#pragma unroll
            for (int c = 0; c < 32; c += 4) {
              const float2 l01 = lds8(ls + cc * 32 + c), l23 = lds8(ls + cc * 32 + c + 2);  // negated
              const float2 a0 = ffma2(sc[c], sc[c + 1], sc2, l01);
              const float2 a1 = ffma2(sc[c + 2], sc[c + 3], sc2, l23);
              acc[0] = fadd2(acc[0], make_float2(ex2_approx(a0.x), ex2_approx(a0.y)));
              acc[1] = fadd2(acc[1], (c & 4) ? ex2_poly2<kExact ? 5 : 4>(a1) : make_float2(ex2_approx(a1.x), ex2_approx(a1.y)));
            }
          } else if (__any_sync(0xffffffffu, c_lo <= cc * 32 + 31 && c_hi >= cc * 32)) {
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              const float pv = ex2_approx(fmaf(sc[c], P.scale_log2, ls[cc * 32 + c]));
              if (cc * 32 + c >= c_lo && cc * 32 + c <= c_hi) acc[c & 1].x += pv;
            }
          }
        }
        total += (acc[0].x + acc[0].y) + (acc[1].x + acc[1].y);
      }
      // every thread owns one slot per key tile: no atomics, and the final sum below has a fixed order
      s_acc[((kt - kt0) * 4 + part) * 128 + krow] = total;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (!(*abort_flag)) {
    // every column in a thread of its own: one round of reads and writes
    const int cols = (int)((P.lk < (int64_t)kt1 * kTile ? P.lk : (int64_t)kt1 * kTile) - (int64_t)kt0 * kTile);
    float* dst = P.score + (int64_t)h * P.score_hs + (int64_t)kt0 * kTile;
    for (int i = threadIdx.x; i < cols; i += blockDim.x) {
      const float* sa = s_acc + (i >> 7) * NB * 128 + (i & 127);
      const float v = (sa[0] + sa[128]) + (sa[256] + sa[384]);
      dst[i] = P.accumulate ? __ldcg(dst + i) + v : v;
    }
  }
  if (P.late_wait) chain_wait();  // whoever follows this kernel follows the one before it too
  // (at the end: what comes next would hold SMs while it waits; from the start it cost a 64K MHA prompt 34.3 ms instead of 32.0)
  chain_trigger();
  if (warp == 17) tmem_dealloc(tmem, 128 * NB);
}

// ---------------------------------------------------------------------------------------- host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encoder() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int encode_tensor_map(CUtensorMap* map, int dtype, const void* base, int rank, const uint64_t* dims,
                      const uint64_t* strides_bytes, const uint32_t* box) {
  EncodeTiledFn enc = get_encoder();
  if (!enc) return fail(INFLLM_E_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  cuuint64_t gd[5], gs[4];
  cuuint32_t bx[5], es[5];
  for (int i = 0; i < rank; ++i) {
    gd[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
  }
  for (int i = 0; i < rank - 1; ++i) gs[i] = strides_bytes[i];
  CUresult r = enc(map, dtype == INFLLM_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16,
                   (cuuint32_t)rank, const_cast<void*>(base), gd, gs, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS)
    return fail(INFLLM_E_BADARG, "cuTensorMapEncodeTiled failed with code %d (rank %d, inner dim %llu)", (int)r, rank,
                (unsigned long long)dims[0]);
  return INFLLM_OK;
}

// rows of 128 elements as (64, rows, 2, heads): a box of `box_rows` rows and one or both halves of the dimensions lands as
// one or two 128-byte-swizzled tiles, one behind the other
int encode_rows_map(CUtensorMap* map, int dtype, const void* base, int64_t rows, int64_t heads, int64_t hs, int64_t ts, TcBox bx) {
  uint64_t dims[4] = {64, (uint64_t)rows, 2, (uint64_t)heads};
  uint64_t strides[3] = {(uint64_t)ts * 2, 128, (uint64_t)hs * 2};
  uint32_t box[4] = {64, bx.rows, bx.halves, 1};
  return encode_tensor_map(map, dtype, base, 4, dims, strides, box);
}

bool tc_rows_ok(const void* base, int64_t hs, int64_t ts) {
  return ((uintptr_t)base % 16) == 0 && (hs * 2) % 16 == 0 && (ts * 2) % 16 == 0 && hs > 0 && ts > 0;
}

int tc_get_error_ptr(int** p) {
  static int* cached[64] = {nullptr};  // per device ordinal
  int dev = 0;
  INFLLM_CUDA_OK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) return fail(INFLLM_E_UNSUPPORTED, "device ordinal %d", dev);
  if (!cached[dev]) {
    void* d = nullptr;
    INFLLM_CUDA_OK(cudaGetSymbolAddress(&d, g_tc_error));
    cached[dev] = (int*)d;
  }
  *p = cached[dev];
  return INFLLM_OK;
}

int attn_tc_combine_launch(const float* acc, const float* m, const float* l, int n_split, int n_heads, int64_t lq, void* out,
                           int64_t o_hs, int64_t o_ts, float* lse, const float* st_acc, const float* st_m,
                           const float* st_l, float* new_acc, float* new_m, float* new_l, int dtype, cudaStream_t s) {
  const int64_t rows = (int64_t)n_heads * lq;
  const int threads = rows >= 4096 ? 256 : 64;  // few rows: spread over the SMs
  INFLLM_DISPATCH_DTYPE(dtype, T, {
    INFLLM_CUDA_OK(launch_chained(attn_tc_combine_kernel<T>, dim3((unsigned)ceil_div(rows, threads / 32)), dim3(threads), 0, s, acc, m,
                                  l, n_split, n_heads, lq, (T*)out, o_hs, o_ts, lse, st_acc, st_m, st_l, new_acc, new_m, new_l));
  });
  INFLLM_LAUNCH_OK("attn_tc_combine_kernel");
  return INFLLM_OK;
}

// Runs of key tiles per (128-query tile, head), as many as the SMs take at once and no more than pay: a run's tiles come one
// after another, 0.8 us each, and the partials cost a merge, two tiles' time for its launch and one more for every 40 runs of the
// grid.  Measured over 4 to 60 tiles for 8 to 64 items (eight kinds of 8 sizes, bf16, both precisions, merge included, every
// count), three times: on the average 0.76 to 0.90 % above the best count, 9.3 % at worst (9 tiles of 8 items: 11.5 us in nine runs, 10.5
// in four; in one of the three 14 %, 4 tiles of 8 items).  Two and a half tiles for the merge: 0.80 to 0.94 %, 9.3 to 9.6 at worst; one
// and a half: 0.72 to 0.97, 9.3 to 14; three: 0.86 to 1.01; one more for every 32 runs 0.84 to 0.97, for every 50 1.05 to 1.31.
int attn_tc3_splits(int64_t lq, int n_heads, int64_t keys) {
  const int64_t items = ceil_div(lq, kTile) * n_heads, tiles = ceil_div(keys, kTile);
  int best = 1;
  for (int64_t n = 2, cost = 40 * tiles; n <= std::min<int64_t>(std::min<int64_t>(148 / items, tiles), 32); ++n) {
    const int64_t c = 40 * (ceil_div(tiles, n) + 2) + n * items;  // in fortieths of a tile
    if (c < cost) cost = c, best = (int)n;
  }
  return best;
}

bool attn_tc3_pairs(int64_t lq, int n_heads, int n_kv_heads) { return ceil_div(lq, kTile) * (n_heads / n_kv_heads) % 2 == 0; }

int attn_tc3_launch(const AttnTcParams& P, int dtype, cudaStream_t s) {
  if (P.lq <= 0) return INFLLM_OK;
  if (P.n_split < 1 || (P.n_split > 1 && (!P.part_acc || !P.part_m || !P.part_l || P.st_acc)))
    return fail(INFLLM_E_BADARG, "attn_tc3: split %d without partial buffers", P.n_split);
  const int items = (int)ceil_div(P.lq, kTile) * (P.n_heads / P.n_kv_heads);
  const bool pair = attn_tc3_pairs(P.lq, P.n_heads, P.n_kv_heads);
  const size_t smem = tc3::kTotal + 1024;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)items, P.n_kv_heads, P.n_split);
  cfg.blockDim = dim3(tc3::kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2, at[1].val.clusterDim.y = 1, at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = pair ? 2 : 1;
  INFLLM_DISPATCH_DTYPE(dtype, T, {
    auto kern = pair ? (P.exact ? attn_tc3_kernel<T, true, true> : attn_tc3_kernel<T, false, true>)
                     : (P.exact ? attn_tc3_kernel<T, true, false> : attn_tc3_kernel<T, false, false>);
    // the opt-in holds for the current device only, and a process may drive several: asked for at every launch
    INFLLM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    INFLLM_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, P));
  });
  INFLLM_LAUNCH_OK("attn_tc3_kernel");
  return INFLLM_OK;
}

int colsum_tc_launch_maps(const CUtensorMap& map_q, const CUtensorMap& map_k, int q_row0, int k_tok0, int n_heads,
                          int n_kv_heads, int64_t lq, int64_t lk, int mask_mode, int64_t mask_offset,
                          int64_t mask_size, const float* lse, float* score, int64_t score_hs, int accumulate,
                          bool late_wait, int dtype, cudaStream_t s) {
  if (lk > (1 << 29)) return fail(INFLLM_E_UNSUPPORTED, "colsum (tensor-core kernel): %lld keys", (long long)lk);
  if (lq > colsum_smem::kQTiles * kTile)
    return fail(INFLLM_E_UNSUPPORTED, "colsum (tensor-core kernel): %lld queries, at most %d", (long long)lq,
                colsum_smem::kQTiles * kTile);
  ColsumTcParams P{};
  P.map_q = map_q; P.map_k = map_k;
  P.q_row0 = q_row0; P.k_tok0 = k_tok0; P.n_heads = n_heads; P.group = n_heads / n_kv_heads;
  P.lq = lq; P.lk = lk; P.accumulate = accumulate; P.late_wait = late_wait;
  auto clamp = [](int64_t v) { return (int)std::max<int64_t>(-(1 << 30) + 1, std::min<int64_t>(1 << 30, v)); };
  P.lo_add = P.hi_add = kNoBound;
  if (mask_mode == INFLLM_MASK_WINDOW) P.lo_add = clamp(-mask_offset), P.hi_add = clamp(-mask_offset + mask_size - 1);
  if (mask_mode == INFLLM_MASK_COMPLEMENT) P.lo_add = clamp(-mask_offset + mask_size);
  P.lse = lse; P.score = score; P.score_hs = score_hs;
  P.scale_log2 = kLog2e / sqrtf(128.f);
  INFLLM_TRY(tc_get_error_ptr(&P.err));
  // one CTA per (head, run of key tiles): about one CTA per SM, never more than kMaxKeyTiles tiles each
  const int n_tiles = (int)ceil_div(lk, kTile);
  int chunks = std::max(1, 148 / n_heads);
  chunks = std::min(chunks, n_tiles);
  int per = (int)ceil_div(n_tiles, chunks);
  per = std::min(per, colsum_smem::kMaxKeyTiles);
  P.tiles_per_cta = per;
  dim3 grid((unsigned)ceil_div(n_tiles, per), n_heads);
  const size_t smem = colsum_smem::kTotal + 1024;
  INFLLM_DISPATCH_DTYPE(dtype, T, {
    auto kern = lq <= kExactQueries ? colsum_tc_kernel<T, true> : colsum_tc_kernel<T, false>;
    // the opt-in holds for the current device only, and a process may drive several: asked for at every launch
    INFLLM_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    INFLLM_CUDA_OK(launch_chained(kern, grid, dim3(colsum_smem::kThreads), smem, s, P));
  });
  INFLLM_LAUNCH_OK("colsum_tc_kernel");
  return INFLLM_OK;
}

int colsum_tc_launch(const void* q, int64_t q_hs, int64_t q_ts, const void* k, int64_t k_hs, int64_t k_ts, int n_heads,
                     int n_kv_heads, int64_t lq, int64_t lk, int mask_mode, int64_t mask_offset, int64_t mask_size,
                     const float* lse, float* score, int64_t score_hs, int accumulate, int dtype, cudaStream_t s) {
  CUtensorMap mq, mk;
  INFLLM_TRY(encode_rows_map(&mq, dtype, q, lq, n_heads, q_hs, q_ts, kBoxTile));
  INFLLM_TRY(encode_rows_map(&mk, dtype, k, lk, n_kv_heads, k_hs, k_ts, kBoxTile));
  return colsum_tc_launch_maps(mq, mk, 0, 0, n_heads, n_kv_heads, lq, lk, mask_mode, mask_offset, mask_size, lse, score,
                               score_hs, accumulate, false, dtype, s);
}

}  // namespace infllm

// Reads and clears the error record of the tensor-core kernels: code 0 = none, 1 = a bounded wait ran out.
// Synchronises the device.
extern "C" int infllm_device_error(int* code, int* where) {
  using namespace infllm;
  int h[4] = {0, 0, 0, 0};
  INFLLM_CUDA_OK(cudaDeviceSynchronize());
  INFLLM_CUDA_OK(cudaMemcpyFromSymbol(h, g_tc_error, sizeof(h)));
  if (h[0] != 0) {
    int z[4] = {0, 0, 0, 0};
    INFLLM_CUDA_OK(cudaMemcpyToSymbol(g_tc_error, z, sizeof(z)));
  }
  if (code) *code = h[0];
  if (where) *where = h[1];
  return INFLLM_OK;
}

extern "C" int infllm_device_error_set(int code, int where) {
  using namespace infllm;
  const int h[4] = {code, where, 0, 0};
  INFLLM_CUDA_OK(cudaDeviceSynchronize());
  INFLLM_CUDA_OK(cudaMemcpyToSymbol(g_tc_error, h, sizeof(h)));
  return INFLLM_OK;
}

