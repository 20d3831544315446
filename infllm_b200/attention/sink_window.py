"""The reference's two sink + window attention types on the CUDA kernels: "infinite-lm" (LM-Infinite,
inf_llm/attention/infinite_lm.py:6-100) and "stream-llm" (StreamingLLM, inf_llm/attention/stream_llm.py:6-111).

Both keep the first n_init tokens (the sink) and the last n_local tokens (the window).  A query attends to its
window with window-relative rotary positions, and to the sink tokens that have left its window with all queries at
one fixed position; the two parts are normalised jointly by the multi-stage attention (a window-masked stage and a
stage with the complement mask — the one caller of the boundary that uses a complement mask that actually hides
pairs).  They differ in the positions of the sink stage:

    infinite-lm   sink keys un-rotated, queries at position n_local - 1
    stream-llm    sink keys at positions 0..n_init-1, queries at position n_local + n_init - 1

Same factory and forward signatures as the reference; the cache object returned as past_key_value is the
reference's tuple (K of [sink | window], V, tokens seen).
"""
import ctypes

import torch

from .. import _lib
from .dot_production_attention import get_multi_stage_dot_production_attention
from .rope import RotaryEmbeddingESM


_NATIVE = (torch.bfloat16, torch.float16)


def _rows(t):
    """A projection (B, L, heads * 128) with 16-byte aligned rows, copied if it has others."""
    a, b, c = t.stride()
    return t if c == 1 and (a | b) % 8 == 0 and t.data_ptr() % 16 == 0 else t.contiguous()


def _cache_rows(t):
    a, b, c, d = t.stride()
    return d == 1 and (a | b | c) % 8 == 0 and t.data_ptr() % 16 == 0


def _run_native(rope, q, k, v, heads, kv, past, n_local, n_init, stream_positions, use_cache):
    """The call in libinfllm_b200 (infllm_sink_window_run) on the projections q (B, L, heads * 128) and k, v
    (B, L, kv * 128); returns (o (B, L, heads * 128), cache or None), or None where the general path is needed."""
    dim = 128
    batch, len_q, _ = q.shape
    q, k, v = _rows(q), _rows(k), _rows(v)
    if k.stride() != v.stride():
        k, v = k.contiguous(), v.contiguous()
    pk = pv = None
    past_len, seen = 0, len_q
    p_bs = p_hs = p_ts = 0
    if past is not None:
        pk, pv = past[0], past[1]
        if not _cache_rows(pk) or pk.stride() != pv.stride() or not _cache_rows(pv):
            pk, pv = pk.contiguous(), pv.contiguous()
        past_len = pk.size(2)
        seen += past[2]
        p_bs, p_hs, p_ts, _ = pk.stride()
    total = past_len + len_q
    head = rows = 0
    kept = ck_at = cv_at = None
    device, dtype = q.device, q.dtype
    if use_cache:  # everything while the history is short, then [first n_init | last n_local]
        short = seen <= n_local + n_init
        head = total if short else min(n_init, total)
        rows = total if short else head + min(n_local, total)
        if rows > total:  # the two parts of a short cache overlap
            return None
        kept = torch.empty((2, batch, kv, rows, dim), dtype=dtype, device=device)
        ck_at = kept.data_ptr()
        cv_at = ck_at + 2 * batch * kv * rows * dim
    cos, sin = rope._tables(max(min(total, len_q + n_local), n_local + n_init), device)
    q_bs, q_ts, _ = q.stride()
    k_bs, k_ts, _ = k.stride()
    q_at, k_at, v_at = q.data_ptr(), k.data_ptr(), v.data_ptr()
    pk_at, pv_at = (pk.data_ptr(), pv.data_ptr()) if past_len else (None, None)
    # fields in the order of the structure
    a = _lib.SinkWindow(
        q_at, k_at, v_at, pk_at, pv_at, ck_at, cv_at, None, None, cos.data_ptr(), sin.data_ptr(), dim, q_ts, dim, k_ts, p_hs,
        p_ts, dim, heads * dim, len_q, past_len, seen, head, rows, cos.size(0), 0, heads, kv, dim, n_local, n_init,
        1 if stream_positions else 0, _lib.dtype_code(dtype), 0)
    ref = ctypes.byref(a)
    lib = _lib.lib
    n = lib.infllm_sink_window_scratch(ref)
    # (allocations of their own: the output, or a view of it, may outlive the call by far, and the scratch is a thousand times
    # a token's output)
    out = torch.empty((batch, len_q, heads * dim), dtype=dtype, device=device)
    scratch = torch.empty(max(n, 16), dtype=torch.uint8, device=device)
    o_at, a.d_scratch = out.data_ptr(), scratch.data_ptr()
    a.scratch_bytes = n
    a.d_out = o_at
    stream = _lib.raw_stream(device)
    for i in range(batch):
        if i:  # 2 bytes per element
            a.d_q, a.d_k, a.d_v = q_at + 2 * i * q_bs, k_at + 2 * i * k_bs, v_at + 2 * i * k_bs
            a.d_out = o_at + 2 * i * len_q * heads * dim
            if past_len:
                a.d_past_k, a.d_past_v = pk_at + 2 * i * p_bs, pv_at + 2 * i * p_bs
            if use_cache:
                a.d_cache_k, a.d_cache_v = ck_at + 2 * i * kv * rows * dim, cv_at + 2 * i * kv * rows * dim
        rc = lib.infllm_sink_window_run(ref, stream)
        if rc:
            _lib.check(rc)
    return out, ((kept[0], kept[1], seen) if use_cache else None)


def _sink_window_forward(n_local, n_init, fattn, stream_positions):
    Attn, _ = get_multi_stage_dot_production_attention(fattn)

    def forward(self, query, key_value, position_bias, use_cache, past_key_value, project_q, project_k, project_v,
                attention_out, dim_head, num_heads, num_heads_kv):
        batch, len_q, len_new = query.size(0), query.size(1), key_value.size(1)

        def heads(x, n, length):  # (B, L, n*D) -> (B, n, L, D)
            return x.view(batch, length, n, dim_head).permute(0, 2, 1, 3)

        q, k, v = project_q(query), project_k(key_value), project_v(key_value)
        # The library does the whole call for the rotary embedding it knows; another one's rotations, other head
        # sizes and self-made caches are put together below from the attention class.
        if type(position_bias) is RotaryEmbeddingESM and position_bias.dim == dim_head == 128 and len_q == len_new and len_q > 0 \
                and q.is_cuda and q.dtype in _NATIVE and k.dtype == v.dtype == q.dtype and num_heads % num_heads_kv == 0 \
                and q.shape == (batch, len_q, num_heads * 128) and k.shape == v.shape == (batch, len_q, num_heads_kv * 128) \
                and (past_key_value is None or (
                    past_key_value[0].dtype == past_key_value[1].dtype == q.dtype and past_key_value[0].is_cuda
                    and past_key_value[0].shape == past_key_value[1].shape == (
                        batch, num_heads_kv, past_key_value[0].size(2), 128))):
            done = _run_native(position_bias, q, k, v, num_heads, num_heads_kv, past_key_value, n_local, n_init,
                               stream_positions, use_cache)
            if done is not None:
                o = attention_out(done[0])
                return (o, done[1]) if use_cache else o
        q, k, v = heads(q, num_heads, len_q), heads(k, num_heads_kv, len_new), heads(v, num_heads_kv, len_new)
        q, k, v = q.contiguous(), k.contiguous(), v.contiguous()
        seen = len_new
        if past_key_value is not None:
            k = torch.cat((past_key_value[0], k), dim=-2)
            v = torch.cat((past_key_value[1], v), dim=-2)
            seen += past_key_value[2]
        cache = None
        if use_cache:  # everything while the history is short, then [first n_init | last n_local]
            if seen <= n_local + n_init:
                cache = (k, v, seen)
            else:
                tail = max(0, k.size(-2) - n_local)
                cache = (torch.cat((k[:, :, :n_init], k[:, :, tail:]), dim=2),
                         torch.cat((v[:, :, :n_init], v[:, :, tail:]), dim=2), seen)
        # window stage over the last len_q + n_local keys
        wk, wv = k, v
        if len_q + n_local < k.size(-2):
            cut = k.size(-2) - len_q - n_local
            wk, wv = k[:, :, cut:].contiguous(), v[:, :, cut:].contiguous()
        wq, wk = position_bias(q, wk)
        # sink stage: only once some token has left the window
        if seen > n_local:
            sk, sv = k[:, :, :n_init].contiguous(), v[:, :, :n_init].contiguous()
            if stream_positions:
                sq = position_bias.apply_rotary_pos_emb_one_angle(q, n_local + n_init)
                sk = position_bias.apply_rotary_pos_emb(sk, sk.size(-2), sk.size(-2), None, None)
            else:
                sq = position_bias.apply_rotary_pos_emb_one_angle(q, n_local)
        else:
            sq = q
            sk = torch.empty((batch, num_heads_kv, 0, dim_head), device=k.device, dtype=k.dtype)
            sv = torch.empty_like(sk)
        attn = Attn(wq.shape, wq.dtype, wq.device)
        attn.append(wq, wk, wv, sliding_window=n_local)
        attn.append(sq, sk, sv, end=True, sliding_window=(seen - len_q, n_local), complement_sliding_window=True)
        o, _ = attn.get_result()
        o = o.view(batch, num_heads, len_q, dim_head).permute(0, 2, 1, 3).reshape(batch, len_q, num_heads * dim_head)
        o = attention_out(o)
        return (o, cache) if use_cache else o

    return forward


def infinite_lm_forward(n_local, n_init, fattn: bool = False, *args, **kwargs):
    """ATTN_FORWRAD["infinite-lm"] (inf_llm/attention/infinite_lm.py:6)."""
    return _sink_window_forward(n_local, n_init, fattn, stream_positions=False)


def stream_llm_forward(n_local, n_init, fattn: bool = False, *args, **kwargs):
    """ATTN_FORWRAD["stream-llm"] (inf_llm/attention/stream_llm.py:6)."""
    return _sink_window_forward(n_local, n_init, fattn, stream_positions=True)
