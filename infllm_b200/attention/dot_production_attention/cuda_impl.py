"""Multi-stage attention on the CUDA kernels of libinfllm_b200, with the interface of the
reference's MultiStageDotProductionAttention (dot_production_attention/base.py:3-30)."""
import torch

from ... import _lib


class CudaMultiStageDotProductionAttention:
    """append() any number of (q, k, v, mask) stages; the softmax is normalised jointly over all of
    them; get_result() returns (out (B, H, Lq, D) in q's dtype, [per-key score (B, H, Lk) or None]).

    Mirrors torch_impl.py:6-96 / triton_impl.py:488-556: `sliding_window` is None, an int w (meaning
    (Lk - Lq, w)) or (offset, size); with `complement_sliding_window` the kept pairs are
    dist >= size instead of 0 <= dist < size, dist = i - j + offset."""

    def __init__(self, q_shape, dtype, device):
        if len(q_shape) != 4:
            raise ValueError("q_shape must be (batch, heads, len_q, dim_head)")
        self.q_shape = tuple(q_shape)
        self.dtype = dtype
        self.device = torch.device(device)
        self._code = _lib.dtype_code(dtype)
        self._state = None  # (acc, m, l) between stages, fp32; a single stage needs none
        self._stages, self._scored = [], []
        self._first = True
        self.end = False
        self.ret = None
        self.score_list = []
        self.score_list_fp32 = []  # the same scores before rounding to the activation dtype

    def append(self, q, k, v, sliding_window=None, complement_sliding_window=False, end=False, get_score=False,
               *args, **kwargs):
        if self.end:
            raise RuntimeError("append after end=True")
        if tuple(q.shape) != self.q_shape:
            raise ValueError(f"q shape {tuple(q.shape)} != {self.q_shape}")
        for t, n in ((q, "q"), (k, "k"), (v, "v")):
            _lib.require_cuda(t, n)
            if t.dtype != self.dtype:
                raise TypeError(f"{n} dtype {t.dtype} != {self.dtype}")
        b, h, lq, d = self.q_shape
        hkv, lk = k.size(1), k.size(2)
        if lk and (k.size(0) < b or v.size(0) < b):  # (addresses are worked out below: nothing else would notice)
            raise IndexError(f"k and v have {k.size(0)} and {v.size(0)} batch elements, q has {b}")
        if sliding_window is None:
            mode, off, size = _lib.MASK_NONE, 0, 0
        else:
            if isinstance(sliding_window, int):
                sliding_window = (lk - lq, sliding_window)  # torch_impl.py:67-68
            off, size = int(sliding_window[0]), int(sliding_window[1])
            mode = _lib.MASK_COMPLEMENT if complement_sliding_window else _lib.MASK_WINDOW
        if q.stride(-1) != 1:
            q = q.contiguous()
        if k.stride(-1) != 1 or k.stride() != v.stride():
            k, v = k.contiguous(), v.contiguous()
        # (the strides of dimensions of one element are arbitrary, also behind contiguous())
        k_hs, k_ts = (k.stride(1) if hkv > 1 else max(lk, 1) * d), (k.stride(2) if lk > 1 else d)
        # addresses of a batch element's parts by arithmetic: a view of each cost 2 us, more than the whole launch
        stream = _lib.raw_stream(self.device)
        lib, f32 = _lib.lib, torch.float32
        if get_score:
            self._scored.append(len(self._stages))
        rows = h * lq
        if self._state is None and not end:
            self._state = torch.empty(b * rows * (d + 2), dtype=f32, device=self.device)
        lse_at = None
        if end:
            self.ret = torch.empty(self.q_shape, dtype=self.dtype, device=self.device)
            lse = torch.empty((b, h, lq), dtype=f32, device=self.device) if self._scored else None
            lse_at = lse.data_ptr() if lse is not None else None
        n_scratch = lib.infllm_attn_stage_scratch(h, hkv, lq, lk, d)
        scratch = torch.empty(n_scratch, dtype=f32, device=self.device) if n_scratch > 0 else None
        scratch_at = None if scratch is None else scratch.data_ptr()
        q_at, q_bs = q.data_ptr(), 2 * q.stride(0)
        k_at, v_at, k_bs = (k.data_ptr(), v.data_ptr(), 2 * k.stride(0)) if lk else (None, None, 0)
        acc = m = l = o_at = None
        if self._state is not None:
            acc = self._state.data_ptr()
            m = acc + 4 * b * rows * d
            l = m + 4 * b * rows
        if end:
            o_at = self.ret.data_ptr()
        for bi in range(b):
            rc = lib.infllm_attn_stage_ex(
                q_at, q.stride(1), q.stride(2), k_at, k_hs, k_ts, v_at, k_hs, k_ts, h, hkv, lq, lk, d, mode, off, size,
                acc, m, l, int(self._first), scratch_at, n_scratch, o_at, lq * d if end else 0, d if end else 0, lse_at,
                self._code, stream)
            if rc:
                _lib.check(rc)
            if bi + 1 < b:
                q_at += q_bs
                if lk:
                    k_at, v_at = k_at + k_bs, v_at + k_bs
                if acc is not None:
                    acc, m, l = acc + 4 * rows * d, m + 4 * rows, l + 4 * rows
                if end:
                    o_at += 2 * rows * d
                if lse_at is not None:
                    lse_at += 4 * rows
        self._first = False
        self._stages.append((q, k, k_hs, k_ts, mode, off, size) if get_score else None)
        if end:
            self._finalize(lse)

    def _finalize(self, lse):
        """The per-key scores of the stages that asked for them, from the final log-sum-exp of every row."""
        self.end = True
        b, h, lq, d = self.q_shape
        stream = _lib.raw_stream(self.device)
        for st in self._stages:
            if st is None:
                self.score_list.append(None)
                self.score_list_fp32.append(None)
                continue
            q, k, k_hs, k_ts, mode, off, size = st
            lk, hkv = k.size(2), k.size(1)
            # every column is written, unless there is nothing to sum
            score = (torch.empty if lq and lk else torch.zeros)((b, h, lk), dtype=torch.float32, device=self.device)
            q_at, lse_at, score_at = q.data_ptr(), lse.data_ptr(), score.data_ptr()
            k_at = k.data_ptr() if lk else None
            for bi in range(b):
                rc = _lib.lib.infllm_attn_colsum(
                    q_at + 2 * bi * q.stride(0), q.stride(1), q.stride(2), k_at + 2 * bi * k.stride(0) if lk else None, k_hs, k_ts,
                    h, hkv, lq, lk, d, mode, off, size, lse_at + 4 * bi * h * lq, score_at + 4 * bi * h * lk, lk, 0, self._code,
                    stream)
                if rc:
                    _lib.check(rc)
            self.score_list_fp32.append(score)
            self.score_list.append(score.to(self.dtype))
        self._stages = []

    def get_result(self):
        return self.ret, self.score_list
