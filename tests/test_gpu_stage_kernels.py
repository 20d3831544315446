"""One stage of the multi-stage attention on each of its kernels (generic, split-K for one query, tcgen05 whole and cut
along the keys), with every way in and out of the running state, against fp32 torch.

Tolerance: probabilities and outputs are rounded to bf16 (2^-9 relative each); the inputs make rows of up to a few
thousand keys average N(0,1) values, so the error of an output is a few 2^-9 of its row's root mean square: 2e-2 of
the largest output covers it, 4e-3 in the 2-norm."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


def _want(stages):
    outs = []
    for q, k, v, win, comp in stages:
        h, hkv = q.shape[1], k.shape[1]
        q, k, v = q.float(), k.float().repeat_interleave(h // hkv, 1), v.float().repeat_interleave(h // hkv, 1)
        s = q @ k.transpose(-1, -2) / math.sqrt(D)
        if win is not None:
            off, size = (k.size(2) - q.size(2), win) if isinstance(win, int) else win
            dist = torch.arange(q.size(2), device=q.device)[:, None] - torch.arange(k.size(2), device=q.device)[None] + off
            keep = dist >= size if comp else (dist >= 0) & (dist < size)
            s = s.masked_fill(~keep, -math.inf)
        outs.append((s, v))
    p = torch.softmax(torch.cat([s for s, _ in outs], -1), -1).nan_to_num(0.0)
    return p @ torch.cat([v for _, v in outs], 2), p


@pytest.mark.parametrize("h,hkv", [(8, 2), (7, 1), (32, 8), (12, 12)])
@pytest.mark.parametrize("lq", [1, 2, 37, 128, 129, 300])
@pytest.mark.parametrize("lks", [(1, 1), (128, 129), (1000, 128), (17, 2500), (700, 0), (3001,)])
def test_stages_match_fp32(h, hkv, lq, lks):
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    g = torch.Generator(device="cuda").manual_seed(lq * 1000 + sum(lks))
    mk = lambda n, l: torch.randn((1, n, l, D), generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    stages = []
    for i, lk in enumerate(lks):
        win = None if i else max(1, (lk * 3) // 5)
        if i == 1 and lk > 200:
            stages.append((mk(h, lq), mk(hkv, lk), mk(hkv, lk), (lk - lq // 2, 100), True))
        else:
            stages.append((mk(h, lq), mk(hkv, lk), mk(hkv, lk), win, False))
    att = get_multi_stage_dot_production_attention(True)[0](stages[0][0].shape, torch.bfloat16, "cuda")
    for i, (q, k, v, win, comp) in enumerate(stages):
        att.append(q, k, v, sliding_window=win, complement_sliding_window=comp, end=i == len(stages) - 1, get_score=i == 0)
    got, scores = att.get_result()
    want, p = _want(stages)
    err = (got.float() - want).abs()
    assert err.max() <= 2e-2 * want.abs().max()
    assert err.norm() <= 4e-3 * want.norm() + 1e-6
    torch.testing.assert_close(att.score_list_fp32[0], p[..., :lks[0]].sum(2), rtol=1e-2, atol=1e-3)
