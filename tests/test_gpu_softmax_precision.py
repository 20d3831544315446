"""Precision of the tcgen05 attention's probabilities where it stands for the shape-generic kernel: exponentials as exact
as exp2f, and the largest of a row without a rounding."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
D = 128


def _softmax(parts, values):
    """fp64 attention of the jointly normalised logits `parts` (H, L, K) over `values` (H, K, D): weights, outputs."""
    p = torch.softmax(torch.cat(parts, -1), -1)
    return p, p @ torch.cat(values, 1)


def _logits(q, k, group):
    return q.double() @ k.double().repeat_interleave(group, 0).transpose(1, 2) / math.sqrt(D)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("lq,lk", [(37, 4133), (64, 1000), (300, 777)])
def test_row_sums_are_exact_to_fp32(dtype, lq, lk):
    """The key scores are fp32 throughout and every one of them is divided by a row sum.  Exponentials within 2e-7 (that is
    what ex2.approx allows as well), sums over up to 4000 of them and products in fp32: 4e-7; the measured norm of the
    error is 1.0e-6 with exponentials that are good to 7.5e-5, 1.2e-7 with exp2f."""
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    g = torch.Generator(device="cuda").manual_seed(lq)
    q, k, v = (torch.randn((1, h, n, D), generator=g, device="cuda").to(dtype) for h, n in ((8, lq), (2, lk), (2, lk)))
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, q.device)
    att.append(q, k, v, end=True, get_score=True)
    p, _ = _softmax([_logits(q[0], k[0], 4)], [v[0].double().repeat_interleave(4, 0)])
    want = p.sum(1)
    assert ((att.score_list_fp32[0][0].double() - want).norm() / want.norm()).item() <= 4e-7


def _check_the_largest(out, z, others, v, some):
    """out (H, L, D): one key of log2-domain logit z (H, L) > 0 and value v (H, D) among `others` (L,) keys of logit and
    value 0.  It is the largest of its row, its probability relative to the maximum is 1 and has no rounding; what is left
    is that of the output, half a unit in the last place, and fp32 sums."""
    mant, low = (7, -126) if out.dtype == torch.bfloat16 else (10, -14)
    want = (torch.exp2(z) / (torch.exp2(z) + others))[..., None] * v.double()[:, None]
    ulp = torch.exp2(torch.floor(torch.log2(want.abs().clamp(min=2.0 ** low))) - mant)
    rows = z > 0.01
    assert rows.sum() >= some
    off = ((out.double() - want).abs() / ulp)[rows]
    assert off.max().item() <= 0.502


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("where", ["stage", "stream-llm", "memory"])
def test_the_largest_probability_is_exact(where, dtype):
    from infllm_b200.attention import (ATTN_FORWRAD, ContextManager, RotaryEmbeddingESM, get_multi_stage_dot_production_attention)

    H, HKV, G = 8, 2, 4
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)  # noqa: E731
    rope = RotaryEmbeddingESM(D, 1e6, 1.0)
    key, val = 2 * rnd(HKV, 1, D), rnd(HKV, 1, D)
    log2e = 1 / math.log(2)
    if where == "stage":
        lq, lk, at = 300, 700, 450
        q, k, v = rnd(1, H, lq, D), torch.zeros(1, HKV, lk, D, device="cuda", dtype=dtype), torch.zeros(1, HKV, lk, D, device="cuda", dtype=dtype)
        k[0, :, at], v[0, :, at] = key[:, 0], val[:, 0]
        att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, q.device)
        att.append(q, k, v, end=True)
        out, z = att.get_result()[0][0], _logits(q[0], key, G)[..., 0] * log2e
        others = torch.full((lq,), lk - 1.0, device="cuda", dtype=torch.float64)
        _check_the_largest(out, z, others, val[:, 0].repeat_interleave(G, 0), 200)
    elif where == "stream-llm":
        n, at, n_local, n_init = 600, 300, 512, 4
        x = torch.zeros(1, n, (H + 2 * HKV) * D, device="cuda", dtype=dtype)
        q = rnd(1, H, n, D)
        x[..., :H * D] = q[0].transpose(0, 1).reshape(n, -1)
        x[0, at, H * D:] = torch.cat((key, val)).reshape(-1)
        forward = ATTN_FORWRAD[where](n_local=n_local, n_init=n_init, fattn=True)
        proj = (lambda t: t[..., :H * D], lambda t: t[..., H * D:(H + HKV) * D], lambda t: t[..., (H + HKV) * D:], lambda o: o)
        out = forward(None, x, x, rope, False, None, *proj, D, H, HKV)[0].view(n, H, D).transpose(0, 1)
        kk = torch.zeros(1, HKV, n, D, device="cuda", dtype=dtype)
        kk[0, :, at] = key[:, 0]
        qr, kr = rope(q, kk)
        z = _logits(qr[0], kr[0, :, at:at + 1], G)[..., 0] * log2e
        i = torch.arange(n, device="cuda")
        others = (i + 1).clamp(max=n_local) + (i - n_local + 1).clamp(0, n_init) - 1.0
        _check_the_largest(out[:, at:], z[:, at:], others[at:].double(), val[:, 0].repeat_interleave(G, 0), 200)
    else:
        n_local, n_init, units, L, at = 512, 64, 3, 40, 400
        zero = lambda *s: torch.zeros(s, dtype=dtype)  # noqa: E731
        cm = ContextManager(rope, n_init, n_local, 128, 8, 4, 256, None, True, 2)
        wk, wv = zero(HKV, n_local, D), zero(HKV, n_local, D)
        wk[:, at], wv[:, at] = key[:, 0].cpu(), val[:, 0].cpu()
        cm.load_synthetic(zero(units, 2, HKV, 128, D), zero(units, H * D), zero(HKV, n_init, D), zero(HKV, n_init, D), wk, wv)
        q, k = rnd(1, H, L, D), torch.zeros(1, HKV, L, D, device="cuda", dtype=dtype)
        out = cm.append(q, k, k, q, k, k)[0]
        qr, kr = rope(q, torch.cat((wk.cuda()[None], k), 2))
        z = _logits(qr[0], kr[0, :, at:at + 1], G)[..., 0] * log2e
        others = torch.full((L,), n_local + units * 128 + n_init + L - 1.0, device="cuda", dtype=torch.float64)
        _check_the_largest(out, z, others, val[:, 0].repeat_interleave(G, 0), 50)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_a_nan_is_seen(dtype):
    """A NaN in one key reaches every query that sees it, whatever the key's place in a tile; one in a query reaches the
    scores of the keys that it sees."""
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    H, HKV, lq, lk = 4, 2, 160, 300
    g = torch.Generator(device="cuda").manual_seed(4)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(dtype)  # noqa: E731
    q, k, v = rnd(1, H, lq, D), rnd(1, HKV, lk, D), rnd(1, HKV, lk, D)

    def run(q, k):
        att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, q.device)
        att.append(q, k, v, end=True, sliding_window=200, get_score=True)
        out, score = att.get_result()
        return out[0], score[0][0]

    for j in list(range(16)) + [lk - 1]:
        bad = k.clone()
        bad[0, 1, j, 5] = float("nan")
        out, _ = run(q, bad)
        i = torch.arange(lq, device="cuda") + lk - lq
        sees = (i >= j) & (i - j < 200)
        assert out[2:, sees].isnan().all() and not out[2:, ~sees].isnan().any() and not out[:2].isnan().any(), j
    for i in list(range(8)) + [lq - 1]:
        bad = q.clone()
        bad[0, 3, i, 7] = float("nan")
        _, score = run(bad, k)
        j = torch.arange(lk, device="cuda")
        d = i + lk - lq - j
        sees = (d >= 0) & (d < 200)
        assert score[3, sees].isnan().all() and not score[3, ~sees].isnan().any() and not score[:3].isnan().any(), i
