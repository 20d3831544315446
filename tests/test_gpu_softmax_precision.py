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
