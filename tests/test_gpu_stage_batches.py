"""A batch through the multi-stage attention class against its elements one at a time, with the per-key scores: the same kernels
on the same numbers, so bit for bit the same.  Operands are parts of larger buffers, in which a batch element's stride is not its
size."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,hkv", [(8, 2), (7, 1)])
@pytest.mark.parametrize("lq,lks", [(1, (300, 40)), (37, (200, 129)), (150, (700, 0)), (256, (600, 300)), (130, (512,))])
def test_batch_with_scores_is_its_elements(h, hkv, lq, lks):
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    b = 3
    g = torch.Generator(device="cuda").manual_seed(1000 * lq + h)

    def part(heads, n):  # (b, heads, n, 128) out of something longer in every dimension
        return torch.randn((b, heads + 1, n + 5, 128), generator=g, device="cuda").to(torch.bfloat16)[:, :heads, 2:2 + n]

    stages = [(part(h, lq), part(hkv, n), part(hkv, n)) for n in lks]

    def run(sl):
        att = get_multi_stage_dot_production_attention(True)[0]((len(range(b)[sl]), h, lq, 128), torch.bfloat16, "cuda")
        for i, (q, k, v) in enumerate(stages):
            att.append(q[sl], k[sl], v[sl], sliding_window=250 if i == 0 else None, end=i == len(stages) - 1, get_score=k.size(2) > 0)
        return att.get_result()[0], att.score_list_fp32

    out, scores = run(slice(None))
    for i in range(b):
        one, its = run(slice(i, i + 1))
        assert torch.equal(out[i:i + 1], one)
        for s, t in zip(scores, its):
            assert s is t is None or torch.equal(s[i:i + 1], t)
    assert not torch.equal(out[0], out[1])
