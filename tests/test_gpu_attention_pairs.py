"""The tcgen05 attention of exec blocks of more than one query tile, in pairs of CTAs and alone (a KV head's query tiles over all
its query heads come out even, or not), against the shape-generic kernel on the same memory.  Every unit is retrieved, so that
both see the same keys.

Tolerance: each kernel rounds probabilities and outputs to bf16; test_gpu_stage_kernels bounds that by 4e-3 in the 2-norm and
2e-2 of the largest output against fp32, two kernels differ by twice that."""
import pytest
import torch

pytestmark = pytest.mark.gpu

D, UNIT = 128, 128


@pytest.mark.parametrize("h,hkv,exec_,n", [
    (7, 1, 384, 2500),    # 21 tiles: alone
    (7, 1, 256, 2500),    # 14 tiles, the middle pair of two query tiles
    (12, 12, 384, 1900),  # 3 tiles of every head: alone
    (12, 12, 200, 1900),  # pairs of a whole and a ragged tile
    (8, 2, 129, 1500),    # a second tile of one query
    (32, 8, 512, 3000),   # pairs of heads
])
@pytest.mark.parametrize("step", [1.0, 4.0])  # keys that grow: the rows' reference maxima move in every tile
def test_pairs_and_lone_ctas_match_the_generic_kernel(monkeypatch, h, hkv, exec_, n, step):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM
    from infllm_b200.attention import context_manager as cmod

    g = torch.Generator(device="cuda").manual_seed(h * exec_)
    q, k, v = (torch.randn((1, m, n, D), generator=g, device="cuda") for m in (h, hkv, hkv))
    k = k * torch.linspace(1.0, step, n, device="cuda")[:, None]
    q, k, v = (x.to(torch.bfloat16) for x in (q, k, v))
    outs = []
    for flags in (0, 1):
        monkeypatch.setattr(cmod, "TEST_OVERRIDES", {"debug_flags": flags})
        cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 100, 600, UNIT, 32, 32, exec_, None, True, 2)
        outs.append(cm.append(q, k, v, q, k, v).float())
    err = (outs[0] - outs[1]).abs()
    assert err.norm() <= 8e-3 * outs[1].norm()
    assert err.max() <= 4e-2 * outs[1].abs().max()


@pytest.mark.parametrize("h,hkv,lq", [(8, 2, 256), (7, 1, 256), (12, 12, 200), (7, 1, 300)])  # pairs of heads, of tiles, ragged; alone
@pytest.mark.parametrize("hidden", [200, 3000])  # keys of the stage that no query sees: one run, and several
@pytest.mark.parametrize("order", ["before", "behind", "only"])
def test_a_stage_that_hides_every_pair_changes_nothing(h, hkv, lq, hidden, order):
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    g = torch.Generator(device="cuda").manual_seed(h * lq + hidden)
    q, k, v, hk, hv = (torch.randn((1, m, n, D), generator=g, device="cuda").to(torch.bfloat16)
                       for m, n in ((h, lq), (hkv, 500), (hkv, 500), (hkv, hidden), (hkv, hidden)))
    stages = [(k, v, 450, False)] * (order != "only")
    stages.insert(order == "behind", (hk, hv, (-10 ** 6, 100), order != "before"))
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cuda")
    for i, (sk, sv, win, comp) in enumerate(stages):
        att.append(q, sk, sv, sliding_window=win, complement_sliding_window=comp, end=i == len(stages) - 1)
    got = att.get_result()[0].float()
    if order == "only":
        assert not got.any()
        return
    s = q.float() @ k.float().repeat_interleave(h // hkv, 1).transpose(-1, -2) / D ** 0.5
    dist = torch.arange(lq, device="cuda")[:, None] - torch.arange(500, device="cuda")[None] + 500 - lq
    want = s.masked_fill((dist < 0) | (dist >= 450), float("-inf")).softmax(-1) @ v.float().repeat_interleave(h // hkv, 1)
    err = (got - want).abs()
    assert err.norm() <= 4e-3 * want.norm()  # (test_gpu_stage_kernels' bounds: one kernel against fp32)
    assert err.max() <= 2e-2 * want.abs().max()
