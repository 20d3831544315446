"""Units whose scores are NaN (a NaN in the keys that represent them) rank with -inf, wherever the ranking happens: on the
device for every exec block, or, with the look-ahead, on the host among the candidates."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("topk", [4, 16])
def test_look_ahead_and_device_rank_alike(monkeypatch, topk):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM
    from infllm_b200.attention import context_manager as cmod

    H, HKV, D, N_INIT, UNIT, n = 8, 2, 128, 64, 128, 64 + 256 + 60 * 128
    g = torch.Generator(device="cuda").manual_seed(topk)
    q, k, v = (torch.randn((1, h, n, D), generator=g, device="cuda").to(torch.bfloat16) for h in (H, HKV, HKV))
    # a NaN in a key makes the accumulated scores around it NaN, and a unit without any score is represented by its first
    # tokens: every third unit's is the NaN
    k[:, :, N_INIT::3 * UNIT, 3] = float("nan")
    ids = []
    for flags in (2, 0):  # no look-ahead: the device ranks; look-ahead: the host ranks
        monkeypatch.setattr(cmod, "TEST_OVERRIDES", {"debug_flags": flags})
        cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), N_INIT, 256, UNIT, topk, topk, 256, None, True, 2)
        cm.append(q, k, v, q, k, v)
        rows = cm.block_k_rows().isnan().any(1)
        assert 0 < rows.sum() < len(rows)
        ids.append(cm.last_topk())
    assert ids[0] == ids[1]
