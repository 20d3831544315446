"""Evicted units stay in their slots until the slots are needed.  A memory of more units than there are slots, retrievals
that wander over all of them: every token's output is checked against fp32 attention over the units it retrieved
(bf16 rotations, probabilities and outputs: 2e-2 of the largest output), through tokens, a prefill and tokens again."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

H, D, UNIT, N_INIT, N_LOCAL, TOPK = 16, 128, 128, 64, 256, 16


def test_retrievals_that_outgrow_the_slots():
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    n_units = 640  # units of 1 MiB: 128 of them, eight times the cache, fit past its own slots
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    units, block_k = rnd(n_units, 2, H, UNIT, D), rnd(n_units, H * D)
    ik, iv, wk, wv = rnd(H, N_INIT, D), rnd(H, N_INIT, D), rnd(H, N_LOCAL, D), rnd(H, N_LOCAL, D)
    rope = RotaryEmbeddingESM(D, 1e4, 1.0)
    cm = ContextManager(rope, N_INIT, N_LOCAL, UNIT, TOPK, TOPK, 128, None, True, 2)
    cm.load_synthetic(*(t.cpu() for t in (units, block_k, ik, iv, wk, wv)))
    raw_k, raw_v = wk, wv  # everything behind the sealed units

    def token(check):
        nonlocal raw_k, raw_v
        q, k, v = rnd(1, H, 1, D), rnd(1, H, 1, D), rnd(1, H, 1, D)
        out = cm.append(q, k, v, q, k, v)[0, :, 0].float()
        raw_k, raw_v = torch.cat((raw_k, k[0]), 1), torch.cat((raw_v, v[0]), 1)
        if not check:
            return
        ids = cm.last_topk()[0]
        ql, kl = rope(q, raw_k[:, -N_LOCAL:][None])
        qg = rope.apply_rotary_pos_emb_one_angle(q, N_LOCAL)
        ov = raw_k.size(1) - N_LOCAL
        kg = torch.cat([units[b, 0] for b in ids] + [ik, raw_k[:, :ov]], 1).float()
        vg = torch.cat([units[b, 1] for b in ids] + [iv, raw_v[:, :ov]], 1).float()
        s = torch.cat((ql[0].float() @ kl[0].float().transpose(1, 2), qg[0].float() @ kg.transpose(1, 2)), -1) / math.sqrt(D)
        want = (torch.softmax(s, -1) @ torch.cat((raw_v[:, -N_LOCAL:].float(), vg), 1))[:, 0]
        assert (out - want).abs().max() <= 2e-2 * want.abs().max()

    for i in range(100):
        token(i % 3 == 2)
    seen = cm.info()
    assert seen["evictions"] > 800 and seen["num_cached"] == TOPK
    n = 20  # a short prefill: the staged copies and the slots set aside for tokens change hands
    q, k, v = rnd(1, H, n, D), rnd(1, H, n, D), rnd(1, H, n, D)
    cm.append(q, k, v, q, k, v)
    raw_k, raw_v = torch.cat((raw_k, k[0]), 1), torch.cat((raw_v, v[0]), 1)
    assert cm.info()["num_blocks"] == n_units
    for i in range(7):  # up to the last token before a sealing
        token(True)
    assert cm.info()["num_blocks"] == n_units
