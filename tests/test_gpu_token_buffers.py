"""Tokens that move to the front of their buffers between calls: the same prompt in one call and in many.  The exec blocks
coincide, so units, representative keys and retrievals do too; outputs are the same sums over the same tiles (equal up to
how the window's tiles are cut: 16-bit roundings of the probabilities)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,H,HKV,n_local,calls", [
    (128, 8, 2, 256, [704] * 14),    # several moves in place, after the buffers have grown once
    (64, 4, 4, 256, [704] * 14),     # rows of 128 bytes
    (128, 8, 1, 4096, [4992] * 4),   # a window as long as the slack
    (128, 28, 4, 300, [64] * 150),   # one exec block per call
    (128, 8, 1, 4000, [4096, 4096] + [128] * 70),  # short calls: the rows that are cleared are among those that move
    (128, 4, 1, 3000, [4096, 4032, 4096, 3968, 128]),  # calls that shrink: some of them are
])
def test_one_call_equals_many(D, H, HKV, n_local, calls):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    g = torch.Generator(device="cuda").manual_seed(D + len(calls))
    n = sum(calls)
    q, k, v = (torch.randn((1, h, n, D), generator=g, device="cuda").bfloat16() for h in (H, HKV, HKV))
    make = lambda: ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 20, n_local, 32, 16, 4, 64, None, True, 2)  # noqa: E731
    whole, parts = make(), make()
    want = whole.append(q, k, v, q, k, v)
    ids, got = [], []
    at = 0
    for call in calls:
        t = [x[:, :, at:at + call] for x in (q, k, v)]
        at += call
        got.append(parts.append(*t, *t))
        ids += parts.last_topk()
    got = torch.cat(got, dim=2)
    last = whole.last_topk()  # of the last native call at least
    differ = sum(a != b for a, b in zip(last[::-1], ids[::-1]))
    assert differ <= len(last) // 50  # near ties
    assert (whole.block_k_rows() != parts.block_k_rows()).any(1).float().mean() <= 0.02
    assert ((got.float() - want.float()).norm(dim=-1) > 1e-2 * want.float().norm(dim=-1)).float().mean() <= 0.02
