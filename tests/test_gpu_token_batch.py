"""One-token calls of several sequences (or heads) share launches: against each sequence as a memory of its own, which has
the chip to itself.  The scores are summed in the same order, so the retrieved ids are equal, in order; outputs differ by
the order in which partial results are added (probabilities and outputs are rounded to 16 bits: a few 2^-9 relative)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

D, UNIT, N_INIT, TOPK = 128, 128, 20, 6


def _manager(n_local, perhead):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    return ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), N_INIT, n_local, UNIT, 2 * TOPK, TOPK, 64, None, True, 2, perhead=perhead)


@pytest.mark.parametrize("B,H,HKV,n_local,dtype,perhead", [
    (2, 32, 32, 257, torch.bfloat16, False),  # two share a launch: the smallest share of the SMs, two runs per KV head
    (3, 8, 2, 300, torch.float16, False),
    (5, 28, 4, 700, torch.bfloat16, False),   # the larger parameter block
    (9, 8, 1, 300, torch.bfloat16, False),    # one more than a launch takes
    (3, 48, 48, 200, torch.bfloat16, False),  # too many KV heads to share
    (2, 6, 2, 300, torch.bfloat16, True),     # every head its own unit, over two sequences
])
def test_sequences_together_equal_sequences_apart(B, H, HKV, n_local, dtype, perhead):
    from infllm_b200 import _lib

    together, apart = _manager(n_local, perhead), [_manager(n_local, perhead) for _ in range(B)]
    g = torch.Generator(device="cuda").manual_seed(B + H)
    rnd = lambda n: [torch.randn((B, h, n, D), generator=g, device="cuda").to(dtype) for h in (H, HKV, HKV)]  # noqa: E731

    q, k, v = rnd(n_local + N_INIT + 20 * UNIT + 5)
    together.append(q, k, v, q, k, v)
    for i, m in enumerate(apart):
        m.append(*(t[i:i + 1] for t in (q, k, v, q, k, v)))
    per = H if perhead else 1
    units = together.num_global_block
    launches = []
    for _ in range(UNIT + 3):  # past a sealing
        n0 = _lib.lib.infllm_launch_count()
        q, k, v = rnd(1)
        a = together.append(q, k, v, q, k, v)
        launches.append(_lib.lib.infllm_launch_count() - n0)
        b = torch.cat([m.append(*(t[i:i + 1] for t in (q, k, v, q, k, v))) for i, m in enumerate(apart)])
        assert (a.float() - b.float()).abs().max() <= 1e-2 * b.float().abs().max()
        if together.num_global_block == units:
            for u in range(B * per):
                assert together.last_topk(u) == apart[u // per].last_topk(u % per)
    assert together.num_global_block == units + 1
    # a launch takes as many as leave each of them two runs per KV head and a ranking CTA, eight at most
    room = max(1, min(8, torch.cuda.get_device_properties(0).multi_processor_count // (2 * (1 if perhead else HKV) + 1)))
    assert min(launches) == -(-B * per // room)
    for i, m in enumerate(apart):
        assert m.cached_blocks == together.cached_blocks[i * per:(i + 1) * per]
