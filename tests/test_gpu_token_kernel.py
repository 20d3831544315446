"""The one-launch decode token (token.cu) against the same tokens as separate kernels (which per-kernel timing asks
for): the scores are summed in the same order, so the retrieved ids are equal, in order; outputs differ by the order in
which partial results are added (probabilities and outputs are rounded to 16 bits: a few 2^-9 relative)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

D, UNIT, N_INIT = 128, 128, 40


def _memory(H, HKV, n_units, n_local, topk, dtype, ties):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    g = torch.Generator().manual_seed(n_units + H)
    pool = torch.randn((min(n_units, 64), 2, HKV, UNIT, D), generator=g).to(dtype)
    units = pool.repeat((-(-n_units // pool.size(0)), 1, 1, 1, 1))[:n_units]
    block_k = torch.randn((n_units, H * D), generator=g).to(dtype)
    if ties:  # every third row is the same: equal scores, also at the cut
        block_k[::3] = block_k[0]
    rnd = lambda n: torch.randn((HKV, n, D), generator=g).to(dtype)  # noqa: E731
    small = (rnd(N_INIT), rnd(N_INIT), rnd(n_local), rnd(n_local))
    out = []
    for apart in (False, True):
        cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), N_INIT, n_local, UNIT, 2 * topk, topk, 128, None, True, 2)
        cm.profile(apart)
        cm.load_synthetic(units, block_k, *small)
        out.append(cm)
    return out


@pytest.mark.parametrize("H,HKV,n_units,n_local,topk,dtype,ties", [
    (32, 8, 17, 1000, 16, torch.bfloat16, False),    # one unit more than a retrieval
    (32, 8, 384, 513, 16, torch.bfloat16, True),     # as many scores as ranking threads
    (32, 8, 385, 4096, 16, torch.float16, True),     # one more
    (28, 4, 500, 700, 64, torch.bfloat16, True),     # the largest retrieval
    (8, 1, 8460, 300, 32, torch.bfloat16, True),     # more scores than the ranking keeps in registers; one KV head
    (8, 1, 8460, 300, 1, torch.bfloat16, False),
    (32, 32, 300, 257, 8, torch.float16, False),     # one query head per KV head, four runs each
    (7, 7, 40, 130, 3, torch.bfloat16, False),       # a width that is no multiple of 2048
    (96, 48, 60, 200, 4, torch.bfloat16, False),     # the widest rows, three runs per KV head
])
def test_one_launch_equals_separate_kernels(H, HKV, n_units, n_local, topk, dtype, ties):
    one, apart = _memory(H, HKV, n_units, n_local, topk, dtype, ties)
    g = torch.Generator(device="cuda").manual_seed(5)
    for i in range(UNIT + 3):  # past a sealing
        q, k, v = (torch.randn((1, h, 1, D), generator=g, device="cuda").to(dtype) for h in (H, HKV, HKV))
        a, b = one.append(q, k, v, q, k, v), apart.append(q, k, v, q, k, v)
        if i % 16 == 0 or i > UNIT - 4:
            assert one.last_topk() == apart.last_topk()
            assert one.cached_blocks == apart.cached_blocks
            assert (a.float() - b.float()).abs().max() <= 1e-2 * b.float().abs().max()
    assert one.info()["num_blocks"] == n_units + 1
    assert torch.equal(one.block_k_rows()[:n_units], apart.block_k_rows()[:n_units])
    # the sealed unit's representative keys come from the accumulated scores: equal unless two tokens tie to 1e-6
    assert (one.block_k_rows()[n_units] != apart.block_k_rows()[n_units]).float().mean() < 0.05


def test_a_word_that_does_not_arrive_is_an_error():
    """The error record that a token's bounded wait leaves (set here from the host) fails the next call."""
    from infllm_b200 import _lib

    one, _ = _memory(8, 2, 20, 200, 4, torch.bfloat16, False)
    q, k, v = (torch.randn((1, h, 1, D), device="cuda").to(torch.bfloat16) for h in (8, 2, 2))
    one.append(q, k, v, q, k, v)
    torch.cuda.synchronize()
    _lib.check(_lib.lib.infllm_device_error_set(1, 700))
    with pytest.raises(_lib.InfLLMError):
        for n in (200, 1, 1):  # a longer call carries the record to the host
            qq, kk, vv = (torch.randn((1, h, n, D), device="cuda").to(torch.bfloat16) for h in (8, 2, 2))
            one.append(qq, kk, vv, qq, kk, vv)
            torch.cuda.synchronize()
    for _ in range(2):  # and the memory goes on
        one.append(q, k, v, q, k, v)
    torch.cuda.synchronize()


def test_a_token_that_gives_up_is_one_error(monkeypatch):
    """The waits inside the sixteenth token give up at once: one of the calls that follow reports it, promptly, and the
    memory goes on as one that never lost a retrieval (the token itself was ingested)."""
    import time

    from infllm_b200 import _lib
    from infllm_b200.attention import context_manager as cmod

    want, _ = _memory(8, 2, 60, 300, 4, torch.bfloat16, False)
    monkeypatch.setattr(cmod, "TEST_OVERRIDES", {"debug_flags": 128})
    got, _ = _memory(8, 2, 60, 300, 4, torch.bfloat16, False)
    g = torch.Generator(device="cuda").manual_seed(6)
    errors = 0
    for i in range(28):
        q, k, v = (torch.randn((1, h, 1, D), generator=g, device="cuda").to(torch.bfloat16) for h in (8, 2, 2))
        b = want.append(q, k, v, q, k, v)
        t0 = time.perf_counter()
        try:
            a = got.append(q, k, v, q, k, v)
        except _lib.InfLLMError:
            errors += 1
            a = got.append(q, k, v, q, k, v)
        if i == 17:
            assert errors == 1
        torch.cuda.synchronize()
        assert time.perf_counter() - t0 < 5
        if i != 15:  # the one that gave up
            assert torch.equal(a, b), i
            if i % 4 == 0:
                assert got.last_topk() == want.last_topk()
    assert errors == 1 and got.info()["length"] == want.info()["length"]


@pytest.mark.parametrize("batch", [1, 3])
def test_a_launch_that_is_refused_leaves_nothing_behind(monkeypatch, batch):
    """The sixteenth token's grid is larger than the device: the runtime refuses it, that token and those behind it are
    separate kernels, and what the refused launch should have told the table of unit addresses is not lost."""
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM
    from infllm_b200.attention import context_manager as cmod

    H, HKV, topk, n = 8, 2, 6, 20 + 30 * UNIT + 256
    make = lambda: ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 20, 256, UNIT, topk, topk, 128, None, True, 2)  # noqa: E731
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda n: [torch.randn((batch, h, n, D), generator=g, device="cuda").to(torch.bfloat16) for h in (H, HKV, HKV)]  # noqa: E731
    q, k, v = rnd(n)
    want = make()
    want.append(q, k, v, q, k, v)
    monkeypatch.setattr(cmod, "TEST_OVERRIDES", {"debug_flags": 64})
    got = make()
    got.append(q, k, v, q, k, v)
    for i in range(40):
        q, k, v = rnd(1)
        a, b = got.append(q, k, v, q, k, v), want.append(q, k, v, q, k, v)
        assert (a.float() - b.float()).abs().max() <= 1e-2 * b.float().abs().max(), i
        if i in (15, 16, 39):
            for u in range(batch):
                assert got.last_topk(u) == want.last_topk(u)
    assert got.cached_blocks == want.cached_blocks
