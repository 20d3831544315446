"""The device memory in which evicted units stay readable has bounds, and a field that sets it (keep_evicted_mb); what is
retrieved, cached and computed does not depend on it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, HKV, D, UNIT_BYTES = 8, 2, 128, 2 * 2 * 128 * 128 * 2


def _memory(max_cached, keep):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 64, 256, 128, max_cached, 8, 256, None, True, 2, keep_evicted_mb=keep)
    x = torch.zeros(1, H, 1, D, device="cuda", dtype=torch.bfloat16)
    cm.append(x, x[:, :HKV], x[:, :HKV], x, x[:, :HKV], x[:, :HKV])
    return cm


def _taken(max_cached, keep, n=1):
    """Device memory of n memories."""
    from infllm_b200.attention import release_idle_memories

    torch.cuda.synchronize()
    release_idle_memories()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    cms = [_memory(max_cached, keep) for _ in range(n)]
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    del cms
    release_idle_memories()
    return used


SLACK = 24 << 20  # allocations are rounded to 2 MiB, and the stream-ordered pool may grow


def test_the_kept_memory_is_what_the_field_says():
    total = torch.cuda.mem_get_info()[1]
    _taken(8, -1)  # (the process's first memory also loads kernels)
    none, some, usual = _taken(8, -1), _taken(8, 40), _taken(8, 0)
    assert abs(some - none - (40 << 20)) <= SLACK
    assert abs(usual - none - 8 * 8 * UNIT_BYTES) <= SLACK  # eight times the cache of eight units
    none, usual = _taken(2000, -1), _taken(2000, 0)
    assert total // 1024 - SLACK - UNIT_BYTES <= usual - none <= total // 1024 + SLACK


def test_all_memories_share_a_budget():
    total = torch.cuda.mem_get_info()[1]
    none = _taken(2000, -1, 1)
    many = _taken(2000, 0, 40)
    assert many - 40 * none <= total // 32 + 40 * SLACK
    assert _taken(2000, 0) > none + total // 1024 - SLACK - UNIT_BYTES  # and it is given back


def test_results_do_not_depend_on_it():
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda n: [torch.randn((1, h, n, D), generator=g, device="cuda").to(torch.bfloat16) for h in (H, HKV, HKV)]  # noqa: E731
    calls = [rnd(n) for n in (6000, 1, 1, 1, 700, 1, 1)]
    got = []
    for keep in (-1, 0, 3):
        cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 64, 256, 128, 4, 4, 128, None, True, 2, keep_evicted_mb=keep)
        got.append(([cm.append(q, k, v, q, k, v) for q, k, v in calls], cm.cached_blocks, cm.info()))
    assert got[0][2]["evictions"] > 20 and got[0][2]["h2d_bytes"] > got[1][2]["h2d_bytes"]
    for outs, cached, info in got[1:]:
        assert cached == got[0][1] and info["cache_misses"] == got[0][2]["cache_misses"]
        assert all(torch.equal(a, b) for a, b in zip(outs, got[0][0]))
