"""Workspaces of dropped memories are handed out again (infllm_ctx_destroy / infllm_ctx_create): a memory that starts
in them, on another stream and behind work that is still running, behaves like the first one, and nothing of the old
sequence is left - not even values that no arithmetic would wipe out."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, HKV, D = 8, 2, 128


def _tokens(n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn((1, h, n, D), generator=g, device="cuda").to(torch.bfloat16) for h in (H, HKV, HKV)]


def _run(calls, stream=None, device_store_mb=0):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 64, 512, 128, 6, 4, 256, None, True, 4,
                        device_store_mb=device_store_mb)
    with torch.cuda.stream(stream) if stream is not None else torch.cuda.stream(torch.cuda.current_stream()):
        outs = [cm.append(q, k, v, q, k, v) for q, k, v in calls]
    return cm, outs


@pytest.mark.parametrize("tail", [1, 37, 300])
def test_a_reused_memory_equals_a_new_one(tail):
    from infllm_b200.attention import release_idle_memories

    calls = [_tokens(2300, 1), _tokens(tail, 2), _tokens(1, 3)]
    torch.cuda.synchronize()
    release_idle_memories()
    cm, want = _run(calls)
    ids = cm.last_topk()
    torch.cuda.synchronize()
    # another sequence in the same workspaces: longer, with infinities in its keys and values, dropped while it runs
    other = [_tokens(4000, 4)]
    other[0][1][:, :, 100::7] = float("inf")
    other[0][2][:, :, ::5] = float("nan")
    torch.cuda.synchronize()
    del cm
    cm, _ = _run(other)
    del cm
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    cm, got = _run(calls, side)
    assert cm.last_topk() == ids
    torch.cuda.synchronize()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_idle_memories_are_bounded_by_their_shape_and_given_back():
    from infllm_b200.attention import release_idle_memories

    torch.cuda.synchronize()
    release_idle_memories()
    calls = [_tokens(1500, 5)]
    cm, _ = _run(calls)
    torch.cuda.synchronize()
    held = torch.cuda.mem_get_info()[0]
    for _ in range(3):  # one at a time: the same workspaces every time
        del cm
        cm, _ = _run(calls)
    torch.cuda.synchronize()
    # (the stream-ordered pool behind the token buffers may grow by a buffer while the old one is still in use)
    assert torch.cuda.mem_get_info()[0] >= held - (64 << 20)
    del cm
    release_idle_memories()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > held


@pytest.mark.parametrize("dropped", [True, False])
def test_a_new_store_waits_for_the_old_memorys_last_token(dropped):
    """The last token of a memory reads its units in place from the host store and is still queued when the memory is
    dropped (or reset) and other units are loaded into the same slabs: its output is that of its own units."""
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM, release_idle_memories

    n_units, n_init, n_local = 40, 64, 256
    g = torch.Generator().manual_seed(6)
    rnd = lambda *s: torch.randn(s, generator=g).to(torch.bfloat16)  # noqa: E731
    block_k = rnd(n_units, H * D)
    small = [rnd(HKV, n, D) for n in (n_init, n_init, n_local, n_local)]
    units = [rnd(n_units, 2, HKV, 128, D) for _ in range(2)]
    q, k, v = _tokens(1, 7)
    make = lambda: ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), n_init, n_local, 128, 8, 8, 256, None, True, 2)  # noqa: E731

    def run(behind_work):
        cm = make()
        cm.load_synthetic(units[0], block_k, *small)
        if behind_work:
            torch.cuda._sleep(400_000_000)  # about 0.2 s
        out = cm.append(q, k, v, q, k, v)
        if not behind_work:
            torch.cuda.synchronize()
        if dropped:
            del cm
            cm = make()
        else:
            cm.reset()
        cm.load_synthetic(units[1], block_k, *small)
        torch.cuda.synchronize()
        return out, cm.append(q, k, v, q, k, v)

    torch.cuda.synchronize()
    release_idle_memories()
    want, got = run(False), run(True)
    assert not torch.equal(want[0], want[1])
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_a_whole_models_memories_are_dropped_and_taken_up_again():
    """32 layers of 32/8 heads, exec blocks of 512, window 4096, dropped at once and started again twice: every one of them
    stays, and the next prompt allocates nothing."""
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM, release_idle_memories

    h, hkv, n = 32, 8, 5000
    g = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (torch.randn((1, x, n, D), generator=g, device="cuda").to(torch.bfloat16) for x in (h, hkv, hkv))
    rope = RotaryEmbeddingESM(D, 1e6, 1.0)

    def model():
        layers = [ContextManager(rope, 128, 4096, 128, 32, 16, 512, None, True, 4) for _ in range(32)]
        outs = [m.append(q, k, v, q, k, v)[0, 0, -1, 0].item() for m in layers]
        torch.cuda.synchronize()
        return layers, outs, torch.cuda.mem_get_info()[0]

    torch.cuda.synchronize()
    release_idle_memories()
    layers, want, live = model()
    for _ in range(2):
        del layers
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] <= live + (256 << 20)  # (one of them is 600 MiB)
        layers, outs, now = model()
        assert outs == want and now >= live - (64 << 20)
    del layers
    release_idle_memories()
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info()[0] > live + 32 * (400 << 20)
