"""infllm_sink_window_run against the same call put together from the attention class (which the golden recordings
pin): outputs within the rounding of the 16-bit types (both round probabilities and outputs to them: 2e-2 of the
largest output), caches bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["infinite-lm", "stream-llm"])
@pytest.mark.parametrize("h,hkv,batch", [(8, 2, 1), (7, 1, 2), (12, 1, 1), (4, 4, 1)])
@pytest.mark.parametrize("n_local,n_init,lens", [
    (256, 128, (700, 1, 1, 130, 1)),       # past the window in the first call
    (300, 4, (100, 1, 203, 1, 1, 64, 1)),  # the history reaches n_local + n_init, one token over, and goes on
    (129, 1, (1, 1, 127, 2, 1, 400)),      # a sink of one token
    (512, 64, (2049,)),
])
def test_call_equals_the_composition(kind, h, hkv, batch, n_local, n_init, lens):
    from infllm_b200.attention import ATTN_FORWRAD, RotaryEmbeddingESM

    class Other(RotaryEmbeddingESM):  # another class: the general path
        pass

    d = 128
    g = torch.Generator(device="cuda").manual_seed(h + n_local)
    forward = ATTN_FORWRAD[kind](n_local=n_local, n_init=n_init, fattn=True)
    proj = (lambda x: x[..., :h * d], lambda x: x[..., h * d:(h + hkv) * d], lambda x: x[..., (h + hkv) * d:], lambda o: o)
    past = [None, None]
    ropes = (RotaryEmbeddingESM(d, 1e6, 1.0), Other(d, 1e6, 1.0))
    for i, n in enumerate(lens):
        x = torch.randn((batch, n, (h + 2 * hkv) * d), generator=g, device="cuda").to(torch.float16)
        outs = []
        for j in range(2):
            o, past[j] = forward(None, x, x, ropes[j], True, past[j], *proj, d, h, hkv)
            outs.append(o)
        assert outs[0].shape == outs[1].shape == (batch, n, h * d)
        err = (outs[0].float() - outs[1].float()).abs().max()
        assert err <= 2e-2 * outs[1].float().abs().max(), (i, n, err)
        assert past[0][2] == past[1][2]
        assert torch.equal(past[0][0], past[1][0]) and torch.equal(past[0][1], past[1][1])
    o = forward(None, x, x, ropes[0], False, past[0], *proj, d, h, hkv)
    w = forward(None, x, x, ropes[1], False, past[1], *proj, d, h, hkv)
    assert (o.float() - w.float()).abs().max() <= 2e-2 * w.float().abs().max()


@pytest.mark.parametrize("n", [1, 2, 70])
def test_an_output_holds_no_more_memory_than_itself(n):
    """attention_out may hand its input on, and a program may keep every token's output."""
    from infllm_b200.attention import ATTN_FORWRAD, RotaryEmbeddingESM

    h, hkv, d = 8, 2, 128
    forward = ATTN_FORWRAD["infinite-lm"](n_local=256, n_init=64, fattn=True)
    proj = (lambda x: x[..., :h * d], lambda x: x[..., h * d:(h + hkv) * d], lambda x: x[..., (h + hkv) * d:], lambda o: o)
    past = None
    for length in (700, n):
        x = torch.randn((1, length, (h + 2 * hkv) * d), device="cuda").to(torch.bfloat16)
        o, past = forward(None, x, x, RotaryEmbeddingESM(d, 1e6, 1.0), True, past, *proj, d, h, hkv)
    assert o.untyped_storage().nbytes() == n * h * d * 2
