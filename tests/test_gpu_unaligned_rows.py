"""C entries that took rows at any alignment, or at 4 bytes, still do."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,lq,dim,acc_off,out_off,pitch", [
    (4, 37, 128, 0, 0, 128), (4, 37, 128, 1, 0, 128), (4, 37, 128, 2, 3, 131), (3, 5, 64, 0, 2, 66), (2, 9, 6, 0, 0, 6), (2, 3, 1, 1, 1, 1),
])
def test_finalize(heads, lq, dim, acc_off, out_off, pitch, dtype):
    from infllm_b200 import _lib

    g = torch.Generator(device="cuda").manual_seed(dim + lq)
    acc = torch.randn(heads * lq * dim + acc_off, generator=g, device="cuda")[acc_off:]
    m = torch.randn(heads * lq, generator=g, device="cuda")
    l = torch.rand(heads * lq, generator=g, device="cuda") + 0.5  # noqa: E741
    l[1] = 0
    buf = torch.full((heads * lq * pitch + out_off + 8,), 7.0, device="cuda", dtype=dtype)
    lse = torch.empty(heads * lq, device="cuda")
    _lib.check(_lib.lib.infllm_attn_finalize(acc.data_ptr(), m.data_ptr(), l.data_ptr(), buf.data_ptr() + 2 * out_off,
                                             lq * pitch, pitch, lse.data_ptr(), heads, lq, dim, _lib.dtype_code(dtype),
                                             _lib.stream_ptr()))
    rows = buf[out_off:out_off + heads * lq * pitch].view(heads * lq, pitch)
    inv = torch.where(l > 0, 1 / l, torch.zeros(()).cuda())
    want = (acc.view(heads * lq, dim) * inv[:, None]).to(dtype)
    ulp = 2.0 ** (-7 if dtype == torch.bfloat16 else -10)  # a reciprocal and a product against a product: one unit at most
    assert ((rows[:, :dim].float() - want.float()).abs() <= ulp * want.float().abs() + 1e-7).all()
    assert (rows[:, dim:] == 7).all() and (buf[:out_off] == 7).all() and (buf[out_off + heads * lq * pitch:] == 7).all()
    assert torch.allclose(lse[l > 0], (m + torch.log2(l))[l > 0], rtol=1e-5, atol=1e-5) and lse[1] == -float("inf")


@pytest.mark.parametrize("n", [2, 37, 64, 200, 700])
@pytest.mark.parametrize("off,pitch", [(2, 128), (4, 130), (0, 132)])
def test_outputs_of_a_memory(n, off, pitch):
    """Output rows on 4-byte boundaries (what infllm_ctx_append asks for), `pitch` elements apart."""
    from infllm_b200 import _lib
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    H, HKV, D = 8, 2, 128
    g = torch.Generator(device="cuda").manual_seed(n)
    calls = [[torch.randn((1, h, x, D), generator=g, device="cuda").to(torch.bfloat16) for h in (H, HKV, HKV)] for x in (1500, n)]
    cms = [ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 64, 512, 128, 6, 4, 512, None, True, 4) for _ in range(2)]
    for cm in cms:
        cm.append(*calls[0], *calls[0])
    want = cms[0].append(*calls[1], *calls[1])[0].float()
    buf = torch.full((H * n * pitch + off + 8,), 7.0, device="cuda", dtype=torch.bfloat16)
    q, k, v = (t[0] for t in calls[1])
    _lib.check(_lib.lib.infllm_ctx_append(
        cms[1]._ctx[0], q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0),
        v.stride(1), buf.data_ptr() + 2 * off, n * pitch, pitch, n, _lib.stream_ptr()))
    rows = buf[off:off + H * n * pitch].view(H, n, pitch)
    # another kernel: probabilities and outputs are rounded to bf16, a few 2^-9 of a row's size
    assert (rows[..., :D].float() - want).abs().max() <= 2e-2 * want.abs().max()
    assert (rows[..., D:] == 7).all() and (buf[:off] == 7).all() and (buf[off + H * n * pitch:] == 7).all()
