"""infllm_attn_colsum at the edges of its tiles and of the 32 query columns it works on at a time: sum over the queries of
exp2(q.k * scale - lse) for every key, against fp64.  Exponentials are good to 3e-6 and sums of up to 512 of them are added
in fp32 (relative 1e-5 of the sum); the scores under them are fp32 sums of 128 products of 16-bit values (absolute error
2e-6 in the exponent at these sizes): 5e-5 relative leaves room."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

D = 128


@pytest.mark.parametrize("H,HKV,lq,lk,mode,offset,size,accumulate", [
    (32, 8, 512, 4608, 1, 4096, 4096, 1),   # a prompt's exec block
    (32, 8, 512, 640, 1, 4096, 4096, 1),    # its part that is sealed next
    (28, 4, 256, 3100, 1, 2844, 3000, 0),   # a ragged last key tile
    (5, 1, 130, 300, 1, 170, 64, 0),        # two query columns in the last tile; keys that nobody sees
    (4, 2, 160, 1000, 1, 840, 500, 1),      # exactly 32 of them
    (2, 2, 161, 1000, 1, 839, 500, 1),      # one more
    (2, 2, 512, 12800, 1, 12288, 4096, 0),  # long runs of keys that nobody sees
    (148, 4, 130, 129, 0, 0, 0, 1),         # no mask
    (3, 3, 512, 17000, 2, 16000, 500, 0),   # complement mask
])
def test_column_sums(H, HKV, lq, lk, mode, offset, size, accumulate):
    from infllm_b200 import _lib as L

    g = torch.Generator(device="cuda").manual_seed(lq + lk)
    q = torch.randn((H, lq, D), generator=g, device="cuda").bfloat16()
    k = torch.randn((HKV, lk, D), generator=g, device="cuda").bfloat16()
    lse = 10 + torch.randn((H, lq), generator=g, device="cuda")
    out = torch.rand((H, lk + 3), generator=g, device="cuda")
    want = torch.zeros((H, lk), dtype=torch.float64, device="cuda")
    i, j = torch.arange(lq, device="cuda")[:, None], torch.arange(lk, device="cuda")[None]
    dist = i + offset - j
    seen = torch.ones_like(dist, dtype=torch.bool) if mode == 0 else (dist >= 0) & (dist < size) if mode == 1 else dist >= size
    for h in range(H):
        s = q[h].double() @ k[h // (H // HKV)].double().T * (math.log2(math.e) / math.sqrt(D))
        want[h] = torch.where(seen, torch.exp2(s - lse[h].double()[:, None]), 0.0).sum(0)
    if accumulate:
        want += out[:, :lk]
    tail = out[:, lk:].clone()
    L.check(L.lib.infllm_attn_colsum(q.data_ptr(), lq * D, D, k.data_ptr(), lk * D, D, H, HKV, lq, lk, D, mode, offset, size,
                                     lse.data_ptr(), out.data_ptr(), lk + 3, accumulate, L.dtype_code(q.dtype), L.stream_ptr()))
    torch.cuda.synchronize()
    assert L.device_error() == (0, 0)
    assert torch.allclose(out[:, :lk].double(), want, rtol=5e-5, atol=1e-9)
    assert torch.equal(out[:, lk:], tail)
