"""Tokens that move to the front of their buffers between calls: the same prompt in one call and in many.  What the
buffers hold afterwards is the tokens, bit for bit (a saved memory shows it); the exec blocks coincide, so where an exec
block retrieves the same units its outputs are the same sums over the same tiles (equal up to how the window's tiles are
cut: 16-bit roundings of the probabilities)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N_INIT, EXEC = 20, 64


def _moves(calls, n_local, unit):
    """How many calls find their buffers full and move what is left in place, by the rule of the native code."""
    cap = t0 = length = frontier = init = n = 0
    for call in calls:
        if length + call - t0 > cap:
            live = length - frontier
            if live + call <= cap and live <= frontier - t0:
                n += 1
            else:
                cap = -(-(live + call + max(4096, n_local + N_INIT + 4 * unit)) // 256) * 256
            t0 = frontier
        for _ in range(0, call, EXEC):
            length += EXEC
            if init < N_INIT and length - frontier > n_local:
                take = min(N_INIT - init, length - frontier - n_local)
                init, frontier = init + take, frontier + take
            while length - frontier - unit >= n_local:
                frontier += unit
    return n


def _saved(path, H, HKV, D, unit):
    """What a saved memory holds: lengths, sink, un-sealed tokens and sealed units (K and V each), accumulated scores."""
    raw = np.fromfile(path, dtype=np.uint8)
    hdr = raw[:192].view(np.int64)
    length, frontier, blocks, init_len, n_lru = int(hdr[8]), int(hdr[9]), int(hdr[10]), int(hdr[11]), int(hdr[14])
    at = 192 + 16 * n_lru

    def take(*shape, dtype=torch.int16):
        nonlocal at
        n = int(np.prod(shape)) * dtype.itemsize
        x = torch.frombuffer(bytearray(raw[at:at + n].tobytes()), dtype=dtype).view(shape) if n else torch.empty(shape, dtype=dtype)
        at += n
        return x

    sink = take(HKV, init_len, D), take(HKV, init_len, D)
    take(blocks, H * D)
    live = take(HKV, length - frontier, D), take(HKV, length - frontier, D)
    score = take(H, length - frontier, dtype=torch.float32)
    units = take(blocks, 2, HKV, unit, D)
    assert at == raw.size
    return length, frontier, sink, live, score, units


@pytest.mark.parametrize("D,H,HKV,n_local,calls,unit", [
    (128, 8, 2, 256, [704] * 14, 32),    # several moves in place, after the buffers have grown once
    (64, 4, 4, 256, [704] * 14, 32),     # rows of 128 bytes
    (128, 8, 1, 4096, [4992] * 4, 32),   # a window as long as the slack
    (128, 28, 4, 300, [64] * 150, 32),   # one exec block per call
    (128, 8, 1, 4000, [4096, 4096] + [128] * 70, 32),  # short calls: the rows that are cleared are among those that move
    (128, 4, 1, 3000, [4096, 4032, 4096, 3968, 128], 32),  # calls that shrink: some of them are
    (128, 8, 2, 256, [704] * 14, 128),   # the tcgen05 kernels, which read rows behind the data
    (128, 8, 1, 4000, [4096, 4096] + [128] * 70, 128),
])
def test_one_call_equals_many(D, H, HKV, n_local, calls, unit, tmp_path):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    assert _moves(calls, n_local, unit) >= 1
    g = torch.Generator(device="cuda").manual_seed(D + len(calls))
    n = sum(calls)
    q, k, v = (torch.randn((1, h, n, D), generator=g, device="cuda").bfloat16() for h in (H, HKV, HKV))
    make = lambda: ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), N_INIT, n_local, unit, 16, 4, EXEC, None, True, 2)  # noqa: E731
    whole, parts = make(), make()
    want = whole.append(q, k, v, q, k, v)
    last = whole.last_topk()
    ids, got = [], []
    at = 0
    for call in calls:
        t = [x[:, :, at:at + call] for x in (q, k, v)]
        at += call
        got.append(parts.append(*t, *t))
        ids += parts.last_topk()
    got = torch.cat(got, dim=2)
    assert len(ids) == len(last) == n // EXEC
    same = torch.tensor([a == b for a, b in zip(last, ids)], device="cuda")
    assert (~same).sum() <= len(last) // 50  # near ties
    assert (whole.block_k_rows() != parts.block_k_rows()).any(1).float().mean() <= 0.02
    rows = same.repeat_interleave(EXEC)
    err, size = ((got.float() - want.float())[0][:, rows].norm(dim=-1), want.float()[0][:, rows].norm(dim=-1))
    assert (err <= 1.5e-2 * size).all()  # every one of them

    for name, cm in (("whole", whole), ("parts", parts)):
        cm.save(str(tmp_path / name))
    kept = [_saved(f"{tmp_path}/{name}.u0", H, HKV, D, unit) for name in ("whole", "parts")]
    length, frontier, sink, live, score, units = kept[1]
    assert (length, frontier) == kept[0][:2] == (n, N_INIT + units.size(0) * unit)
    for i, x in enumerate((k, v)):
        x = x[0].view(torch.int16).cpu()
        assert torch.equal(sink[i], x[:, :N_INIT])
        assert torch.equal(live[i], x[:, frontier:])
        assert torch.equal(units[:, i].transpose(0, 1).reshape(HKV, -1, D), x[:, N_INIT:frontier])
    # probabilities of bf16 logits, summed in fp32
    torch.testing.assert_close(score, kept[0][4], rtol=2e-2, atol=1e-3)
