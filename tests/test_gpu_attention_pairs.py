"""The tcgen05 attention of exec blocks of more than one query tile, in pairs of CTAs and alone (a KV head's query tiles over all
its query heads come out even, or not), against the shape-generic kernel on the same memory.  Every unit is retrieved, so that
both see the same keys.

Tolerance: each kernel rounds probabilities and outputs to bf16; test_gpu_stage_kernels bounds that by 4e-3 in the 2-norm and
2e-2 of the largest output against fp32, two kernels differ by twice that."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

D, UNIT = 128, 128


@pytest.mark.parametrize("h,hkv,exec_,n", [
    (7, 1, 384, 2500),    # 21 tiles: alone
    (7, 1, 256, 2500),    # 14 tiles, the middle pair of two query tiles
    (12, 12, 384, 1900),  # 3 tiles of every head: alone
    (12, 12, 200, 1900),  # pairs of a whole and a ragged tile
    (8, 2, 129, 1500),    # a second tile of one query
    (32, 8, 512, 3000),   # pairs of heads
])
@pytest.mark.parametrize("step", [1.0, 4.0])  # keys that grow: of a few rows the reference maximum moves, once
def test_pairs_and_lone_ctas_match_the_generic_kernel(monkeypatch, h, hkv, exec_, n, step):
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM
    from infllm_b200.attention import context_manager as cmod

    g = torch.Generator(device="cuda").manual_seed(h * exec_)
    q, k, v = (torch.randn((1, m, n, D), generator=g, device="cuda") for m in (h, hkv, hkv))
    k = k * torch.linspace(1.0, step, n, device="cuda")[:, None]
    q, k, v = (x.to(torch.bfloat16) for x in (q, k, v))
    outs = []
    for flags in (0, 1):
        monkeypatch.setattr(cmod, "TEST_OVERRIDES", {"debug_flags": flags})
        cm = ContextManager(RotaryEmbeddingESM(D, 1e6, 1.0), 100, 600, UNIT, 32, 32, exec_, None, True, 2)
        outs.append(cm.append(q, k, v, q, k, v).float())
    err = (outs[0] - outs[1]).abs()
    assert err.norm() <= 8e-3 * outs[1].norm()
    assert err.max() <= 4e-2 * outs[1].abs().max()


# what a row's maximum grows by from a key tile to the next, as a power of two.  A reference moves where that is more than 8.
GROWTH = {
    "every tile": [10] * 10,
    "tiles of the first team": [0, 20] * 5,
    "tiles of the second team": [20, 0] * 5,
    "uneven": [9, 25, 0, 9, 9, 25, 0, 0, 9, 14],
}


@pytest.mark.parametrize("h,hkv,exec_", [
    (32, 8, 512),   # pairs, one run
    (36, 12, 384),  # alone, one run
    (8, 2, 256),    # pairs, several runs
    (7, 1, 384),    # alone, several runs
])
@pytest.mark.parametrize("growth", list(GROWTH))
def test_references_that_move_from_tile_to_tile(h, hkv, exec_, growth):
    """Exec blocks of more than one query tile (lazy references) over one window, against 64 bits, row by row.

    One pair of dimensions that RoPE hardly turns carries the growth of the keys; of a tile's rows those of the first warp follow
    it, one of the second's, every other of the third's and none of the fourth's.  The values fall as the weights of those rows
    grow, so that every key tile has the same part of their outputs and a factor of O that is wrong or missing anywhere shows: at
    least 1 / 11 of an output's square, 0.3 of its norm.  Of a row's sum only the last moves matter.

    Tolerance: a row's error is the rounding of P (2^-9 of a weight at most, 1.1e-3 in the 2-norm), of rotated queries and keys
    (1.1e-3 of a weight) and of the output (2^-9 at most).  Their worst sum over the few keys of an early row, with three standard
    deviations for the middle one: 2^-9 + 3.3e-3 + 2^-9 = 7.2e-3, and twice that is allowed; over all rows 4e-3 (test_gpu_stage_kernels' bound)."""
    from infllm_b200.attention import ContextManager, RotaryEmbeddingESM

    step = torch.tensor([0] + GROWTH[growth], device="cuda")
    n, tiles, c, base = 128 * step.numel(), step.numel(), D // 2 - 1, 1e6
    s = step.cumsum(0).repeat_interleave(128).double()
    log2 = 1 / (D ** 0.5 * math.log(2))  # of a score
    g = torch.Generator(device="cuda").manual_seed(h * exec_ + tiles)
    q, k, v = (torch.randn((1, m, n, D), generator=g, device="cuda") for m in (h, hkv, hkv))
    r = torch.arange(n, device="cuda") % 128
    follows = (r < 32) | (r == 37) | ((r >= 64) & (r < 96) & (r % 2 == 1))
    q *= 0.25
    for x, y in ((q, 8.0 * follows), (k, s / (8.0 * log2))):
        x[..., c], x[..., c + D // 2] = y.float(), 0
    v *= torch.exp2(s[-1] - s).float()[:, None]
    q, k, v = (x.to(torch.bfloat16) for x in (q, k, v))
    cm = ContextManager(RotaryEmbeddingESM(D, base, 1.0), 100, n, UNIT, 32, 32, exec_, None, True, 2)
    got = cm.append(q, k, v, q, k, v).double()

    ang = torch.arange(n, device="cuda")[:, None] / base ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
    cos, sin = ang.cos().repeat(1, 2), ang.sin().repeat(1, 2)

    def turned(x):
        a, b = x.double().chunk(2, -1)
        return x.double() * cos + torch.cat((-b, a), -1) * sin

    kk, vv = (x.repeat_interleave(h // hkv, 1) for x in (turned(k), v.double()))
    score = turned(q) @ kk.transpose(-1, -2) * log2
    score.masked_fill_(r.new_ones((n, n), dtype=torch.bool).triu(1), float("-inf"))
    # the references of the last query tile's rows, which see whole tiles but the last
    ref = torch.full((1, h, 128), float("-inf"), device="cuda", dtype=torch.float64)
    for t in range(tiles):
        m = score[:, :, -128:, t * 128:(t + 1) * 128].amax(-1)
        moves = m - ref > 8
        if t:
            assert torch.equal(moves, (follows[-128:] & (step[t] > 0)).expand_as(moves))
        ref = torch.where(moves, m, ref)
    want = torch.softmax(score * math.log(2), -1) @ vv
    err = (got - want).norm(dim=-1) / want.norm(dim=-1)
    assert err.max() <= 1.5e-2
    assert err.square().mean().sqrt() <= 4e-3


@pytest.mark.parametrize("h,hkv,lq", [(8, 2, 256), (7, 1, 256), (12, 12, 200), (7, 1, 300)])  # pairs of heads, of tiles, ragged; alone
@pytest.mark.parametrize("hidden", [200, 3000])  # keys of the stage that no query sees: one run, and several
@pytest.mark.parametrize("order", ["before", "behind", "only"])
def test_a_stage_that_hides_every_pair_changes_nothing(h, hkv, lq, hidden, order):
    from infllm_b200.attention import get_multi_stage_dot_production_attention

    g = torch.Generator(device="cuda").manual_seed(h * lq + hidden)
    q, k, v, hk, hv = (torch.randn((1, m, n, D), generator=g, device="cuda").to(torch.bfloat16)
                       for m, n in ((h, lq), (hkv, 500), (hkv, 500), (hkv, hidden), (hkv, hidden)))
    stages = [(k, v, 450, False)] * (order != "only")
    stages.insert(order == "behind", (hk, hv, (-10 ** 6, 100), order != "before"))
    att = get_multi_stage_dot_production_attention(True)[0](q.shape, q.dtype, "cuda")
    for i, (sk, sv, win, comp) in enumerate(stages):
        att.append(q, sk, sv, sliding_window=win, complement_sliding_window=comp, end=i == len(stages) - 1)
    got = att.get_result()[0].float()
    if order == "only":
        assert not got.any()
        return
    s = q.float() @ k.float().repeat_interleave(h // hkv, 1).transpose(-1, -2) / D ** 0.5
    dist = torch.arange(lq, device="cuda")[:, None] - torch.arange(500, device="cuda")[None] + 500 - lq
    want = s.masked_fill((dist < 0) | (dist >= 450), float("-inf")).softmax(-1) @ v.float().repeat_interleave(h // hkv, 1)
    err = (got - want).abs()
    assert err.norm() <= 4e-3 * want.norm()  # (test_gpu_stage_kernels' bounds: one kernel against fp32)
    assert err.max() <= 2e-2 * want.abs().max()
