"""Workloads of the context-memory attention framework, through its public entry points.

Kinds of work (the "kind" of a case):

token         one decode token of every sequence of the batch through ContextManager.append, over a memory of
              `units` sealed units per sequence (each pass is the next token of a stream, the memory grows by it)
turn          a few tokens at once on top of such a memory: a chat turn, or the drafts of a speculative decoder
prompt        chunked prefill of a whole prompt; "fresh" through ATTN_FORWRAD["inf-llm"] with no past, as the patched
              model's generation loop starts every prompt, otherwise a kept ContextManager that is reset
sink_prompt   the same for ATTN_FORWRAD["stream-llm"] / ["infinite-lm"]
sink_token    one decode token of those two with a full cache
multi_stage   the multi-stage attention class itself: a windowed stage with key scores and a global stage

Shapes are those of the repository's benchmark configurations (32 query heads over 8 or 32 KV heads, head_dim 128,
window 4096 or 1024, units of 128 tokens) and odd ones of the same kind.

Inputs are N(0,1) with topics planted in them, so that retrieval has real winners: the queries of a stretch of text lean
towards the direction of its topic, some memory units are about one topic, and the first units of a sequence (its
preamble) are relevant to everything by graded amounts.  The keys' noise has no component along the topics, which
keeps the winners clear of the rest: which units are retrieved does not hang on the last bits of a score.
"""
import math

import torch

from infllm_b200.attention import (ATTN_FORWRAD, ContextManager, RotaryEmbeddingESM, device_store_info,
                                   device_store_reserve, get_multi_stage_dot_production_attention)

D = 128    # head dimension
UNIT = 128  # tokens of a memory unit
TOPICS = 8
LEAN_Q = 2.0     # how far a query leans towards its topic
RING = 192       # distinct tokens (or turns) of a stream before it repeats

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _memory(kind, name=None, **over):
    c = dict(kind=kind, heads=32, kv_heads=8, dtype="bf16", n_init=128, n_local=4096, topk=16, max_cached=32, exec=512,
             repr_topk=4, base=1e6, device_store_mb=0)
    c.update(over)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call there is, and the most frequent one: a decode token at a moderate context (24K tokens)
        _memory("token", "token_24k", units=160, batch=1),
        # the decode benchmark: one token over 1,048,576 tokens of context, topk 32
        _memory("token", "token_1m", units=8192, batch=1, topk=32),
        # decode of four sequences at once, fp16, 28 query heads over 4 KV heads
        _memory("token", "token_batch4_fp16", units=75, batch=4, heads=28, kv_heads=4, dtype="fp16"),
        # a short chat turn, or a speculative decoder's drafts: 37 tokens on top of 64K tokens
        _memory("turn", "turn_37", units=480, tokens=37),
        # the small layer configuration: 8192 tokens in one call, exec blocks of 128, window 1024, topk 4; new memory
        _memory("prompt", "prompt_8k_fresh_fp16", tokens=8192, chunk=8192, n_local=1024, topk=4, max_cached=16, exec=128,
                dtype="fp16", fresh=True, dwell=5),
        # a 32K-token prompt as a patched model sees it: a new memory for every prompt, 8192-token chunks
        _memory("prompt", "prompt_32k_fresh", tokens=32768, chunk=8192, fresh=True, dwell=3),
        # odd sizes everywhere: ragged prompt and chunks, 28/4 heads, exec blocks of 256, device copy of the store
        _memory("prompt", "prompt_20k_ragged", tokens=19997, chunk=4099, heads=28, kv_heads=4, exec=256, n_local=3000,
                n_init=100, device_store_mb=512, fresh=False, dwell=4),
        # the headline: a 131072-token prompt through a kept memory
        _memory("prompt", "prompt_128k", tokens=131072, chunk=8192, fresh=False, dwell=3),
        # cache thrash: 32 KV heads, a cache of exactly one retrieval, another topic in every exec block
        _memory("prompt", "prompt_64k_thrash", tokens=65536, chunk=8192, kv_heads=32, exec=256, repr_topk=8, max_cached=16,
                fresh=False, dwell=1),
        # sink + window attention, ragged prompt in 4096-token chunks
        dict(name="sink_prompt_13k", kind="sink_prompt", type="stream-llm", heads=32, kv_heads=8, dtype="bf16", n_init=128,
             n_local=4096, tokens=13001, chunk=4096, base=1e6),
        # its decode token
        dict(name="sink_token", kind="sink_token", type="infinite-lm", heads=32, kv_heads=8, dtype="fp16", n_init=128,
             n_local=4096, base=1e6),
        # the attention class by itself at the shapes of one exec block, odd lengths
        dict(name="multi_stage", kind="multi_stage", heads=32, kv_heads=8, dtype="bf16", queries=509, window=4096,
             window_keys=4605, global_keys=2691),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "token", "turn", "prompt", "prompt", "prompt", "sink_prompt", "sink_token", "multi_stage"])
    heads, kv_heads = rng.choice([(32, 8), (32, 8), (28, 4), (16, 2), (32, 32), (12, 12), (8, 1)])
    dtype = rng.choice(["bf16", "bf16", "fp16"])
    if kind == "multi_stage":
        lq = _log(rng, 1, 1024)
        return dict(kind=kind, heads=heads, kv_heads=kv_heads, dtype=dtype, queries=lq, window=_log(rng, 256, 4096),
                    window_keys=lq + rng.randint(0, 4096), global_keys=_log(rng, 64, 4096))
    if kind in ("sink_prompt", "sink_token"):
        c = dict(kind=kind, type=rng.choice(["stream-llm", "infinite-lm"]), heads=heads, kv_heads=kv_heads, dtype=dtype,
                 n_init=rng.choice([4, 64, 128]), n_local=_log(rng, 512, 4096), base=rng.choice([1e4, 5e5, 1e6]))
        if kind == "sink_prompt":
            c["tokens"] = _log(rng, 700, 16384)
            c["chunk"] = max(_log(rng, 512, 8192), -(-c["tokens"] // 24))
        return c
    topk = rng.choice([4, 8, 16, 16, 32])
    exec_ = rng.choice([128, 256, 512, 512])
    c = _memory(kind, heads=heads, kv_heads=kv_heads, dtype=dtype, n_init=rng.choice([32, 100, 128]),
                n_local=max(exec_, _log(rng, 700, 4096)), topk=topk, max_cached=rng.choice([topk, 2 * topk, 48]), exec=exec_,
                repr_topk=rng.choice([1, 4, 8]), base=rng.choice([1e4, 5e5, 1e6]))
    if kind == "token":
        c["batch"] = rng.choice([1, 1, 1, 2, 4])
        # one memory is installed as it is; several sequences are prefilled
        c["units"] = _log(rng, 50, min(6000, (1 << 16) // kv_heads)) if c["batch"] == 1 else _log(rng, 50, 120)
    elif kind == "turn":
        c["units"] = _log(rng, 50, 1000)
        c["tokens"] = _log(rng, 2, 200)
    else:
        c["tokens"] = _log(rng, 3000, 65536 if kv_heads == 32 else 98304)
        c["chunk"] = min(8192, max(_log(rng, 1000, 8192), -(-c["tokens"] // 48)))
        c["fresh"] = rng.random() < 0.5
        c["dwell"] = rng.choice([1, 3, 6])
        if rng.random() < 0.3:
            c["device_store_mb"] = 4096
    return c


# ------------------------------------------------------------------------------------------------------------ inputs
def _unrotate(u, pos, base):
    """The direction that RoPE at position `pos` turns into u (..., D)."""
    ang = pos / base ** (torch.arange(0, D, 2, device=u.device, dtype=torch.float64) / D)
    a, b = u[..., :D // 2].double(), u[..., D // 2:].double()
    return torch.cat((a * ang.cos() + b * ang.sin(), b * ang.cos() - a * ang.sin()), dim=-1).float()


def _frame(gen, kv_heads, n):
    """n orthonormal directions per KV head, (kv_heads, n, D)."""
    x = torch.randn((kv_heads, D, n), generator=gen, device="cuda")
    return torch.linalg.qr(x)[0].transpose(1, 2).contiguous()


class _Text:
    """q, k and v of a sequence.  Direction 0 is the preamble's, 1..TOPICS the topics'."""

    def __init__(self, c, gen, n_units):
        self.c, self.gen = c, gen
        self.u = _frame(gen, c["kv_heads"], TOPICS + 1)
        w = _unrotate(self.u, c["n_local"] - 1, c["base"])  # retrieval rotates the mean query to that position
        self.w = w.repeat_interleave(c["heads"] // c["kv_heads"], dim=0)
        # strength of unit b along direction z
        s = torch.zeros((n_units + 1, TOPICS + 1))
        grades = 0.5 + 0.25 * torch.arange(c["topk"])
        s[:min(c["topk"], n_units), 0] = grades[:min(c["topk"], n_units)]
        rest = torch.arange(c["topk"], n_units)
        host = torch.Generator().manual_seed(int(torch.randint(0, 1 << 30, (1,), generator=gen, device="cuda")))
        rest = rest[torch.randperm(rest.numel(), generator=host)]
        rest = rest[:min(rest.numel(), TOPICS * c["topk"], max(rest.numel() // 2, TOPICS))]
        s[rest, 1 + torch.arange(rest.numel()) % TOPICS] = float(grades[-1]) + 0.75
        self.s = s.cuda()

    def noise(self, heads, n):
        return torch.randn((heads, n, D), generator=self.gen, device="cuda")

    def keys(self, n):
        k = self.noise(self.c["kv_heads"], n)
        return k - (k @ self.u.transpose(1, 2)) @ self.u

    def tokens(self, start, n, topic):
        """(heads, n, D) q, (kv_heads, n, D) k and v of tokens [start, start + n); `topic` (n,) of each token."""
        c = self.c
        q = self.noise(c["heads"], n) + LEAN_Q * (self.w[:, :1] + self.w[:, 1 + topic])
        unit = ((torch.arange(start, start + n, device="cuda") - c["n_init"]) // UNIT).clamp(-1, self.s.size(0) - 1)
        strength = torch.where((unit >= 0)[:, None], self.s[unit], torch.zeros((), device="cuda"))
        k = self.keys(n) + strength @ self.u
        return q, k, self.noise(c["kv_heads"], n)


def _fused(dst, q, k, v):
    """Token-major rows [q | k | v], as a fused projection leaves them."""
    dst.copy_(torch.cat((q, k, v)).transpose(0, 1).reshape(dst.shape))


def _split(c, x):
    """The head-major views of token-major rows (B, L, width)."""
    h, n = c["heads"], c["kv_heads"]
    x = x.view(x.size(0), x.size(1), h + 2 * n, D).permute(0, 2, 1, 3)
    return x[:, :h], x[:, h:h + n], x[:, h + n:]


def _manager(c, rope):
    return ContextManager(rope, c["n_init"], c["n_local"], UNIT, c["max_cached"], c["topk"], c["exec"], None, True,
                          c["repr_topk"], device_store_mb=c["device_store_mb"])


def _install(c, text, cm, dtype):
    """The memory a decode starts from: its sealed units in the store, full sink and window."""
    gen, kv = text.gen, c["kv_heads"]
    group = c["heads"] // kv
    n = c["units"]
    pool = min(n, 256 * 8 // kv)  # distinct K/V contents; the representative keys are all different
    units = torch.randn((pool, 2, kv, UNIT, D), generator=gen, device="cuda").to(dtype)
    units = units.cpu().repeat((-(-n // pool), 1, 1, 1, 1))[:n]
    block_k = torch.empty((n, c["heads"] * D), dtype=dtype)
    for b in range(0, n, 512):
        m = min(512, n - b)
        rows = text.keys(m) / math.sqrt(c["repr_topk"]) + text.s[b:b + m] @ text.u
        rows = rows.repeat_interleave(group, dim=0) + 0.3 * text.noise(c["heads"], m) / math.sqrt(c["repr_topk"])
        block_k[b:b + m] = rows.transpose(0, 1).reshape(m, -1).to(dtype).cpu()
    small = [text.noise(kv, m).to(dtype).cpu() for m in (c["n_init"], c["n_init"], c["n_local"], c["n_local"])]
    cm.load_synthetic(units, block_k, *small)


def _prepare_stream(c, gen, dtype, per_pass):
    """Token and turn: a memory and the next RING passes of the stream.  A topic lasts 16 tokens, or two turns."""
    rope = RotaryEmbeddingESM(D, c["base"], 1.0)
    cm = _manager(c, rope)
    batch = c.get("batch", 1)
    texts = [_Text(c, gen, c["units"]) for _ in range(batch)]
    width = (c["heads"] + 2 * c["kv_heads"]) * D
    if batch == 1:
        _install(c, texts[0], cm, dtype)
    else:
        total = c["n_init"] + c["units"] * UNIT + c["n_local"]
        for st in range(0, total, 4096):
            n = min(4096, total - st)
            x = torch.empty((batch, n, width), dtype=dtype, device="cuda")
            for b, text in enumerate(texts):
                topic = (torch.arange(st, st + n, device="cuda") // (3 * c["exec"])) % TOPICS
                _fused(x[b], *text.tokens(st, n, topic))
            cm.append(*_split(c, x), *_split(c, x)[:3])
    ring = torch.empty((RING, batch, per_pass, width), dtype=dtype, device="cuda")
    at = c["n_init"] + (c["units"] + 1) * UNIT + c["n_local"]  # past the planted units: fresh text
    topic = (torch.arange(RING, device="cuda") // (16 if per_pass == 1 else 2) % TOPICS).repeat_interleave(per_pass)
    for b, text in enumerate(texts):
        for i in range(0, RING, 16):
            t = topic[i * per_pass:(i + 16) * per_pass]
            q, k, v = text.tokens(at, 16 * per_pass, t)
            _fused(ring[i:i + 16, b].view(16 * per_pass, width), q, k, v)
    return dict(kind=c["kind"], cm=cm, at=0, steps=[_split(c, x) for x in ring])


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    dtype = _DTYPES[c["dtype"]]
    if c["kind"] == "multi_stage":
        def mk(heads, n):
            return torch.randn((1, heads, n, D), generator=gen, device="cuda").to(dtype)
        return dict(kind=c["kind"], cls=get_multi_stage_dot_production_attention(True)[0], window=c["window"],
                    q=(mk(c["heads"], c["queries"]), mk(c["heads"], c["queries"])),
                    k=(mk(c["kv_heads"], c["window_keys"]), mk(c["kv_heads"], c["global_keys"])),
                    v=(mk(c["kv_heads"], c["window_keys"]), mk(c["kv_heads"], c["global_keys"])))
    if c["kind"] == "token":
        return _prepare_stream(c, gen, dtype, 1)
    if c["kind"] == "turn":
        return _prepare_stream(c, gen, dtype, c["tokens"])
    h, n = c["heads"] * D, c["kv_heads"] * D
    width = h + 2 * n
    s = dict(kind=c["kind"], rope=RotaryEmbeddingESM(D, c["base"], 1.0), heads=c["heads"], kv_heads=c["kv_heads"],
             project=(lambda x: x[..., :h], lambda x: x[..., h:h + n], lambda x: x[..., h + n:], lambda o: o))
    if c["kind"] == "prompt":
        text = _Text(c, gen, max(0, c["tokens"] - c["n_init"] - c["n_local"]) // UNIT)
        x = torch.empty((1, c["tokens"], width), dtype=dtype, device="cuda")
        for st in range(0, c["tokens"], 8192):
            m = min(8192, c["tokens"] - st)
            topic = (torch.arange(st, st + m, device="cuda") // (c["dwell"] * c["exec"])) % TOPICS
            _fused(x[0, st:st + m], *text.tokens(st, m, topic))
        s["chunks"] = list(x.split(c["chunk"], dim=1))
        s["fresh"] = c["fresh"]
        if c["device_store_mb"]:  # the program reserves the pool for the memories it keeps, once
            while True:
                total, used = device_store_info()
                if total - used >= 4 * c["device_store_mb"]:
                    break
                device_store_reserve(c["device_store_mb"])
        if c["fresh"]:
            s["forward"] = ATTN_FORWRAD["inf-llm"](
                n_local=c["n_local"], n_init=c["n_init"], topk=c["topk"], block_size=UNIT, max_cached_block=c["max_cached"],
                exc_block_size=c["exec"], fattn=True, repr_topk=c["repr_topk"], device_store_mb=c["device_store_mb"])
        else:
            s["cm"] = _manager(c, s["rope"])
            s["chunks"] = [_split(c, x) for x in s["chunks"]]
        return s
    s["forward"] = ATTN_FORWRAD[c["type"]](n_local=c["n_local"], n_init=c["n_init"], fattn=True)
    if c["kind"] == "sink_prompt":
        x = torch.randn((1, c["tokens"], width), generator=gen, device="cuda").to(dtype)
        s["chunks"] = list(x.split(c["chunk"], dim=1))
        return s
    full = c["n_init"] + c["n_local"]
    s["past"] = tuple(torch.randn((1, c["kv_heads"], full, D), generator=gen, device="cuda").to(dtype) for _ in range(2)) + (
        full + 5000,)
    s["steps"] = list(torch.randn((RING, 1, 1, width), generator=gen, device="cuda").to(dtype))
    s["at"] = 0
    return s


# ------------------------------------------------------------------------------------------------------------- a pass
def _forward(s, x, past):
    return s["forward"](None, x, x, s["rope"], True, past, *s["project"], D, s["heads"], s["kv_heads"])


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("token", "turn"):
        q, k, v = s["steps"][s["at"] % RING]
        s["at"] += 1
        return s["cm"].append(q, k, v, q, k, v)
    if kind == "multi_stage":
        att = s["cls"](s["q"][0].shape, s["q"][0].dtype, s["q"][0].device)
        att.append(s["q"][0], s["k"][0], s["v"][0], sliding_window=s["window"], get_score=True)
        lq, lk = s["q"][1].size(2), s["k"][1].size(2)
        att.append(s["q"][1], s["k"][1], s["v"][1], end=True, sliding_window=(lk + lq, s["window"]),
                   complement_sliding_window=True)
        return att.get_result()
    if kind == "sink_token":
        x = s["steps"][s["at"] % RING]
        s["at"] += 1
        o, s["past"] = _forward(s, x, s["past"])
        return o, s["past"]
    if kind == "sink_prompt" or s["fresh"]:
        past, outs = None, []
        for x in s["chunks"]:
            o, past = _forward(s, x, past)
            outs.append(o)
        return (outs, past) if kind == "sink_prompt" else outs
    s["cm"].reset()
    return [s["cm"].append(q, k, v, q, k, v) for q, k, v in s["chunks"]]


# ----------------------------------------------------------------------------------------------------------- its bounds
def _window_pairs(first, n, width):
    """Visible pairs of n queries at positions first.. over a causal window of `width` keys."""
    full = max(0, min(n, first + n - width + 1)) if first + n >= width else 0
    part = n - full
    return part * first + part * (part + 1) // 2 + full * width


def _memory_work(c, length, tokens, chunk):
    """Operations and bytes of appending `tokens` tokens in `chunk`-token calls to a memory of `length` tokens."""
    h, kv = c["heads"], c["kv_heads"]
    n_init, n_local, exec_ = c["n_init"], c["n_local"], c["exec"]
    init_len = n_init if length > n_local + n_init else 0
    frontier = n_init + (length - n_init - n_local) // UNIT * UNIT if init_len else 0
    flops, rows, sealed = 0, 0, 0
    done = 0
    while done < tokens:
        call = min(chunk, tokens - done)
        for st in range(0, call, exec_):
            lq = min(exec_, call - st)
            end = length + lq
            units = max(0, (frontier - n_init) // UNIT) if init_len == n_init else 0
            local = _window_pairs(length, lq, n_local)
            glob = lq * (min(units, c["topk"]) * UNIT + init_len + max(0, end - frontier - n_local))
            flops += 4 * D * h * (local + glob) + 2 * D * h * local + 2 * D * h * units
            rows = max(rows, units)
            length = end
            if init_len < n_init and end - frontier > n_local:
                take = min(n_init - init_len, end - frontier - n_local)
                init_len += take
                frontier += take
            while end - frontier - UNIT >= n_local:
                frontier += UNIT
                sealed += 1
        done += call
    moved = tokens * (2 * h + 2 * kv) * D * 2 + sealed * (2 * kv * UNIT * D * 2 + h * D * 2)
    return flops, moved


def work(case):
    c = case
    h, kv = c["heads"], c["kv_heads"]
    if c["kind"] in ("token", "turn"):
        length = c["n_init"] + c["units"] * UNIT + c["n_local"]
        tokens = c.get("tokens", 1)
        flops, moved = _memory_work(c, length, tokens, tokens)
        n_exec = -(-tokens // c["exec"])
        keys = c["n_local"] + min(c["topk"], c["units"]) * UNIT + c["n_init"] + UNIT // 2
        moved += n_exec * c["units"] * h * D * 2 + keys * kv * D * 4 + 2 * h * c["n_local"] * 4
        b = c.get("batch", 1)
        return {"bytes": b * moved, "flops": b * flops}
    if c["kind"] == "prompt":
        flops, moved = _memory_work(c, 0, c["tokens"], c["chunk"])
        return {"bytes": moved, "flops": flops}
    if c["kind"] == "multi_stage":
        lq, lk, glk = c["queries"], c["window_keys"], c["global_keys"]
        local = _window_pairs(lk - lq, lq, c["window"])
        return {"bytes": (3 * h * lq + 2 * kv * (lk + glk)) * D * 2 + h * lk * 2,
                "flops": 4 * D * h * (local + lq * glk) + 2 * D * h * local}
    full = c["n_init"] + c["n_local"]
    if c["kind"] == "sink_token":
        return {"bytes": 4 * kv * full * D * 2 + (2 * h + 2 * kv) * D * 2, "flops": 4 * D * h * full}
    t = c["tokens"]
    pairs = _window_pairs(0, t, c["n_local"]) + max(0, t - c["n_local"]) * min(c["n_init"], t)
    return {"bytes": t * (2 * h + 2 * kv) * D * 2 + 2 * kv * min(full, t) * D * 2, "flops": 4 * D * h * pairs}


def tolerance(case):
    """Outputs are rounded to the 16-bit type and so are the probabilities that weight the values: a few units of its
    last place, relative to a row's size; "max" leaves room for the largest of tens of millions of values."""
    return {"rel": 1e-2, "max": 0.1} if case["dtype"] == "bf16" else {"rel": 3e-3, "max": 0.05}
