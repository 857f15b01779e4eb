"""The work that users of this framework have it do, as measurable cases.

Two entry points carry a serving engine's attention layer: the op
``pth_flash_attn_fwd`` (planned by ``planner.plan_launch``), which reads the paged int8
cache, and ``host.write_kv``, which quantises new tokens into it.  A case is one call of
one of them on one layer's batch.

A batch is written as text, one term per group of requests: ``count*q+prior``, where ``q``
(query tokens of the call) and ``prior`` (tokens already in the cache) are numbers or
ranges ``lo-hi`` drawn uniformly with ``lens_seed``.  ``8*1+0-4095`` is eight decode
requests of 1 to 4,096 keys.  ``kind`` says which reservation of split workspace the
caller makes: ``decode`` (also verification and drafter steps), ``prefill`` or ``mixed``.
"""
from __future__ import annotations

import random

import torch

from pth_flash_attn_b200 import host, ops, planner

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
_WRITE_STEP = 1 << 18   # rows (token, KV head) filled at once while a cache is made


def _case(op, kind, batch, Hq, Hkv, D, *, page=16, layout="NHD", dtype="bf16", window=0, lens_seed=1, name=None):
    c = dict(op=op, kind=kind, batch=batch, Hq=Hq, Hkv=Hkv, D=D, page=page, layout=layout, dtype=dtype,
             window=window, lens_seed=lens_seed)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # A small interactive batch: eight users, contexts of a few thousand tokens at most.
        # Little to read, so launches and pipeline fill decide the latency of a token.
        _case("attention", "decode", "8*1+0-4095", 32, 8, 128, name="decode_b8"),
        # One very long document being continued: all the parallelism has to come from the keys.
        _case("attention", "decode", "1*1+131071", 32, 8, 128, name="decode_long_b1"),
        # Throughput serving: a full batch of medium contexts, bound by the cache's bytes.
        _case("attention", "decode", "64*1+8191", 32, 8, 128, name="decode_b64"),
        # The same load at 256 dims with few KV heads and large per-head pages (816 slots).
        _case("attention", "decode", "64*1+8191", 12, 2, 256, page=816, layout="HND", name="decode_d256"),
        # Small heads, float16 queries, ragged contexts.
        _case("attention", "decode", "64*1+4095-12287", 32, 8, 64, dtype="fp16", name="decode_d64"),
        # Speculative decoding: four draft tokens of each request are verified at once.
        _case("attention", "decode", "32*4+16380-32764", 32, 8, 128, name="verify4"),
        # The draft model's layer: sixteen tokens each under a sliding window.
        _case("attention", "decode", "32*16+16368-32752", 32, 8, 128, window=4096, name="drafter16"),
        # New prompts of every length, nothing cached yet: short key ranges, ragged tiles.
        _case("attention", "prefill", "12*37-2500+0", 32, 8, 128, dtype="fp16", name="prefill_fresh"),
        # Long prompts fed chunk by chunk: the heaviest call, bound by the tensor cores.
        _case("attention", "prefill", "4*2048+30720", 64, 8, 128, name="prefill_chunked"),
        # Chunks at 256 dims over large per-head pages.
        _case("attention", "prefill", "4*2048+30720", 12, 2, 256, page=816, layout="HND", name="prefill_d256"),
        # One call for a whole engine step: decode, verification and prefill requests together.
        _case("attention", "mixed", "48*1+4095-131071 8*4+32764 2*1024+16384", 64, 8, 128, name="mixed"),
        # The step in front of attention: a prefill step's keys and values into the cache.
        _case("write", "prefill", "4*2048+0", 64, 8, 128, name="write_prefill"),
    ]


# (query heads, KV heads, head size) met in draws: the listed ones, and the share of one of
# several GPUs when the KV heads are divided among them
_HEADS = ((32, 8, 128), (64, 8, 128), (8, 2, 128), (8, 1, 128), (32, 8, 64), (12, 2, 256), (32, 8, 256))


def _log_int(rng, lo, hi):
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def _span(rng, hi, lo=0):
    """All requests alike, or ragged from ``lo`` (or anything between) up to ``hi``."""
    if rng.random() < 0.25:
        return str(hi)
    low = lo + round((hi - lo) * rng.choice((0.0, rng.random())))
    return f"{low}-{hi}" if low < hi else str(hi)


def _draw_any(rng):
    family = rng.choice(("decode", "decode", "verify", "drafter", "prefill", "prefill", "mixed", "write"))
    Hq, Hkv, D = rng.choice(_HEADS)
    opt = dict(layout=rng.choice(("NHD", "HND")), dtype=rng.choice(("bf16", "bf16", "fp16")),
               page=rng.choice((16, 16, 32, 64, 816)), lens_seed=rng.randrange(1 << 30))
    if family == "decode":
        batch = f"{_log_int(rng, 1, 128)}*1+{_span(rng, _log_int(rng, 128, 131071))}"
        return _case("attention", "decode", batch, Hq, Hkv, D, **opt)
    if family == "verify":
        batch = f"{_log_int(rng, 1, 64)}*{rng.randint(2, 8)}+{_span(rng, _log_int(rng, 256, 32764))}"
        return _case("attention", "decode", batch, Hq, Hkv, D, **opt)
    if family == "drafter":   # sliding windows exist at 128 dims
        batch = f"{_log_int(rng, 1, 64)}*{rng.randint(8, 16)}+{_span(rng, _log_int(rng, 512, 32752))}"
        return _case("attention", "decode", batch, *rng.choice([h for h in _HEADS if h[2] == 128]),
                     window=rng.randint(512, 4096), **opt)
    if family == "mixed":
        batch = (f"{_log_int(rng, 1, 48)}*1+{_span(rng, _log_int(rng, 256, 131071))} "
                 f"{rng.randint(1, 8)}*4+{_span(rng, _log_int(rng, 256, 32764))} "
                 f"{rng.randint(1, 4)}*{_span(rng, _log_int(rng, 64, 2048), 1)}+{_span(rng, _log_int(rng, 64, 16384))}")
        return _case("attention", "mixed", batch, Hq, Hkv, D, **opt)
    if family == "prefill":
        prior = rng.choice(("0", _span(rng, _log_int(rng, 64, 30720))))
        batch = f"{rng.randint(1, 16)}*{_span(rng, _log_int(rng, 16, 4096), 1)}+{prior}"
        return _case("attention", "prefill", batch, Hq, Hkv, D, **opt)
    if rng.random() < 0.5:    # a decode step's tokens, or a prefill step's
        batch = f"{_log_int(rng, 1, 256)}*1+{_span(rng, 255)}"
    else:
        batch = f"{rng.randint(1, 8)}*{_span(rng, _log_int(rng, 16, 4096), 1)}+0"
    return _case("write", "prefill", batch, Hq, Hkv, D, **opt)


def draw(rng):
    """A case of the listed cases' ranges, no heavier in bytes or in operations than the heaviest of them."""
    heaviest = [max(work(c)[unit] for c in listed()) for unit in ("bytes", "flops")]
    while True:
        case = _draw_any(rng)
        w = work(case)
        if w["bytes"] <= heaviest[0] and w["flops"] <= heaviest[1]:
            return case


def _range(text, rng):
    lo, _, hi = text.partition("-")
    return rng.randint(int(lo), int(hi)) if hi else int(lo)


def _lengths(case):
    """(query tokens, keys in the cache) of every request of the call."""
    rng = random.Random(case["lens_seed"])
    out = []
    for term in case["batch"].split():
        count, _, rest = term.partition("*")
        q, _, prior = rest.partition("+")
        for _ in range(int(count)):
            n = _range(q, rng)
            out.append((n, n + _range(prior, rng)))
    return out


def work(case):
    """Queries, outputs and every visible cache cell once; two contractions per visible (query, key) pair."""
    D, Hq, Hkv, window = case["D"], case["Hq"], case["Hkv"], case["window"]
    cell = Hkv * (2 * D + 8)
    lengths = _lengths(case)
    tokens = sum(q for q, _ in lengths)
    if case["op"] == "write":   # 16-bit keys and values in, cells out; absmax, divide, round per element
        return {"bytes": tokens * (2 * Hkv * D * 2 + cell + 8), "flops": 6 * tokens * Hkv * D}
    keys = pairs = 0
    for q, n in lengths:
        keys += n if not window else min(n, window + q - 1)
        if not window:
            pairs += q * (n - q) + q * (q + 1) // 2
        else:
            pairs += sum(min(n - q + i + 1, window) for i in range(q))
    return {"bytes": keys * cell + 2 * tokens * Hq * D * 2, "flops": 4 * D * Hq * pairs}


def tolerance(case):
    """Cache bytes are exact.  Attention against the same call in 64 bits: 2.9e-3 at most in bf16 (1.7e-3 of
    it the rounding of the output) and 2.7e-4 in fp16 (2.1e-4), single values 2.1e-2 and 4.4e-3; four times that."""
    if case["op"] == "write":
        return "exact"
    return {"rel": 1.1e-2, "max": 8e-2} if case["dtype"] == "bf16" else {"rel": 1.1e-3, "max": 1.8e-2}


class _Cache:
    """A layer's paged cache in one of the two page layouts, and the op's four views of it."""

    def __init__(self, case, blocks, device):
        D, Hkv, page = case["D"], case["Hkv"], case["page"]
        cell = 2 * D + 8
        inner = (page, Hkv) if case["layout"] == "NHD" else (Hkv, page)
        self.storage = torch.zeros((blocks, *inner, cell), dtype=torch.uint8, device=device)
        cells, words = self.storage.view(torch.int8), self.storage.view(torch.float32)
        if case["layout"] == "HND":
            cells, words = cells.transpose(1, 2), words.transpose(1, 2)
        self.k, self.v = cells[..., :D], cells[..., D + 4:2 * D + 4]
        self.k_scale, self.v_scale = words[..., D // 4], words[..., D // 2 + 1]
        self.views = host.CacheViews.from_tensors(self.k, self.v, self.k_scale, self.v_scale)
        self.slots, self.shape = blocks * page, (Hkv, D)

    def fill(self, gen, device):
        """Normally distributed keys and values, quantised by the framework's own writer."""
        step = max(1, _WRITE_STEP // self.shape[0])
        for s0 in range(0, self.slots, step):
            n = min(step, self.slots - s0)
            kv = torch.randn((2, n, *self.shape), generator=gen, device=device, dtype=torch.bfloat16)
            host.write_kv(kv[0], kv[1], self.views, torch.arange(s0, s0 + n, device=device))


def prepare(case, seed):
    """A layer's cache, block table and lengths, and the call's tensors, plan and workspace."""
    device = torch.device("cuda")
    gen = torch.Generator(device=device).manual_seed(seed)
    D, Hq, Hkv, page, dtype = case["D"], case["Hq"], case["Hkv"], case["page"], _DTYPES[case["dtype"]]
    lengths = _lengths(case)
    q_lens, seq_lens = [q for q, _ in lengths], [n for _, n in lengths]
    R, T = len(lengths), sum(q_lens)

    pages = [-(-n // page) for n in seq_lens]
    cache = _Cache(case, sum(pages), device)
    order = torch.randperm(sum(pages), generator=gen, device=device).to(torch.int32)
    block_table = torch.zeros((R, max(pages)), dtype=torch.int32, device=device)
    for r, ids in enumerate(order.split(pages)):
        block_table[r, :pages[r]] = ids

    if case["op"] == "write":
        slots = []
        for r, (q, n) in enumerate(lengths):
            at = torch.arange(n - q, n, device=device)
            slots.append(block_table[r, at // page].long() * page + at % page)
        kv = torch.randn((2, T, Hkv, D), generator=gen, device=device).to(dtype)
        return dict(op="write", key=kv[0], value=kv[1], cache=cache, slots=torch.cat(slots))

    cache.fill(gen, device)
    longest = max(q_lens)
    if case["kind"] == "decode":
        reserved = planner.workspace_token_splits(max_num_seqs=R, q_dec_max=longest, Hkv=Hkv, D=D, num_sms=_sms(device))
    elif case["kind"] == "mixed":   # its long decode requests only balance if they may be cut
        reserved = 8 * T
    else:
        reserved = 0
    plan = planner.plan_launch(num_tokens=T, num_reqs=R, max_query_len=longest, G=Hq // Hkv, Hkv=Hkv, D=D,
                               num_sms=_sms(device), is_prefill=case["kind"] != "decode", ws_token_splits=reserved,
                               window=case["window"])
    starts = torch.tensor([0] + q_lens, device=device).cumsum(0).to(torch.int32)
    q = torch.randn((T, Hq, D), generator=gen, device=device).to(dtype)
    return dict(op="attention", cache=cache, args=(
        torch.zeros_like(q), q, cache.k, cache.v, cache.k_scale, cache.v_scale, block_table,
        torch.tensor(seq_lens, dtype=torch.int32, device=device), starts, longest, plan.wm, plan.num_splits,
        D ** -0.5, torch.empty(plan.ws_o_shape, dtype=torch.float32, device=device),
        torch.empty(plan.ws_lse_shape, dtype=torch.float32, device=device), case["window"], True))


def _sms(device):
    return torch.cuda.get_device_properties(device).multi_processor_count


def run(state):
    if state["op"] == "write":
        host.write_kv(state["key"], state["value"], state["cache"].views, state["slots"])
        return state["cache"].storage
    ops.pth_flash_attn_fwd(*state["args"])
    return state["args"][0]
