"""The workloads whose speed this library is kept to: what a training job and a serving loop ask of the
attention operator, through its public entry points.

A case is a dict of plain values.  `kind` says which entry point it calls:

* ``train``   ``parallax_func`` forward and the backward of all four inputs (dense, causal)
* ``varlen``  ``parallax_varlen_func`` forward and backward on packed sequences
* ``decode``  ``parallax_decode``: one token per row against a dense cache
* ``kvcache`` ``parallax_attn_with_kvcache``: one token per row (``lq`` = 1), or a chunk of ``lq`` > 1 new
  tokens per row (chunked prefill), against a dense or a paged cache
* ``graph``   ``GraphedDecode``: the captured decode step of a serving loop

Inputs are iid N(0, 1), as in the configurations the operator is quoted on.  Row lengths and sequence lengths
belong to the case (they decide its work); everything else comes from the seed.
"""
import math
import random

import torch

import parallax_b200 as plx

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def listed():
    return [
        # one user, a short context, eager calls: the smallest call there is
        _decode("decode_b1_t1024", b=1, hq=8, hkv=8, t=1024),
        # a serving loop's captured step: a few users whose lengths differ, the cache sized for the longest
        dict(name="graph_b4_t4096", kind="graph", b=4, hq=8, hkv=8, t=4096, d=128, dtype="bf16", window=-1, ragged=True),
        # a full batch at a short context, one query head per kv head
        _decode("decode_b32_t1024", b=32, hq=8, hkv=8, t=1024),
        # the largest dense cache: a pure sweep of the memory
        _decode("decode_b64_t32768", b=64, hq=8, hkv=8, t=32768),
        # grouped-query heads, one user with a long chat
        _kvcache("kvcache_gqa_b1_t8192", b=1, hq=32, hkv=8, t=8192),
        # grouped-query heads, a batch over a paged cache, every row with a length of its own
        _kvcache("kvcache_gqa_paged_b16_t8192", b=16, hq=32, hkv=8, t=8192, page=64, ragged=True),
        # chunked prefill: four rows bring 512 new tokens each to paged caches of different lengths
        _kvcache("prefill_gqa_paged_b4_lq512_t4096", b=4, hq=32, hkv=8, t=4096, lq=512, page=64, ragged=True),
        # a small training step, where launches and host work show
        _train("train_b2_h8_l1024", b=2, hq=8, hkv=8, l=1024),
        # the training step the operator is quoted on ...
        _train("train_b8_h16_l4096", b=8, hq=16, hkv=16, l=4096),
        # ... and its head_dim 64 variant, in the other data type
        _train("train_b8_h16_l4096_d64_fp16", b=8, hq=16, hkv=16, l=4096, d=64, dtype="fp16"),
        # pre-training on packed documents: 65536 tokens in sequences of 64 to 8192
        _varlen("varlen_65536", hq=16, hkv=16, total=65536, lo=64, hi=8192),
        # fine-tuning on short packed samples, grouped-query heads
        _varlen("varlen_short_gqa", hq=16, hkv=4, total=32768, lo=1, hi=256),
    ]


def draw(rng):
    """One more case of the same ranges; none costs more than the largest listed one of its kind."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    d = rng.choice((128, 128, 128, 64))
    dtype = rng.choice(("bf16", "bf16", "fp16"))
    kind = rng.choice(("decode", "decode", "kvcache", "kvcache", "prefill", "graph", "train", "train", "varlen", "varlen"))
    if kind in ("decode", "kvcache", "graph"):
        hq, hkv = rng.choice(((8, 8), (16, 16), (32, 8), (16, 2)) if kind != "kvcache" else ((32, 8), (16, 4), (16, 2), (8, 8)))
        t = log_int(200, 32768)
        b = log_int(1, max(1, min(64, 2 ** 24 // (t * hkv))))
        window = rng.choice((-1, -1, -1, max(1, t // 4)))
        if kind == "decode":
            return _decode(None, b=b, hq=hq, hkv=hkv, t=t, d=d, dtype=dtype, window=window, start=rng.random() < 0.3)
        if kind == "graph":
            return dict(kind="graph", b=b, hq=hq, hkv=hkv, t=t, d=d, dtype=dtype, window=window, ragged=True)
        page = rng.choice((0, 16, 64, 256))
        return _kvcache(None, b=b, hq=hq, hkv=hkv, t=-(-t // page) * page if page else t, page=page, d=d, dtype=dtype,
                        window=window, ragged=rng.random() < 0.7)
    if kind == "prefill":
        hq, hkv = rng.choice(((32, 8), (16, 4), (8, 8)))
        lq = log_int(8, 1024)
        t = log_int(2 * lq, 8192)
        b = log_int(1, 8)
        page = rng.choice((0, 16, 64, 256))
        return _kvcache(None, b=b, hq=hq, hkv=hkv, t=-(-t // page) * page if page else t, lq=lq, page=page, d=d, dtype=dtype,
                        ragged=rng.random() < 0.7)
    hq, hkv = rng.choice(((8, 8), (16, 16), (16, 4), (32, 8)))
    if kind == "train":
        l = log_int(100, 8192)
        b = log_int(1, max(1, min(16, 2 ** 31 // (l * l * hq))))
        return _train(None, b=b, hq=hq, hkv=hkv, l=l, d=d, dtype=dtype, window=rng.choice((-1, -1, -1, max(1, l // 4))))
    hi = log_int(128, 5000)
    return _varlen(None, hq=min(hq, 16), hkv=min(hkv, 16), total=log_int(8192, 65536), lo=1, hi=hi, d=d, dtype=dtype,
                   lens_seed=rng.randrange(1000))


def _named(name, case):
    return dict(name=name, **case) if name is not None else case


def _decode(name, *, b, hq, hkv, t, d=128, dtype="bf16", window=-1, start=False):
    return _named(name, dict(kind="decode", b=b, hq=hq, hkv=hkv, t=t, d=d, dtype=dtype, window=window, start=start))


def _kvcache(name, *, b, hq, hkv, t, lq=1, d=128, dtype="bf16", window=-1, page=0, ragged=False):
    return _named(name, dict(kind="kvcache", b=b, hq=hq, hkv=hkv, t=t, lq=lq, d=d, dtype=dtype, window=window, page=page,
                             ragged=ragged))


def _train(name, *, b, hq, hkv, l, d=128, dtype="bf16", window=-1):
    return _named(name, dict(kind="train", b=b, hq=hq, hkv=hkv, l=l, d=d, dtype=dtype, window=window))


def _varlen(name, *, hq, hkv, total, lo, hi, d=128, dtype="bf16", lens_seed=0):
    return _named(name, dict(kind="varlen", hq=hq, hkv=hkv, total=total, lo=lo, hi=hi, d=d, dtype=dtype, lens_seed=lens_seed))


def _row_lengths(case):
    """Active keys per batch row: all of the cache, or spread evenly from the longest row down to a third of it."""
    b, t, lq = case["b"], case["t"], case.get("lq", 1)
    if not case.get("ragged"):
        return [t] * b
    return [max(lq, t - (2 * t * i) // (3 * b)) for i in range(b)]


def _row_starts(case):
    """First valid key per batch row of a left-padded batch: up to a third of the cache is padding."""
    b, t = case["b"], case["t"]
    return [(t * i) // (3 * b) for i in range(b)] if case.get("start") else [0] * b


def _sequence_lengths(case):
    rng = random.Random(case["lens_seed"])
    lens, left = [], case["total"]
    while left > 0:
        n = min(left, rng.randint(case["lo"], case["hi"]))
        lens.append(n)
        left -= n
    return lens


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    kind, hq, hkv, d = case["kind"], case["hq"], case["hkv"], case["d"]

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)

    def ints(values):
        return torch.tensor(values, dtype=torch.int32, device="cuda")

    if kind in ("train", "varlen"):
        if kind == "train":
            qs, ks = (case["b"], hq, case["l"], d), (case["b"], hkv, case["l"], d)
        else:
            qs, ks = (1, case["total"], hq, d), (1, case["total"], hkv, d)
        leaves = [normal(*s).requires_grad_(True) for s in (qs, qs, ks, ks)]
        state = dict(case=case, leaves=leaves, grad=normal(*qs))
        if kind == "varlen":
            cu = [0]
            for n in _sequence_lengths(case):
                cu.append(cu[-1] + n)
            state["cu"] = ints(cu)
        return state

    b, t, lq = case["b"], case["t"], case.get("lq", 1)
    q, r = normal(b, lq, hq, d), normal(b, lq, hq, d)
    if kind == "graph":
        step = plx.GraphedDecode(b, hq, max_kv_len=t, head_dim=d, H_kv=hkv, dtype=dtype,
                                 window_size=None if case["window"] < 0 else case["window"])
        step.k.copy_(normal(b, t, hkv, d))
        step.v.copy_(normal(b, t, hkv, d))
        return dict(case=case, step=step, q=q, r=r, lens=_row_lengths(case))
    page = case.get("page", 0)
    state = dict(case=case, q=q, r=r, start=None, lens=None, table=None)
    if page:
        # a pool with a few spare pages, the rows' pages scattered over it
        per_row = t // page
        pool = b * per_row + 7
        state["k"], state["v"] = normal(pool, page, hkv, d), normal(pool, page, hkv, d)
        order = torch.randperm(pool, generator=gen, device="cuda")[:b * per_row]
        state["table"] = order.to(torch.int32).view(b, per_row)
    else:
        state["k"], state["v"] = normal(b, t, hkv, d), normal(b, t, hkv, d)
    if case.get("start"):
        state["start"] = ints(_row_starts(case))
    if case.get("ragged"):
        state["lens"] = ints(_row_lengths(case))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "train":
        o = plx.parallax_func(*state["leaves"], window_size_left=case["window"])
        return (o.detach(), *torch.autograd.grad(o, state["leaves"], state["grad"]))
    if kind == "varlen":
        o = plx.parallax_varlen_func(*state["leaves"], cu_seqlens=state["cu"])
        return (o.detach(), *torch.autograd.grad(o, state["leaves"], state["grad"]))
    if kind == "decode":
        return plx.parallax_decode(state["q"], state["r"], state["k"], state["v"], window_size_left=case["window"],
                                   cache_start=state["start"])
    if kind == "graph":
        return state["step"](q=state["q"], r=state["r"], cache_seqlens=state["lens"])
    return plx.parallax_attn_with_kvcache(state["q"], state["r"], state["k"], state["v"], page_table=state["table"],
                                          seqused_k=state["lens"],
                                          window_size=None if case["window"] < 0 else case["window"])


def _exact_heads(q, r, k, v, window, first=0):
    """The operator in 64 bits for some heads: q, r (heads, lq, d) at the last positions of k, v (heads, lk, d);
    keys before `first` are padding.  With S1 = q.k / sqrt(d), S2 = r.k and P = softmax(S1) over the visible keys
    the result is (1 + sum(P S2)) P v - (P S2) v."""
    lq, lk = q.shape[1], k.shape[1]
    at = torch.arange(lk - lq, lk, device=q.device).view(-1, 1)
    key = torch.arange(lk, device=q.device).view(1, -1)
    hidden = (key > at) | (key < first)
    if window >= 0:
        hidden = hidden | (key <= at - window)
    p = torch.softmax((q @ k.mT * q.shape[2] ** -0.5).masked_fill(hidden, -math.inf), dim=-1)
    ps2 = p * (r @ k.mT)
    return (1 + ps2.sum(-1, keepdim=True)) * (p @ v) - ps2 @ v


def _exact_sequence(q, r, k, v, window, first=0, grad=None):
    """`_exact_heads` for one sequence of 16-bit tensors (tokens, heads, d), a few kv heads at a time; with `grad`
    the gradients of the four inputs too."""
    hq, hkv = q.shape[1], k.shape[1]
    rep = hq // hkv
    step = max(1, 2 ** 26 // (q.shape[0] * k.shape[0] * rep))
    parts = []
    for h in range(0, hkv, step):
        n = min(step, hkv - h)
        x = [t[:, a:b].transpose(0, 1).double().requires_grad_(grad is not None)
             for t, a, b in ((q, h * rep, (h + n) * rep), (r, h * rep, (h + n) * rep), (k, h, h + n), (v, h, h + n))]
        with torch.set_grad_enabled(grad is not None):
            o = _exact_heads(x[0], x[1], *(t.repeat_interleave(rep, 0) for t in x[2:]), window, first)
        got = [o.detach()]
        if grad is not None:
            got += torch.autograd.grad(o, x, grad[:, h * rep:(h + n) * rep].transpose(0, 1).double())
        parts.append([t.transpose(0, 1) for t in got])
    return [torch.cat(t, 1) for t in zip(*parts)]


def exact(case, seed):
    """What `run` returns, in 64 bits and plain torch."""
    state, kind, window = prepare(case, seed), case["kind"], case["window"] if "window" in case else -1
    if kind == "train":
        x = [t.detach().transpose(1, 2) for t in (*state["leaves"], state["grad"])]
        rows = [_exact_sequence(*(t[i] for t in x[:4]), window, grad=x[4][i]) for i in range(case["b"])]
        return tuple(torch.stack(t).transpose(1, 2) for t in zip(*rows))
    if kind == "varlen":
        x = [t.detach()[0] for t in (*state["leaves"], state["grad"])]
        parts, at = [], 0
        for n in _sequence_lengths(case):
            parts.append(_exact_sequence(*(t[at:at + n] for t in x[:4]), window, grad=x[4][at:at + n]))
            at += n
        return tuple(torch.cat(t).unsqueeze(0) for t in zip(*parts))
    caches = (state["step"].k, state["step"].v) if kind == "graph" else (state["k"], state["v"])
    rows = []
    for i, (n, first) in enumerate(zip(_row_lengths(case), _row_starts(case))):
        if case.get("page"):
            k, v = (c[state["table"][i].long()].flatten(0, 1)[:n] for c in caches)
        else:
            k, v = (c[i, :n] for c in caches)
        rows.append(_exact_sequence(state["q"][i], state["r"][i], k, v, window, first)[0])
    return torch.stack(rows)


def _causal_pairs(lq, lk, window):
    """Visible (query, key) pairs of one head: the lq queries are the last positions of lk keys."""
    if window < 0 or window >= lk:
        return lq * lk - lq * (lq - 1) // 2
    return sum(min(lk - lq + i + 1, window) for i in range(lq))


def work(case):
    """Bytes: every input read once, every output written once (16-bit tensors).  Flops: the matrix products of
    the visible pairs, four forward (q.k, r.k and the two value sums) and eight more for the gradients."""
    kind, hq, hkv, d = case["kind"], case["hq"], case["hkv"], case["d"]
    if kind in ("train", "varlen"):
        if kind == "train":
            tokens = case["b"] * case["l"]
            pairs = case["b"] * _causal_pairs(case["l"], case["l"], case["window"])
        else:
            tokens = case["total"]
            pairs = sum(_causal_pairs(n, n, -1) for n in _sequence_lengths(case))
        # q, r, grad, o, dq, dr by query head; k, v, dk, dv by kv head
        return {"bytes": tokens * d * 2 * (6 * hq + 4 * hkv), "flops": 12 * 2 * pairs * hq * d}
    lq, window = case.get("lq", 1), case["window"]
    keys = pairs = 0
    for n, first in zip(_row_lengths(case), _row_starts(case)):
        lo = first if window < 0 else max(first, n - lq - window + 1)
        keys += n - max(lo, 0)
        pairs += n - max(lo, 0) if lq == 1 else _causal_pairs(lq, n, window)
    return {"bytes": 2 * d * (2 * keys * hkv + 3 * case["b"] * lq * hq), "flops": 4 * 2 * pairs * hq * d}


def tolerance(case):
    # Four times the distance from the same path in 64 bits: 2.9e-3 (bf16) and 3.2e-4 (fp16) are the largest
    # seen over the outputs and gradients of every kind, at 100 to 32768 keys.
    return {"rel": 1.2e-2 if case["dtype"] == "bf16" else 1.3e-3}
