"""Decode launches that overlap the end of the kernel before them, the grouped-head sweep at the edges of its tiles and
stages, and the lengths that reach the host beside a launch."""
import pytest
import torch

import parallax_b200 as plx
from oracle import parallax_oracle as orc
from parallax_b200 import _cabi
from tests._util import DECODE_MAX_REL, DECODE_REL_L2, assert_close, seeded_bf16

pytestmark = pytest.mark.gpu


def inputs(bsz, hq, hkv, t, d=128, seed=0):
    return [seeded_bf16(s, seed + i).cuda() for i, s in enumerate(((bsz, 1, hq, d), (bsz, 1, hq, d), (bsz, t, hkv, d), (bsz, t, hkv, d)))]


# (hq, hkv, page): one q head per kv head in split groups and by warps, grouped heads, grouped heads over pages
@pytest.mark.parametrize("bsz,hq,hkv,t,page", [(1, 8, 8, 700, 0), (12, 8, 8, 3000, 0), (2, 16, 4, 900, 0), (3, 8, 2, 1024, 16)])
def test_calls_that_feed_each_other(bsz, hq, hkv, t, page):
    """Each call reads what the kernels right before it wrote -- its query, a cache entry, the lengths -- and its
    workspace is the one the call before has just left: the answers are those of calls with the GPU idle in between."""
    def chain(wait):
        q, r, k, v = inputs(bsz, hq, hkv, t)
        table = None
        if page:
            order = torch.randperm(bsz * t // page, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda()
            table = order.view(bsz, t // page)
            k, v = (x.view(-1, page, hkv, 128).contiguous() for x in (k, v))
        got = []
        for i in range(12):
            lens = torch.full((bsz,), t - i, dtype=torch.int32, device="cuda")
            o = plx.parallax_attn_with_kvcache(q, r, k, v, page_table=table, seqused_k=lens if i % 3 else None)
            wait()
            k[:, i % k.shape[1]] = o[0, 0, :hkv]              # the next call sees it
            wait()
            q = (o * 3).to(o.dtype)
            wait()
            o = plx.parallax_attn_with_kvcache(q, q, k, v, page_table=table)
            wait()
            q = plx.parallax_attn_with_kvcache(o, q, k, v, page_table=table)    # straight from call to call
            wait()
            got += [o, q]
        return got

    want = chain(torch.cuda.synchronize)
    for x, y in zip(chain(lambda: None), want):
        assert torch.equal(x, y)


@pytest.mark.parametrize("bsz,n,h,d,hkv", [(1, 1500, 8, 128, 8), (2, 900, 16, 64, 4), (1, 2600, 8, 128, 2)])
def test_a_decode_call_right_behind_a_backward(bsz, n, h, d, hkv):
    """dk/dv lets dq/dr in early and dq/dr waits for it at its end: a decode launch behind them, which comes early too, reads dk and
    dv as its caches and a row of dq and of dr as its query, with no synchronisation in between."""
    gen = torch.Generator(device="cuda").manual_seed(3)

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda").bfloat16()

    leaves = [randn(bsz, n, heads, d).requires_grad_(True) for heads in (h, h, hkv, hkv)]
    o = plx.parallax_varlen_func(*leaves)
    grads = [randn(bsz, n, h, d) for _ in range(6)]

    def chain(wait):
        got = []
        for go in grads:
            dq, dr, dk, dv = torch.autograd.grad(o, leaves, go, retain_graph=True)
            wait()
            got.append(plx.parallax_decode(dq[:, -1:], dr[:, -1:], dk, dv))
            wait()
            got.append(plx.parallax_decode(got[-1], dr[:, :1], dv, dk))
        return got

    want = chain(torch.cuda.synchronize)
    torch.cuda.synchronize()
    for x, y in zip(chain(lambda: None), want):
        assert torch.equal(x, y)


@pytest.mark.parametrize("hq,hkv,d", [(4, 1, 128), (18, 1, 128), (32, 8, 64)])
def test_grouped_heads_at_the_edges_of_tiles_and_stages(hq, hkv, d, monkeypatch):
    """0 to 5 tiles of 16 keys per warp (three stages), the last one whole, of one key and one key short."""
    monkeypatch.setenv("PLX_DECODE_SPLITS", "2")
    for t in (1, 15, 16, 17, 33, 47, 48, 63, 64, 65, 95, 96, 97, 129, 160):
        q, r, k, v = inputs(1, hq, hkv, t, d, seed=t)
        o = plx.parallax_decode(q, r, k, v)
        assert_close(o.float().cpu(), orc.decode(*[x.cpu() for x in (q, r, k, v)]), DECODE_REL_L2, DECODE_MAX_REL, f"{hq}:{hkv} {t}")
        if t % 16 == 0:
            table = torch.arange(t // 16, device="cuda", dtype=torch.int32).flip(0).view(1, -1)
            kp, vp = (x.view(t // 16, 16, hkv, d).flip(0).contiguous() for x in (k, v))
            assert torch.equal(plx.parallax_attn_with_kvcache(q, r, kp, vp, page_table=table), o)


# 9, 12, 16 and 18 q heads per kv head: rows of the second half of a tile, all or some of them; 2 and 8: half a tile
@pytest.mark.parametrize("hq,hkv,d", [(9, 1, 128), (12, 1, 64), (16, 1, 128), (36, 2, 64), (64, 8, 128), (4, 2, 64)])
def test_grouped_heads_whose_records_meet_in_memory(hq, hkv, d, monkeypatch):
    """Splits that leave one warp of a row in a CTA, and 1 to 32 records a row to merge there: either side of 8 and 16."""
    for bsz, t, splits in ((4, 1000, 15), (3, 400, 9), (2, 1100, 17), (1, 4100, 63), (1, 4100, 65), (1, 2100, 128), (1, 2100, 130), (1, 4100, 256)):
        monkeypatch.setenv("PLX_DECODE_SPLITS", str(splits))
        q, r, k, v = inputs(bsz, hq, hkv, t, d, seed=splits)
        o = plx.parallax_decode(q, r, k, v)
        assert_close(o.float().cpu(), orc.decode(*[x.cpu() for x in (q, r, k, v)]), DECODE_REL_L2, DECODE_MAX_REL, f"{hq}:{hkv} {bsz} {t} {splits}")


@pytest.mark.parametrize("bsz,hq,hkv", [(1, 8, 8), (64, 8, 8), (64, 8, 2), (65, 8, 8)])
def test_a_graphed_step_in_one_launch(bsz, hq, hkv):
    """Up to 64 rows the inputs and the sweep are one launch; its buffers and answer are those of the copies and the replay."""
    t = 400
    gd = plx.GraphedDecode(bsz, hq, max_kv_len=t, H_kv=hkv)
    q, r, k, v = inputs(bsz, hq, hkv, t)
    lens = [t - (i * 37) % (t - 1) for i in range(bsz)]
    want = gd(q=q, r=r, k=k, v=v, cache_seqlens=torch.tensor(lens)).clone()
    assert torch.equal(gd.replay(), want)
    for t_ in (gd.q, gd.r, gd.out, gd.cache_seqlens):
        t_.zero_()
    gd.cache_seqlens += 1
    before = _cabi.launch_count()
    assert torch.equal(gd(q=q, r=r, cache_seqlens=lens), want)
    assert _cabi.launch_count() == before + 1
    assert torch.equal(gd.q, q) and torch.equal(gd.r, r) and gd.cache_seqlens.tolist() == lens
    gd.out.zero_()
    assert torch.equal(gd.replay(), want)
    assert torch.equal(gd(), want)
    # an input that shares memory with the output or the buffers
    two = gd(q=gd.out).clone()
    assert torch.equal(gd.q, want) and torch.equal(gd.replay(), two)
    assert torch.equal(gd(q=gd.r, r=gd.q), gd.replay())


@pytest.mark.parametrize("bsz,hq,hkv,d,dtype,window,static", [
    (4, 8, 8, 128, torch.bfloat16, None, False), (64, 8, 8, 64, torch.float16, 50, False), (3, 36, 2, 128, torch.bfloat16, None, False),
    (16, 12, 1, 64, torch.bfloat16, 70, False), (20, 32, 8, 128, torch.float16, None, False), (2, 16, 16, 128, torch.bfloat16, None, True),
    (5, 8, 2, 128, torch.bfloat16, 33, True), (65, 8, 8, 128, torch.bfloat16, None, False)])
def test_which_way_a_step_goes(bsz, hq, hkv, d, dtype, window, static):
    """Up to 64 rows a step leaves its graph alone, beyond them it replays it once; either way its buffers and answer are those of
    copies and a replay, with q, r and lengths given or only some of them, with lengths that are dealt out (far apart), windows,
    two groups of heads per kv head, and at a static length."""
    t = 900
    gd = plx.GraphedDecode(bsz, hq, **({"kv_len": t} if static else {"max_kv_len": t}), head_dim=d, H_kv=hkv, dtype=dtype, window_size=window)
    ref = plx.GraphedDecode(bsz, hq, **({"kv_len": t} if static else {"max_kv_len": t}), head_dim=d, H_kv=hkv, dtype=dtype, window_size=window)
    q, r, k, v = (x.to(dtype) for x in inputs(bsz, hq, hkv, t, d))
    for g in (gd, ref):
        g.k.copy_(k)
        g.v.copy_(v)
    graph, replays = gd.graph, []

    class Counted:
        def replay(self):
            replays.append(1)
            graph.replay()

    gd.graph = Counted()
    lens = [t if i % 5 == 0 else 1 + (i * 37) % 200 for i in range(bsz)]
    steps = [dict(q=q, r=r), dict(r=q), dict(q=r), dict()]
    if not static:
        steps += [dict(q=q, r=r, cache_seqlens=lens), dict(r=q), dict(cache_seqlens=lens[::-1]), dict(q=r, cache_seqlens=t)]
    for i, given in enumerate(steps):
        for name in ("q", "r"):
            if name in given:
                getattr(ref, name).copy_(given[name])
        if "cache_seqlens" in given:
            n = given["cache_seqlens"]
            ref.cache_seqlens.copy_(torch.tensor(n if isinstance(n, list) else [n] * bsz, dtype=torch.int32))
        want = ref.replay()
        replays.clear()
        gd.out.zero_()
        got = gd(**given)
        assert len(replays) == (0 if bsz <= 64 else 1), i
        assert torch.equal(got, want), i
        for x, y in ((gd.q, ref.q), (gd.r, ref.r), (gd.cache_seqlens, ref.cache_seqlens)):
            assert (x is None and y is None) or torch.equal(x, y), i


def test_inputs_that_share_memory_but_not_a_storage():
    """The buffers of a step behind a zero-copy import have storages of their own: the answers are still those of copies to q,
    then to r, then the sweep."""
    gd = plx.GraphedDecode(4, 8, max_kv_len=400)
    q, r, k, v = inputs(4, 8, 8, 400)
    gd(k=k, v=v)

    def foreign(x):
        y = torch.from_dlpack(x)
        assert y.data_ptr() == x.data_ptr() and not torch._C._is_alias_of(x, y)
        return y

    def same(got, q, r):
        assert torch.equal(gd.q, q) and torch.equal(gd.r, r)
        assert torch.equal(got, plx.parallax_decode(q, r, k, v))

    same(gd(q=q, r=foreign(gd.q)), q, q)
    gd(q=q, r=r)
    same(gd(q=foreign(gd.r), r=q), r, q)
    want = gd(q=q, r=r).clone()
    same(gd(q=foreign(gd.out)), want, r)
    same(gd(q=foreign(gd.k[:, 5:6]).contiguous()), k[:, 5:6], r)


@pytest.mark.parametrize("through", [lambda x: x, torch.from_dlpack])
def test_inputs_are_copied_in_the_order_of_the_arguments(through):
    """q, r, k, v: a q or an r that is part of the object's own caches is read before new caches arrive, and a k or a v that is
    the object's q after the new q has."""
    t = 400
    (q, r, k, v), (q2, _, k2, v2) = inputs(4, 8, 8, t), inputs(4, 8, 8, t, seed=50)

    def step(**given):
        gd = plx.GraphedDecode(4, 8, max_kv_len=t)
        gd(q=q, r=r, k=k, v=v)
        out = gd(**{n: through(x(gd)) if callable(x) else x for n, x in given.items()})
        return gd, out

    def holds(got, q, r, k, v):
        gd, out = got
        for x, y in ((gd.q, q), (gd.r, r), (gd.k, k), (gd.v, v), (out, plx.parallax_decode(q, r, k, v))):
            assert torch.equal(x, y)

    holds(step(q=lambda gd: gd.k[:, 7:8], k=k2), k[:, 7:8], r, k2, v)
    holds(step(r=lambda gd: gd.v[:, :1], k=k2, v=v2, cache_seqlens=t), q, v[:, :1], k2, v2)
    holds(step(q=q2, k=lambda gd: gd.q.expand(4, t, 8, 128)), q2, r, q2.expand(4, t, 8, 128), v)
    holds(step(q=q2, r=lambda gd: gd.q, k=k2, v=lambda gd: gd.k), q2, q2, k2, k2)
    holds(step(q=q2, k=k2, v=v2), q2, r, k2, v2)          # nothing shared: one launch behind the copies


@pytest.mark.parametrize("bsz,hq,hkv,t,lq", [(2, 32, 8, 4096, 1), (8, 16, 16, 2048, 1), (2, 32, 8, 700, 64)])
def test_lengths_beside_a_long_launch(bsz, hq, hkv, t, lq):
    """The lengths are checked as they are in stream order -- written by a kernel that is still to run when the call is made,
    on any stream -- and a length out of range raises, whichever row it is in."""
    _, _, k, v = inputs(bsz, hq, hkv, t)
    q = seeded_bf16((bsz, lq, hq, 128), 9).cuda()
    lens = torch.full((bsz,), t, dtype=torch.int32, device="cuda")
    want = plx.parallax_attn_with_kvcache(q, q, k, v, seqused_k=lens)
    big = torch.randn(4096, 4096, device="cuda")
    for stream in (torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()):
        with torch.cuda.stream(stream):
            for row in range(bsz):
                lens.fill_(t)
                for _ in range(8):
                    big @ big
                bad = lens.clone()
                bad[row] = t + 1
                with pytest.raises(ValueError):
                    plx.parallax_attn_with_kvcache(q, q, k, v, seqused_k=bad)
                bad[row] = t
                assert torch.equal(plx.parallax_attn_with_kvcache(q, q, k, v, seqused_k=bad), want)
        torch.cuda.synchronize()


def test_lengths_beside_launches_on_many_streams():
    """More streams than the library keeps one beside: the answers and the errors are the same, and none is made anew each time."""
    q, r, k, v = inputs(2, 32, 8, 4096)
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(24)]
    assert len({s.cuda_stream for s in streams}) > 40
    lens = torch.tensor([4096, 3000], dtype=torch.int32, device="cuda")
    bad = torch.tensor([4096, 4097], dtype=torch.int32, device="cuda")
    want = plx.parallax_attn_with_kvcache(q, r, k, v, seqused_k=lens)
    torch.cuda.synchronize()
    made = None
    for _ in range(3):
        for s in streams:
            with torch.cuda.stream(s):
                got = plx.parallax_attn_with_kvcache(q, r, k, v, seqused_k=lens)
                with pytest.raises(ValueError):
                    plx.parallax_attn_with_kvcache(q, r, k, v, seqused_k=bad)
            s.synchronize()
            assert torch.equal(got, want)
        if made is not None:
            assert _cabi.host().side_streams_made() == made
        made = _cabi.host().side_streams_made()
