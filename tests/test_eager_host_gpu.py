"""The C++ short cut of eager calls against the Python path over the custom ops (which a torch function mode
selects): the same bits, and every call that is not plainly eager is left to the Python path."""
import pytest
import torch
from torch.overrides import TorchFunctionMode

import parallax_b200 as plx
from parallax_b200 import _cabi, ops

pytestmark = pytest.mark.gpu


class PythonPath(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def randn(*shape, dtype=torch.bfloat16, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed + sum(shape))).to(dtype).cuda()


class Recorder:
    """The C++ host side, with a note of which of its entry points answered."""

    def __init__(self, host):
        self.host, self.answered = host, set()

    def __getattr__(self, name):
        def entry(*args):
            res = getattr(self.host, name)(*args)
            if res is not None and res is not False:
                self.answered.add(name)
            return res

        return entry


def both(call, by):
    """`call` by the short cut -- the entry points `by` answer, and no others -- and by the Python path."""
    recorder = Recorder(_cabi.host())
    with pytest.MonkeyPatch.context() as patch:
        patch.setattr(_cabi, "_host", recorder)
        fast = call()
    assert recorder.answered == by
    with PythonPath():
        slow = call()
    for a, b in zip(fast, slow):
        assert a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b)
    return fast


@pytest.mark.parametrize("layout,window,dtype,d", [("BHLD", -1, torch.bfloat16, 128), ("BLHD view", 50, torch.float16, 64), ("packed", -1, torch.bfloat16, 64)])
def test_training(layout, window, dtype, d):
    hq, hkv, n = 4, 2, 200
    if layout == "BHLD":
        mk = lambda h, s: randn(2, h, n, d, dtype=dtype, seed=s)
        call = lambda *x: plx.parallax_func(*x, window_size_left=window)
    elif layout == "BLHD view":
        mk = lambda h, s: randn(2, n, h, d, dtype=dtype, seed=s).transpose(1, 2)
        call = lambda *x: plx.parallax_func(*x, 0.1, window)
    else:
        mk = lambda h, s: randn(1, n, h, d, dtype=dtype, seed=s)
        cu = torch.tensor([0, 3, 130, n], dtype=torch.int32, device="cuda")
        call = lambda *x: plx.parallax_varlen_func(*x, cu_seqlens=cu)
    leaves = [mk(h, s).requires_grad_(True) for s, h in enumerate((hq, hq, hkv, hkv))]
    go = mk(hq, 9)

    def step():
        o = call(*leaves)
        return (o.detach(), *torch.autograd.grad(o, leaves, go))

    by = {"train", "train_ready"}
    both(step, by)
    both(lambda: (call(*leaves[:3], leaves[3].detach()).detach(),), by)
    with torch.no_grad():
        both(lambda: (call(*leaves),), by)
    with torch.inference_mode():
        both(lambda: (call(*leaves),), by)
        both(lambda: (call(*[x.clone() for x in leaves]),), by)
    # a gradient in another layout, saved-tensor hooks, and a recorded backward
    o = call(*leaves)
    want = torch.autograd.grad(o, leaves, go, retain_graph=True)
    other = torch.empty(go.shape[::-1], dtype=dtype, device="cuda").permute(3, 2, 1, 0).copy_(go)
    assert all(torch.equal(a, b) for a, b in zip(want, torch.autograd.grad(o, leaves, other, retain_graph=True)))
    recorded = torch.autograd.grad(o, leaves, go, create_graph=True)
    assert all(torch.equal(a, b) for a, b in zip(want, recorded))
    with pytest.raises(RuntimeError):
        torch.autograd.grad(recorded[0].float().sum(), leaves[0])
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(1) or t.cpu(), lambda t: t.cuda()):
        o = call(*leaves)
    assert len(packed) >= 7
    got = torch.autograd.grad(o, leaves, go)
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    # an input overwritten in place is noticed
    o = call(*leaves)
    with torch.no_grad():
        leaves[0].mul_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(o, leaves, go)


@pytest.mark.parametrize("hq,hkv,page", [(8, 8, 0), (8, 2, 0), (8, 2, 32)])
def test_decode_and_prefill(hq, hkv, page):
    bsz, n, d = 3, 320, 128
    k, v = (randn(bsz * n // page + 2, page, hkv, d, seed=s) if page else randn(bsz, n, hkv, d, seed=s) for s in (1, 2))
    table = torch.randperm(bsz * n // page + 2)[:bsz * n // page].view(bsz, -1).int().cuda() if page else None
    t32 = lambda *x: torch.tensor(x, dtype=torch.int32, device="cuda")
    for lq in (1, 7):
        q, r = randn(bsz, lq, hq, d, seed=3), randn(bsz, lq, hq, d, seed=4)
        call = lambda **args: (plx.parallax_attn_with_kvcache(q, r, k, v, page_table=table, **args),)
        for args in (dict(), dict(seqused_k=t32(300, 7, 320)), dict(window_size=40, scale=0.2)):
            both(lambda: call(**args), {"attend"})
        both(lambda: call(window_size=(40, 0)), set())
        with torch.inference_mode():
            both(lambda: call(seqused_k=t32(300, 7, 320)), {"attend"})
        for bad in (t32(0, 7, 320), t32(1, 321, 7), t32(-5, 10 ** 9, 9)):
            with pytest.raises(ValueError, match="seqused_k"):
                plx.parallax_attn_with_kvcache(q, r, k, v, page_table=table, seqused_k=bad)
        if lq > 1:
            with pytest.raises(ValueError, match="L_q"):
                plx.parallax_attn_with_kvcache(q, r, k, v, page_table=table, seqused_k=t32(300, lq - 1, 320))
    if not page:
        q, r = randn(bsz, 1, hq, d, seed=3), randn(bsz, 1, hq, d, seed=4)
        for args in (dict(), dict(cache_start=t32(0, 5, 320)), dict(seqused_k=t32(300, 7, 320), window_size_left=33), dict(qk_scale=0.3)):
            both(lambda: (plx.parallax_decode(q, r, k, v, **args),), {"decode"})
        with torch.inference_mode():
            both(lambda: (plx.parallax_decode(q, r, k, v),), {"decode"})


def test_what_is_left_to_the_python_path():
    host = _cabi.host()
    q = randn(1, 4, 64, 64)
    scalars = (0.125, -1, ops.BHLD, None)
    assert host.train(q, q, q, q, *scalars) is not None
    assert host.train(q.cpu(), q, q, q, *scalars) is None
    assert host.train(q.float(), q, q, q, *scalars) is None
    assert host.train(q.as_subclass(type("Sub", (torch.Tensor,), {})), q, q, q, *scalars) is None
    assert host.train(q[..., 1:], q, q, q, *scalars) is None
    assert host.train(q, q, q, randn(1, 4, 64, 64).transpose(1, 2).contiguous().transpose(1, 2), *scalars) is None
    assert host.train(q, q, q, q, 0.125, -2, ops.BHLD, None) is None
    assert host.train(q, q, q, q, 1, -1, ops.BHLD, None) is None
    with PythonPath():
        assert host.train(q, q, q, q, *scalars) is None
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(q, torch.ones_like(q))
        assert host.train(dual, q, q, q, *scalars) is None
    torch.func.vmap(lambda x: (_ for _ in ()).throw(AssertionError) if host.train(x, q, q, q, *scalars) is not None else x)(q[None])
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    with Mode():
        assert host.train(q, q, q, q, *scalars) is None
    x = randn(1, 1, 4, 64).requires_grad_(True)
    kv = randn(1, 64, 4, 64)
    assert host.decode(x, x, kv, kv, None, -1, None, None, None) is None
    assert host.decode(x.detach(), x.detach(), kv, kv, None, -1, None, None, None) is not None


def test_two_streams_at_once():
    """A workspace belongs to its stream: two streams that decode one shape at the same time do not disturb each other."""
    q, r, k, v = randn(4, 1, 8, 128), randn(4, 1, 8, 128, seed=1), randn(4, 9000, 2, 128, seed=2), randn(4, 9000, 2, 128, seed=3)
    want = [plx.parallax_decode(q * s, r, k, v) for s in (1, 2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    got = [[], []]
    for _ in range(20):
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                got[i].append(plx.parallax_decode(q * (i + 1), r, k, v))
    torch.cuda.synchronize()
    assert all(torch.equal(x, want[i]) for i in range(2) for x in got[i])


@pytest.mark.parametrize("bsz,h,d", [(1, 1, 64), (4, 8, 128), (512, 1, 64), (513, 1, 64)])
def test_staging_of_a_captured_step(bsz, h, d):
    """q, r and the lengths of a step reach the buffers of the captured launch: in one launch (up to 512 rows, host
    lengths), and by the copies where that does not apply."""
    gd = plx.GraphedDecode(bsz, h, max_kv_len=96, head_dim=d)
    gd.k.copy_(randn(bsz, 96, h, d, seed=1))
    gd.v.copy_(randn(bsz, 96, h, d, seed=2))
    q, r = randn(bsz, 1, h, d, seed=3), randn(bsz, 1, h, d, seed=4)
    lens = [1 + (i * 31) % 96 for i in range(bsz)]
    for given in (lens, tuple(lens), torch.tensor(lens, dtype=torch.int32, device="cuda")):
        gd.q.zero_(), gd.r.zero_(), gd.cache_seqlens.fill_(1)
        before = _cabi.launch_count()
        out = gd(q=q, r=r, cache_seqlens=given).clone()
        assert _cabi.launch_count() - before == (1 if given is lens and bsz <= 512 else 0)
        assert torch.equal(gd.q, q) and torch.equal(gd.r, r) and gd.cache_seqlens.tolist() == lens
        assert torch.equal(out, plx.parallax_decode(q, r, gd.k, gd.v, seqused_k=gd.cache_seqlens))
    gd(q=r)                                                    # the others stay
    assert torch.equal(gd.q, r) and torch.equal(gd.r, r) and gd.cache_seqlens.tolist() == lens
    gd(q=q.transpose(0, 1).contiguous().transpose(0, 1), cache_seqlens=96)
    assert torch.equal(gd.q, q) and gd.cache_seqlens.tolist() == [96] * bsz
    gd(r=q.float())                                            # converted, as copy_ does
    assert torch.equal(gd.r, q)
    for bad in ([0] * bsz, [97] * bsz, 0, 97):
        with pytest.raises(ValueError, match="out of range"):
            gd(cache_seqlens=bad)
    assert gd.cache_seqlens.tolist() == [96] * bsz


def test_a_profiler_sees_the_ops():
    """A call by the short cut shows up in a profile under the name of the op it stands for, with its input shapes."""
    from torch.profiler import ProfilerActivity, profile

    leaves = [randn(1, 2, 128, 64, seed=s).requires_grad_(True) for s in range(4)]
    q, kv = randn(2, 1, 4, 64), randn(2, 128, 4, 64)
    chunk = randn(2, 3, 4, 64)
    with profile(activities=[ProfilerActivity.CPU], record_shapes=True) as prof:
        plx.parallax_func(*leaves).sum().backward()
        plx.parallax_decode(q, q, kv, kv)
        plx.parallax_attn_with_kvcache(chunk, chunk, kv, kv)
    shapes = {e.name: e.input_shapes for e in prof.events() if e.name.startswith("plx::")}
    assert shapes["plx::train_fwd"][:4] == [[1, 2, 128, 64]] * 4
    assert shapes["plx::train_bwd"][0] == [1, 2, 128, 64]
    assert shapes["plx::decode_out"][:3] == [[2, 1, 4, 64], [2, 1, 4, 64], [2, 128, 4, 64]]
    assert shapes["plx::train_extend"][0] == [2, 3, 4, 64]
