"""The two plans of the backward that depend on the problem.  head_dim 64, whose element-wise groups take the streamed tiles in
turn: work items of every small tile count in a row on one CTA, so that items begin with either group and a group has no
tile of some of them.  head_dim 128, whose dq/dr keeps dO in shared memory where items see few keys and in tensor memory else."""
import pytest
import torch

import parallax_b200 as plx
from oracle import parallax_oracle as orc
from tests._util import TRAIN_MAX_REL, TRAIN_REL_L2, assert_close
from tests import test_varlen_gpu as tv

pytestmark = pytest.mark.gpu


# lengths either side of the 64-wide streamed tiles and the 128-wide resident ones: 1 to 5 streamed tiles an item.  160 heads
# are more items than SMs, so a CTA walks several.
@pytest.mark.parametrize("lens,hq,hkv,window,dtype", [
    ([63, 64, 65, 129, 191, 257, 40, 320], 32, 32, -1, torch.bfloat16),
    ([65, 128, 130, 193, 33, 127], 48, 16, -1, torch.float16),
    ([200, 64, 310, 129], 64, 64, 70, torch.bfloat16),
    ([96], 160, 160, -1, torch.bfloat16),
])
def test_items_begin_with_either_group(lens, hq, hkv, window, dtype):
    *x, cu = tv.make(lens, hq, hkv, 64, 77)
    q, r, k, v, go = (t.to(dtype) for t in x)
    got = tv.run_gpu(q, r, k, v, go, cu, window)
    ref_o = orc.varlen_forward(q, r, k, v, cu, None, window)["o"]
    ref_g = orc.varlen_backward(q, r, k, v, go.float(), cu, None, window)
    for name, g, e in zip(("o", "dq", "dr", "dk", "dv"), got, (ref_o, *ref_g)):
        assert_close(g, e, TRAIN_REL_L2, TRAIN_MAX_REL, f"{lens} {hq}:{hkv} W={window} {dtype} {name}")


@pytest.mark.parametrize("hq,hkv,window", [(4, 4, -1), (8, 2, 200)])
def test_dq_dr_on_either_side_of_1024_tokens(hq, hkv, window):
    """Under a causal mask the first 1024 rows of a longer problem are the shorter problem, bit for bit."""
    gen = torch.Generator(device="cuda").manual_seed(5)
    q, r, go = (torch.randn(2, hq, 1100, 128, generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(3))
    k, v = (torch.randn(2, hkv, 1100, 128, generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2))

    def grads(n):
        leaves = [x[:, :, :n].contiguous().requires_grad_(True) for x in (q, r, k, v)]
        return torch.autograd.grad(plx.parallax_func(*leaves, window_size_left=window), leaves[:2], go[:, :, :n].contiguous())

    short = grads(1024)
    for n in (1025, 1100):
        for x, y in zip(short, grads(n)):
            assert torch.equal(x, y[:, :, :1024])


@pytest.mark.parametrize("hq,hkv,window,dtype", [(4, 4, -1, torch.bfloat16), (8, 2, 900, torch.bfloat16), (4, 2, -1, torch.float16)])
def test_dq_dr_by_the_keys_of_the_mean_item(hq, hkv, window, dtype):
    """The form of dq/dr goes by the keys that the mean item of 128 rows sees, up to 896 of them: 1600 tokens are on one side as a
    dense problem and on the other as one packed sequence, 256 of 1024 rows are on the other side than all of them."""
    gen = torch.Generator(device="cuda").manual_seed(7)
    q, r, go = (torch.randn(1, hq, 1600, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(3))
    k, v = (torch.randn(1, hkv, 1600, 128, generator=gen, device="cuda", dtype=dtype) for _ in range(2))

    def dense(lq, lk):
        x = [t[:, :, lk - lq:lk] for t in (q, r, go)] + [t[:, :, :lk] for t in (k, v)]
        x = [t.contiguous().requires_grad_(True) for t in x]
        o = plx.parallax_func(x[0], x[1], x[3], x[4], window_size_left=window)
        return torch.autograd.grad(o, (x[0], x[1], x[3], x[4]), x[2].detach())

    leaves = [t.transpose(1, 2).contiguous().requires_grad_(True) for t in (q, r, k, v)]
    cu = torch.tensor([0, 1600], dtype=torch.int32, device="cuda")
    o = plx.parallax_varlen_func(*leaves, window_size_left=window, cu_seqlens=cu)
    for x, y in zip(dense(1600, 1600), torch.autograd.grad(o, leaves, go.transpose(1, 2).contiguous())):
        assert torch.equal(x, y.transpose(1, 2))
    for x, y in zip(dense(256, 1024)[:2], dense(1024, 1024)[:2]):
        assert torch.equal(x, y[:, :, 768:])


@pytest.mark.parametrize("lq,lk,window", [(1300, 1300, 100), (300, 1500, 64), (150, 2000, -1), (1100, 1300, 500)])
def test_dq_dr_of_few_and_many_keys(lq, lk, window):
    gen = torch.Generator().manual_seed(8)
    q, r, go = (torch.randn(1, 2, lq, 128, generator=gen).bfloat16() for _ in range(3))
    k, v = (torch.randn(1, 1, lk, 128, generator=gen).bfloat16() for _ in range(2))
    leaves = [t.cuda().requires_grad_(True) for t in (q, r, k, v)]
    o = plx.parallax_func(*leaves, window_size_left=window)
    got = (o.detach(), *torch.autograd.grad(o, leaves, go.cuda()))
    ref = (orc.train_forward(q, r, k, v, None, window)["o"], *orc.train_backward(q, r, k, v, go.float(), None, window))
    for name, g, e in zip(("o", "dq", "dr", "dk", "dv"), got, ref):
        assert_close(g, e, TRAIN_REL_L2, TRAIN_MAX_REL, f"{lq} {lk} W={window} {name}")


@pytest.mark.parametrize("lens,lk,window,short", [
    ([1024], 1024, -1, True), ([1664], 1664, -1, True), ([1665], 1665, -1, False), ([3000], 3000, 768, True), ([3000], 3000, 769, False), ([128], 4096, -1, False), ([512], 2048, -1, False),
    ([128], 512, -1, True), ([3000], 3000, 100, True), ([3000], 3000, 1100, False), ([100] * 20, 0, -1, True), ([3000, 2000], 0, -1, False),
    ([3000, 2000], 0, 64, True)])
def test_which_dq_dr_runs(lens, lk, window, short):
    """Long items are many tiles per item, not many tokens per sequence: the kernel that ran, by its name in a profile."""
    from torch.profiler import ProfilerActivity, profile

    shape = (1, sum(lens), 2, 128) if lk == 0 else (1, 2, lens[0], 128)
    leaves = [torch.randn(shape if i < 2 or lk == 0 else (1, 2, lk, 128), device="cuda").bfloat16().requires_grad_(True) for i in range(4)]
    if lk == 0:
        cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
        o = plx.parallax_varlen_func(*leaves, window_size_left=window, cu_seqlens=cu)
    else:
        o = plx.parallax_func(*leaves, window_size_left=window)
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as prof:
        torch.autograd.grad(o, leaves, o.detach())
        torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "bwd_sm100_kernel" in e.name]
    if not names:
        pytest.skip("the profiler does not see kernels here")
    ran = [n for n in names if "128, 0, " in n]
    assert len(ran) == 1 and ("true" in ran[0].split(">")[0]) == short, names
