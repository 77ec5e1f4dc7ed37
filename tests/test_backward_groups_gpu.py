"""The two plans of the backward that depend on the problem.  head_dim 64, whose element-wise groups take the streamed tiles in
turn: work items of every small tile count in a row on one CTA, so that items begin with either group and a group has no
tile of some of them.  head_dim 128, whose dq/dr keeps dO in shared memory up to 1024 tokens and in tensor memory above."""
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
