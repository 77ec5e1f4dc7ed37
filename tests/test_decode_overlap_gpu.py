"""Decode launches that overlap the end of the kernel before them."""
import pytest
import torch

import parallax_b200 as plx
from tests._util import seeded_bf16

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
