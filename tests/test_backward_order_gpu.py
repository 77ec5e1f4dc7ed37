"""The three kernels of the backward overlap (row statistics, dk/dv, dq/dr): whatever way the call is made, its results are
those of the three launched one by one."""
import pytest
import torch

import parallax_b200 as plx
from parallax_b200 import ops

pytestmark = pytest.mark.gpu

# batch, hq, hkv, tokens, head_dim, window: one item per CTA, fewer and more items than SMs, grouped heads
CASES = [(1, 2, 2, 200, 128, -1), (2, 8, 8, 1024, 128, -1), (2, 8, 2, 1100, 64, -1), (4, 16, 16, 1000, 128, 300), (1, 4, 1, 3000, 64, -1)]


def randn(shape, seed):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)).bfloat16()


class Step:
    """One backward of the case with inputs of its own, on a workspace that the steps share."""

    def __init__(self, case, seed):
        bsz, hq, hkv, n, d, window = case
        q, r, go = (randn((bsz, hq, n, d), 10 * seed + i) for i in range(3))
        k, v = (randn((bsz, hkv, n, d), 10 * seed + 3 + i) for i in range(2))
        self.scalars = (d ** -0.5, window, ops.BHLD, None)
        o, barv, d1, bart, m = ops.train_fwd(q, r, k, v, *self.scalars)
        self.inputs = (q, r, k, v, o, barv, d1, bart, m, go)

    def workspace(self):
        return ops.train_bwd_workspace(self.inputs[0], self.inputs[2], self.inputs[6], ops.BHLD, None)

    def outputs(self):
        return [torch.full_like(x, float("nan")) for x in self.inputs[:4]]

    def launch(self, stages, out, ws):
        ops.train_bwd_stages(stages, *self.inputs, *out, ws, *self.scalars)

    def one_by_one(self, ws):
        out = self.outputs()
        for stage in (ops.BWD_STATS, ops.BWD_DQR, ops.BWD_DKV):
            self.launch(stage, out, ws)
            torch.cuda.synchronize()
        return out


def same(a, b):
    return all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("case", CASES)
def test_calls_in_a_row_on_one_workspace(case):
    """The statistics of a call lie where those of the call before lay, and the inputs are others each time."""
    steps = [Step(case, s) for s in range(4)]
    ws = steps[0].workspace()
    want = [s.one_by_one(ws) for s in steps]
    for _ in range(5):
        got = [s.outputs() for s in steps]
        for s, out in zip(steps, got):
            s.launch(ops.BWD_ALL, out, ws)
        torch.cuda.synchronize()
        assert all(same(g, w) for g, w in zip(got, want))
    # the two gradient kernels alone, behind statistics of their own call
    for s, w in zip(steps, want):
        out = s.outputs()
        s.launch(ops.BWD_STATS, out, ws)
        s.launch(ops.BWD_DKV | ops.BWD_DQR, out, ws)
        torch.cuda.synchronize()
        assert same(out, w)


@pytest.mark.parametrize("case", CASES[:3])
def test_a_captured_backward_is_replayed_on_new_inputs(case):
    steps = [Step(case, s) for s in range(3)]
    ws = steps[0].workspace()
    want = [s.one_by_one(ws) for s in steps]
    static, out = Step(case, 0), steps[0].outputs()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        static.launch(ops.BWD_ALL, out, ws)
        static.launch(ops.BWD_ALL, out, ws)
    for i in (0, 1, 2, 1, 0, 2):
        for dst, src in zip(static.inputs, steps[i].inputs):
            dst.copy_(src)
        for x in out:
            x.fill_(float("nan"))
        graph.replay()
        assert same(out, want[i])


@pytest.mark.parametrize("case", CASES[:3])
def test_another_stream_sees_all_gradients_after_an_event(case):
    steps = [Step(case, s) for s in range(6)]
    ws = steps[0].workspace()
    want = [s.one_by_one(ws) for s in steps]
    got = [s.outputs() for s in steps]
    seen = [[torch.empty_like(x) for x in out] for out in got]
    reader, event = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    for s, out, copy in zip(steps, got, seen):
        s.launch(ops.BWD_ALL, out, ws)
        event.record()
        with torch.cuda.stream(reader):
            event.wait()
            for dst, src in zip(copy, out):
                dst.copy_(src)
    torch.cuda.synchronize()
    assert all(same(c, w) for c, w in zip(seen, want))


def test_a_captured_training_step():
    """Forward, loss and backward through autograd inside one graph, replayed on new inputs."""
    shape = (2, 4, 300, 64)
    leaves = [randn(shape, s).requires_grad_(True) for s in range(4)]
    others = [randn(shape, 50 + s) for s in range(4)]

    def step():
        o = plx.parallax_func(*leaves)
        return (o.detach(), *torch.autograd.grad(o.float().pow(2).mean(), leaves))

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    for source in (others, [-x for x in others], others):
        with torch.no_grad():
            for x, y in zip(leaves, source):
                x.copy_(y)
        graph.replay()
        got = [x.clone() for x in out]
        assert same(got, step())
