"""The backward writes a gradient by the strides of the input it belongs to, so every gradient has to be allocated with
those strides.  Checked on what reaches the library (a fake of its entry point records it), without a GPU."""
import contextlib

import pytest
import torch

from parallax_b200 import _cabi, ops


class FakeLibrary:
    """plx_train_workspace_bytes and plx_train_bwd_stages as far as the host side sees them."""

    def plx_train_workspace_bytes(self, p, need):
        need._obj.value = 64
        return 0

    def plx_train_bwd_stages(self, p, stages, *pointers):
        self.problem, self.pointers = p._obj, [x.value for x in pointers[:14]]
        return 0


@pytest.fixture
def library(monkeypatch):
    fake = FakeLibrary()
    monkeypatch.setattr(_cabi, "lib", lambda: fake)
    monkeypatch.setattr(_cabi, "raise_if_device_error", lambda what: None)
    monkeypatch.setattr(ops, "_stream", lambda device: None)
    monkeypatch.setattr(torch.cuda, "device", lambda device: contextlib.nullcontext())
    return fake


def last_element(ptr, shape, strides):
    return ptr + 2 * sum((n - 1) * s for n, s in zip(shape, strides))


# (batch, tokens, heads, head_dim) tensors: dense, a slice of a longer cache, some heads of a wider one
@pytest.mark.parametrize("q_cut,k_cut", [("none", "none"), ("none", "tokens"), ("none", "heads"), ("tokens", "none"), ("heads", "tokens")])
def test_gradients_have_the_strides_they_are_written_with(library, q_cut, k_cut):
    bsz, n, d = 3, 24, 64

    def mk(heads, cut):
        if cut == "tokens":
            return torch.zeros(bsz, n + 40, heads, d, dtype=torch.bfloat16)[:, :n]
        if cut == "heads":
            return torch.zeros(bsz, n, heads + 2, d, dtype=torch.bfloat16)[:, :, :heads]
        return torch.zeros(bsz, n, heads, d, dtype=torch.bfloat16)

    q, r, o, barv, go = (mk(4, q_cut) for _ in range(5))
    k, v = mk(2, k_cut), mk(2, k_cut)
    for t in (k, v, q, r):
        t.normal_()
    stats = [torch.zeros(bsz, n, 4) for _ in range(3)]
    dq, dr, dk, dv = ops.train_bwd._init_fn(q, r, k, v, o, barv, *stats, go, 0.125, -1, ops.BTHD, None)
    p = library.problem
    q_like, kv_like = (p.q_stride_b, p.q_stride_t, p.q_stride_h, 1), (p.kv_stride_b, p.kv_stride_t, p.kv_stride_h, 1)
    assert dq.stride() == dr.stride() == q_like and dk.stride() == dv.stride() == kv_like
    at = dict(zip(("q", "r", "k", "v", "o", "barv", "d1", "bart", "m", "go", "dq", "dr", "dk", "dv"), library.pointers))
    for name, grad in (("dq", dq), ("dr", dr), ("dk", dk), ("dv", dv)):
        strides = q_like if name in ("dq", "dr") else kv_like
        storage = grad.untyped_storage()
        assert at[name] == grad.data_ptr()
        assert last_element(at[name], grad.shape, strides) < storage.data_ptr() + storage.nbytes()


def test_the_forward_writes_its_outputs_with_their_own_strides(library):
    """The same of plx::train_fwd, whose outputs are written by the strides of q."""
    recorded = {}

    def plx_train_fwd(p, *pointers):
        recorded["p"] = p._obj
        return 0

    library.plx_train_fwd = plx_train_fwd
    q, r = (torch.zeros(3, 64, 4, 64, dtype=torch.bfloat16)[:, :24] for _ in range(2))
    k, v = (torch.zeros(3, 24, 4, 64, dtype=torch.bfloat16) for _ in range(2))
    o, barv, *_ = ops.train_fwd_op._init_fn(q, r, k, v, 0.125, -1, ops.BTHD, None)
    p = recorded["p"]
    assert o.stride() == barv.stride() == (p.q_stride_b, p.q_stride_t, p.q_stride_h, 1)
