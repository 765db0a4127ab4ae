"""Scratch that was sized once for a shape serves the calls of that shape whose kernels would like more of it."""
import ctypes as C

import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import _lib, api

pytestmark = pytest.mark.gpu


def _sized_by(monkeypatch, op, change):
    """Every call's scratch is what faws_workspace_bytes says for `op` and the call's problem after `change`."""
    def workspace(self, _, split=0):
        p = _lib.Problem.from_buffer_copy(self.p)
        change(p)
        n = self.lib.faws_workspace_bytes(op, C.byref(p), split)
        return torch.empty(n, device=self.dev, dtype=torch.uint8), n
    monkeypatch.setattr(api._Call, "workspace", workspace)


def _inputs(M, N, D):
    g = torch.Generator(device="cuda").manual_seed(D)
    return [torch.randn(2, h, s, D, device="cuda", generator=g).half() for h, s in ((4, M), (2, N), (2, N), (4, M))]


def test_backward_with_the_scratch_of_a_call_without_dropout(monkeypatch):
    q, k, v, do = _inputs(200, 200, 64)
    for t in (q, k, v):
        t.requires_grad_(True)

    def grads(backend):
        out = F.attention(q, k, v, True, dropout_p=0.2, philox=(3, 0), backend=backend)
        with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
            return torch.autograd.grad(out, (q, k, v), do)
    grads(None)
    assert F.last_backend() == "tcgen05"
    _sized_by(monkeypatch, _lib.OP_ATTENTION_BACKWARD, lambda p: setattr(p, "dropout_p", 0.0))
    got = grads(None)
    assert F.last_backend() == "generic"
    for x, y in zip(got, grads("generic")):
        assert (x.double() - y.double()).norm() <= 2e-3 * y.double().norm()
    with pytest.raises(RuntimeError, match="workspace"):
        grads("tcgen05")


@pytest.mark.parametrize("split", [64, 129])
def test_buffered_sums_with_the_scratch_of_aligned_tensors(monkeypatch, split):
    q, k, v, _ = _inputs(200, 200, 64)
    shifted = torch.empty(2, 4, 200, 72, device="cuda", dtype=q.dtype)[..., 1:65].copy_(q)  # rows TMA cannot address
    want = F.attention_cross_token_softmax_sum_buffered(shifted, k, v, split, True)
    assert F.last_backend() == "generic"
    _sized_by(monkeypatch, _lib.OP_CROSS_SOFTMAX_SUM, lambda p: None)
    got = F.attention_cross_token_softmax_sum_buffered(shifted, k, v, split, True)
    for x, y, tol in zip(got, want, (1e-3, 1e-5)):  # out in fp16, the sums in fp32, keys in another order
        assert (x.double() - y.double()).norm() <= tol * y.double().norm()
    with pytest.raises(RuntimeError, match="workspace"):  # the buffer is what forcing the CUDA-core kernels asks for
        F.attention_cross_token_softmax_sum_buffered(shifted, k, v, split, True, backend="generic")
