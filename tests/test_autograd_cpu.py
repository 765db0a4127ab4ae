"""attention() under autograd, the part that needs no kernels: a gradient that never arrives."""
import types

import torch

from flash_attn_with_score_b200 import api


class _NoGradient(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x.sum()

    @staticmethod
    def backward(ctx, g):
        return None


def test_an_undefined_output_gradient_gives_zero_gradients(monkeypatch):
    def forward(q, k, v, *args, **kwargs):
        return types.SimpleNamespace(q=q, k=k, v=v, out=q + v, L=q.sum(-1), p=types.SimpleNamespace(sm_scale=1.0),
                                     seed=None, offset=None), None
    monkeypatch.setattr(api, "_attention_forward", forward)
    q, k, v = (torch.randn(1, 2, 4, 16, requires_grad=True) for _ in range(3))
    grads = torch.autograd.grad(_NoGradient.apply(api.attention(q, k, v)), (q, k, v))
    for g, t in zip(grads, (q, k, v)):
        assert g.shape == t.shape and torch.count_nonzero(g) == 0
