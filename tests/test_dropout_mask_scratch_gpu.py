"""Backward pass with dropout: the mask drawn once into scratch, and by both kernels where scratch has no room for it."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("B,Hq,Hk,M,N,D,causal", [
    (1, 1, 1, 1, 1, 64, False), (2, 4, 2, 200, 333, 64, True), (1, 2, 2, 257, 129, 128, False),
    (1, 3, 3, 128, 128, 32, True), (1, 2, 1, 300, 130, 16, True), (2, 2, 1, 31, 640, 128, True)])
def test_mask_in_scratch_is_the_mask_drawn_in_the_kernels(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    q, k, v, do = [torch.randn(B, h, s, D, device="cuda", generator=g).to(dtype)
                   for h, s in ((Hq, M), (Hk, N), (Hk, N), (Hq, M))]
    for t in (q, k, v):
        t.requires_grad_(True)

    def grads():
        out = F.attention(q, k, v, causal, dropout_p=0.3, philox=(11, 8))
        with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
            got = torch.autograd.grad(out, (q, k, v), do)
        assert F.last_backend() == "tcgen05"
        return got
    kept = grads()
    sizes = []
    mask_bytes = B * Hq * ((M + 127) // 128) * ((N + 127) // 128) * 2048
    whole = api._Call.workspace

    def workspace(self, op, split=0):
        ws, n = whole(self, op, split)
        sizes.append(n)
        return ws[:n - mask_bytes], n - mask_bytes
    monkeypatch.setattr(api._Call, "workspace", workspace)
    drawn = grads()
    assert len(sizes) == 1 and sizes[0] > mask_bytes
    for x, y in zip(kept, drawn):  # the same arithmetic on the same mask
        assert torch.equal(x, y)
