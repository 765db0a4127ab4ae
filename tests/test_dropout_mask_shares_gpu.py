"""Backward pass with dropout where the mask of all heads is more than the scratch holds: the heads take turns."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hk,M,N,D,causal,dtype,shares", [
    (3, 3, 1, 16384, 16384, 32, True, torch.float16, 2),     # 32 MB a head: five heads, then four; a batch in both
    (1, 17, 17, 11520, 11500, 64, False, torch.bfloat16, 2),  # 15.8 MB a head, ragged keys; nine and eight
    (1, 2, 2, 8000, 2000, 128, True, torch.float16, 1)])
def test_shares_are_the_mask_drawn_in_the_kernels(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype, shares):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    q, k, v, do = [torch.randn(B, h, s, D, device="cuda", generator=g).to(dtype)
                   for h, s in ((Hq, M), (Hk, N), (Hk, N), (Hq, M))]
    for t in (q, k, v):
        t.requires_grad_(True)
    out = F.attention(q, k, v, causal, dropout_p=0.2, philox=(5, 4))
    tiles = ((M + 127) // 128) * ((N + 127) // 128)
    mask_bytes = -(-B * Hq // shares) * tiles * 2048
    whole, sizes = api._Call.workspace, []

    def grads(leave_out):
        def workspace(self, op, split=0):
            ws, n = whole(self, op, split)
            sizes.append(n)
            return ws[:n - leave_out], n - leave_out
        monkeypatch.setattr(api._Call, "workspace", workspace)
        before = F.launch_count()
        with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
            got = torch.autograd.grad(out, (q, k, v), do, retain_graph=True)
        assert F.last_backend() == "tcgen05"
        return got, F.launch_count() - before
    group_sum = 1 if Hq > Hk else 0
    in_turns, launches = grads(0)
    assert launches == 3 * shares + group_sum and sizes[0] > mask_bytes
    drawn, launches = grads(mask_bytes)
    assert launches == 3 + group_sum
    for x, y in zip(in_turns, drawn):  # the same arithmetic on the same mask
        assert torch.equal(x, y)
