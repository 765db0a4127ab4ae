"""Backward pass with dropout: the mask drawn once into scratch, and by both kernels where scratch has no room for it."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import api
from oracle import oracle as orc

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

    out = F.attention(q, k, v, causal, dropout_p=0.3, philox=(11, 8))
    nqt, nkt = (M + 127) // 128, (N + 127) // 128
    mask_bytes = B * Hq * nqt * nkt * 2048
    whole, held = api._Call.workspace, []

    def grads(left_out):
        def workspace(self, op, split=0):
            ws, n = whole(self, op, split)
            assert n > mask_bytes
            ws[n - mask_bytes:].fill_(0x5a)
            held.append(ws)
            return ws, n - left_out
        monkeypatch.setattr(api._Call, "workspace", workspace)
        with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
            got = torch.autograd.grad(out, (q, k, v), do, retain_graph=True)
        assert F.last_backend() == "tcgen05"
        return got
    kept, drawn = grads(0), grads(mask_bytes)
    for x, y in zip(kept, drawn):  # the same arithmetic on the same mask
        assert torch.equal(x, y)
    # the first call left the mask of every tile with a visible entry in its scratch, the second wrote nothing there
    words = [ws[ws.numel() - mask_bytes:].cpu().view(torch.int32).view(B, Hq, nqt, nkt, 128, 4) for ws in held]
    assert bool((words[1] == 0x5a5a5a5a).all())
    bits = (words[0][..., None] >> torch.arange(32, dtype=torch.int32)) & 1
    bits = bits.permute(0, 1, 2, 4, 3, 5, 6).reshape(B, Hq, nqt * 128, nkt * 128)[:, :, :M, :N].bool()
    want = orc.dropout_keep_mask(11, 8, B, Hq, M, N, 0.3)
    qt, kt = torch.arange(nqt)[:, None], torch.arange(nkt)
    seen = (kt * 128 <= qt * 128 + 127 + N - M) if causal else torch.ones(nqt, nkt, dtype=torch.bool)
    assert bool((words[0][:, :, ~seen] == 0x5a5a5a5a).all())
    seen = seen.repeat_interleave(128, 0).repeat_interleave(128, 1)[:M, :N]
    assert torch.equal(bits[:, :, seen], want[:, :, seen])
