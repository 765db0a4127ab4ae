"""Backward pass with dropout where a softmax weight is not finite: the gradient of v shows it for dropped entries too."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask_in_scratch", [True, False])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_nan_query_reaches_every_key_it_sees(monkeypatch, D, dtype, mask_in_scratch):
    H, M, N = 2, 130, 200
    g = torch.Generator(device="cuda").manual_seed(D)
    q, k, v, do = [torch.randn(1, H, s, D, device="cuda", generator=g).to(dtype) for s in (M, N, N, M)]
    q[0, 0, 57, 3] = float("nan")  # causal: this row sees keys 0 .. 57 + N - M
    for t in (q, k, v):
        t.requires_grad_(True)
    if not mask_in_scratch:
        whole = api._Call.workspace
        mask_bytes = H * 2 * 2 * 2048  # 2 x 2 tiles a head

        def workspace(self, op, split=0):
            ws, n = whole(self, op, split)
            return ws[:n - mask_bytes], n - mask_bytes
        monkeypatch.setattr(api._Call, "workspace", workspace)
    out = F.attention(q, k, v, True, dropout_p=0.5, philox=(3, 0))
    with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
        dv, = torch.autograd.grad(out, (v,), do)
    assert F.last_backend() == "tcgen05"
    seen = 57 + N - M + 1
    assert bool(dv[0, 0, :seen].isnan().all())  # half of these entries are dropped
    assert not bool(dv[0, 0, seen:].isnan().any()) and not bool(dv[0, 1].isnan().any())
