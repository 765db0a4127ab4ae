"""Launches of fewer than two 256-row CTAs per SM: both row counts of a CTA, on either side of the choice between them."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hk,M,N,D,causal", [
    (40, 40, 512, 512, 64, False), (32, 32, 512, 512, 64, False), (144, 36, 300, 300, 64, True),
    (32, 8, 513, 1025, 128, True), (48, 12, 700, 700, 128, True), (20, 20, 1030, 1030, 64, True),
    (150, 50, 257, 129, 32, False)])
def test_attention_and_sums_near_the_line(H, Hk, M, N, D, causal):
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q, k, v = [torch.randn(1, h, s, D, device="cuda", generator=g).half() for h, s in ((H, M), (Hk, N), (Hk, N))]
    kf, vf = k.float().repeat_interleave(H // Hk, 1), v.float().repeat_interleave(H // Hk, 1)
    s = (q.float() @ kf.mT) * D ** -0.5
    seen = torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M) if causal else torch.ones(M, N, dtype=torch.bool, device="cuda")
    want = s.masked_fill(~seen, float("-inf")).softmax(-1) @ vf
    raw = s.masked_fill(~seen, 0.0)
    for out in (F.attention(q, k, v, causal, kv_splits=1), F.attention_with_row_sum(q, k, v, causal)[0],
                F.attention_with_col_sum(q, k, v, causal)[0]):
        assert F.last_backend() == "tcgen05"
        ok, err = orc.check_out(out.cpu(), want.cpu())
        assert ok, err
    ok, viol = orc.check_sum(F.attention_with_row_sum(q, k, v, causal)[1].cpu(), raw.sum(-1).cpu())
    assert ok, viol
    ok, viol = orc.check_sum(F.attention_with_col_sum(q, k, v, causal, per_q_head=True)[1].cpu(), raw.sum(-2).cpu())
    assert ok, viol
