"""Persistent launches of causal problems with more query rows than keys: work items without a visible key, several of
them in a row on one CTA."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("H,Hk,M,N,D", [
    (20, 20, 2048, 700, 128), (40, 8, 2048, 700, 64),  # 160 and 320 items of 256 rows
    (48, 48, 2300, 1, 64), (75, 25, 1000, 130, 32), (300, 300, 600, 200, 64)])
def test_rows_without_a_key(H, Hk, M, N, D, dtype):
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q, k, v = [torch.randn(1, h, s, D, device="cuda", generator=g).to(dtype) for h, s in ((H, M), (Hk, N), (Hk, N))]
    kf, vf = k.float().repeat_interleave(H // Hk, 1), v.float().repeat_interleave(H // Hk, 1)
    seen = torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M)
    s = (q.float() @ kf.mT) * D ** -0.5
    want = torch.nan_to_num(s.masked_fill(~seen, float("-inf")).softmax(-1)) @ vf  # zero rows where nothing is seen
    raw = s.masked_fill(~seen, 0.0)
    slack = None
    if dtype == torch.bfloat16:
        slack = orc.bf16_out_slack(s.masked_fill(~seen, float("-inf")).cpu(), v.cpu(), want.cpu())
    for twice in range(2):
        outs = [F.attention(q, k, v, True, kv_splits=1), *F.attention_with_row_sum(q, k, v, True),
                *F.attention_with_col_sum(q, k, v, True, per_q_head=True)]
        assert F.last_backend() == "tcgen05" and F.device_status() == 0
        for out in (outs[0], outs[1], outs[3]):
            ok, err = orc.check_out(out.cpu(), want.cpu(), slack)
            assert ok, err
        for got, dim in ((outs[2], -1), (outs[4], -2)):
            ok, viol = orc.check_sum(got.cpu(), raw.sum(dim).cpu())
            assert ok, viol
    dropped = F.attention(q, k, v, True, dropout_p=0.25, philox=(1, 0))
    assert F.device_status() == 0
    assert not bool(dropped[:, :, :M - N].any()) and bool(dropped[:, :, M - N:].any(-1).float().mean() > 0.5)
    assert bool(dropped.isfinite().all())


@pytest.mark.parametrize("H,Hk,M,N,D,causal", [
    (200, 50, 300, 100, 64, False), (160, 160, 300, 100, 128, False),  # the second block of a head has one query tile
    (150, 150, 390, 260, 128, True), (100, 25, 650, 500, 64, True)])   # the first query tile that sees a key is a block's second
def test_items_of_one_query_tile(H, Hk, M, N, D, causal):
    """Items in which one of the two softmax warpgroups has nothing to do, between items in which it has."""
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q, k, v = [torch.randn(1, h, s, D, device="cuda", generator=g).half() for h, s in ((H, M), (Hk, N), (Hk, N))]
    kf, vf = k.float().repeat_interleave(H // Hk, 1), v.float().repeat_interleave(H // Hk, 1)
    seen = torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M if causal else N)
    s = (q.float() @ kf.mT) * D ** -0.5
    want = torch.nan_to_num(s.masked_fill(~seen, float("-inf")).softmax(-1)) @ vf
    raw = s.masked_fill(~seen, 0.0)
    for twice in range(4):
        outs = [F.attention(q, k, v, causal, kv_splits=1), *F.attention_with_row_sum(q, k, v, causal),
                *F.attention_with_col_sum(q, k, v, causal, per_q_head=True)]
        assert F.last_backend() == "tcgen05" and F.device_status() == 0
        for out in (outs[0], outs[1], outs[3]):
            ok, err = orc.check_out(out.cpu(), want.cpu())
            assert ok, err
        for got, dim in ((outs[2], -1), (outs[4], -2)):
            ok, viol = orc.check_sum(got.cpu(), raw.sum(dim).cpu())
            assert ok, viol
