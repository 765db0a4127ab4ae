"""Head dims 16 and 32 on the tcgen05 kernels (their D = 64 instances with boxes that reach past the row's end): every
operator family and the backward pass against the CPU oracle, at the edges of the 128-row tiles and with the heads
of a row next to each other in memory, where a box that was not clipped would touch the next head."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _rows(b, h, s, d, dtype, g, interleaved):
    t = torch.randn(b, s, h, d, generator=g) if interleaved else torch.randn(b, h, s, d, generator=g)
    return (t.transpose(1, 2) if interleaved else t).to(dtype)


@pytest.mark.parametrize("M,N", [(1, 300), (127, 127), (129, 257), (300, 140)])
@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("interleaved", [False, True], ids=["bhsd", "bshd"])
def test_small_head_dims_match_the_oracle(M, N, D, dtype, interleaved):
    B, Hq, Hk, causal = 2, 4, 2, M != 1
    g = torch.Generator().manual_seed(M + N + D)
    q, k, v = (_rows(B, h, s, D, dtype, g, interleaved) for h, s in ((Hq, M), (Hk, N), (Hk, N)))
    ref_out, ref_scores = orc.naive_attention_with_scores(q, k, v, causal, p_seq=N - M)
    slack = orc.bf16_out_slack(ref_scores, v, ref_out) if dtype == torch.bfloat16 else None
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    assert qd.stride(2) == q.stride(2)
    split = max(1, N // 3)

    def check(got, want, what):
        ok, err = orc.check_out(got[0].cpu(), ref_out, slack)
        assert ok, (what, err)
        assert F.last_backend() == "tcgen05", what
        if want is not None:
            ok, viol = orc.check_sum(got[1].cpu(), want)
            assert ok, (what, viol)

    check((F.attention(qd, kd, vd, causal),), None, "attention")
    check(F.attention_with_row_sum(qd, kd, vd, causal), orc.row_sum(ref_scores), "row_sum")
    check(F.attention_with_col_sum(qd, kd, vd, causal), orc.group_sum(orc.col_sum(ref_scores), Hk), "col_sum")
    check(F.attention_with_softmax_col_sum(qd, kd, vd, causal),
          orc.group_sum(orc.softmax_col_sum(ref_scores), Hk), "softmax_col_sum")
    check(F.attention_cross_token_softmax_sum(qd, kd, vd, split, causal),
          orc.group_sum(orc.cross_token_softmax_sum(ref_scores, split), Hk), "cross_softmax")
    o, s = F.attention_with_scores(qd, kd, vd, causal)
    check((o,), None, "scores")
    ok, viol, ok_mask = orc.check_scores(s.cpu(), ref_scores)
    assert ok and ok_mask, viol
    assert F.device_status() == 0


@pytest.mark.parametrize("M,N", [(128, 128), (129, 257)])
@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("interleaved", [False, True], ids=["bhsd", "bshd"])
def test_small_head_dims_backward(M, N, D, interleaved):
    B, Hq, Hk = 1, 4, 2
    g = torch.Generator().manual_seed(D + M)
    q, k, v, do = (_rows(B, h, s, D, torch.float16, g, interleaved) for h, s in ((Hq, M), (Hk, N), (Hk, N), (Hq, M)))
    ref = orc.attention_backward(q, k, v, do, True, p_seq=N - M)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
        got = torch.autograd.grad(F.attention(qd, kd, vd, True), (qd, kd, vd), do.cuda())
    assert F.last_backend() == "tcgen05"
    for name, x, r, sl in zip(("dq", "dk", "dv"), got, ref, orc.grad_slack(q, k, v, do, True, p_seq=N - M)):
        ok, viol, err = orc.check_grad(x.cpu(), r, False, sl)
        assert ok, (name, viol, err)
    assert F.device_status() == 0
