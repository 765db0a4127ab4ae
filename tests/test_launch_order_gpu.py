"""Launches whose order or overlap is chosen by their size: key-major softmax sums of heads whose last CTA has few keys, the
column sums' reduce that begins before the forward pass has ended, and score launches that fetch their first tiles into L2."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [257, 384, 385, 513, 640, 641])  # last CTA of 1 to 256 keys: the first ones come last up to 128
@pytest.mark.parametrize("B,H,Hk,M,D", [(2, 6, 2, 300, 64), (1, 8, 8, 129, 128), (3, 4, 4, 1, 32)])
def test_softmax_sums_of_a_few_last_keys(N, B, H, Hk, M, D):
    g = torch.Generator(device="cuda").manual_seed(N + M)
    q, k, v = [torch.randn(B, h, s, D, device="cuda", generator=g).half() for h, s in ((H, M), (Hk, N), (Hk, N))]
    w = ((q.double() @ k.double().repeat_interleave(H // Hk, 1).mT) * D ** -0.5).softmax(-1)
    _, got = F.attention_with_softmax_col_sum(q, k, v, False, per_q_head=True)
    assert F.last_backend() == "tcgen05"
    ok, viol = orc.check_sum(got.cpu(), w.sum(-2).float().cpu())
    assert ok, viol
    S = N + 40  # the same over the keys before a split, from the queries behind it
    q, k, v = [torch.randn(B, h, S, D, device="cuda", generator=g).half() for h in (H, Hk, Hk)]
    w = ((q.double() @ k.double().repeat_interleave(H // Hk, 1).mT) * D ** -0.5).softmax(-1)
    _, got = F.attention_cross_token_softmax_sum(q, k, v, N, False, per_q_head=True)
    ok, viol = orc.check_sum(got.cpu(), w[:, :, N:, :N].sum(-2).float().cpu())
    assert ok, viol
    assert F.device_status() == 0


@pytest.mark.parametrize("B,H,Hk,S,D", [(1, 8, 8, 512, 64), (1, 16, 4, 300, 128), (1, 37, 37, 512, 64), (1, 38, 19, 512, 64)])
def test_keys_written_just_before_the_column_sums(B, H, Hk, S, D):
    """148 CTAs of 128 rows or fewer, whose reduce reads the keys early, and more: keys that the kernel before the call wrote,
    and writes again right behind it."""
    g = torch.Generator(device="cuda").manual_seed(S)
    q, v = [torch.randn(B, h, S, D, device="cuda", generator=g).half() for h in (H, Hk)]
    keys = [torch.randn(B, Hk, S, D, device="cuda", generator=g).half() for _ in range(4)]
    want = []
    for x in keys:
        want.append(F.attention_with_col_sum(q, x, v, True)[1])
        torch.cuda.synchronize()
    k = torch.zeros_like(keys[0])
    for _ in range(5):
        got = []
        for x in keys:
            k.copy_(x)
            got.append(F.attention_with_col_sum(q, k, v, True)[1])
            k.fill_(float("nan"))
        for x, y in zip(got, want):
            assert torch.equal(x, y)
    assert F.device_status() == 0


@pytest.mark.parametrize("H,M,N,D,causal", [(64, 300, 640, 64, True), (64, 300, 641, 64, True), (37, 300, 644, 128, False),
                                            (36, 300, 644, 128, False), (40, 512, 1024, 128, True), (300, 100, 700, 32, True),
                                            (111, 200, 385, 64, True), (148, 200, 384, 64, False), (110, 200, 640, 64, True), (148, 100, 256, 128, False),
                                            (147, 90, 130, 128, True)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16], ids=["fp32", "fp16"])
def test_inputs_written_just_before_the_scores(H, M, N, D, causal, dtype):
    """Key tiles and CTAs on either side of the lines: inputs that the kernels before the call wrote, and write again right
    behind it."""
    g = torch.Generator(device="cuda").manual_seed(N + H)
    sets = [[torch.randn(1, H, s, D, device="cuda", generator=g).half() for s in (M, N, N)] for _ in range(3)]
    want = []
    for x in sets:
        want.append(F.attention_with_scores(*x, causal, scores_dtype=dtype))
        torch.cuda.synchronize()
        ref = (x[0].float() @ x[1].float().mT) * D ** -0.5
        if causal:
            ref = ref.masked_fill(~torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M), float("-inf"))
        ok, err = orc.check_out(want[-1][0].cpu(), (ref.softmax(-1) @ x[2].float()).cpu())
        assert ok, err
    now = [torch.zeros_like(t) for t in sets[0]]
    for _ in range(3):
        for x, y in zip(sets, want):
            for t, u in zip(now, x):
                t.copy_(u)
            got = F.attention_with_scores(*now, causal, scores_dtype=dtype)
            for t in now:
                t.fill_(float("nan"))
            assert torch.equal(got[0], y[0]) and torch.equal(got[1], y[1])
    assert F.last_backend() == "tcgen05" and F.device_status() == 0


@pytest.mark.parametrize("B,H,Hk,S,D,causal", [(8, 28, 28, 270, 32, True), (5, 28, 28, 385, 16, False), (2, 28, 4, 270, 32, True),
                                               (4, 28, 28, 512, 32, False), (1, 8, 8, 1029, 64, True)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_column_sums_of_two_and_three_reduce_ctas(B, H, Hk, S, D, causal, dtype):
    """More key tiles of output heads than two per SM (296 of them) and fewer; sums of 1 to 9 terms a thread group."""
    g = torch.Generator(device="cuda").manual_seed(S + H)
    q, k, v = [torch.randn(B, h, S, D, device="cuda", generator=g).to(dtype) for h in (H, Hk, Hk)]
    s = (q.double() @ k.double().repeat_interleave(H // Hk, 1).mT) * D ** -0.5
    if causal:
        s = s.tril()
    for per_head in (False, True):
        _, got = F.attention_with_col_sum(q, k, v, causal, per_q_head=per_head)
        assert F.last_backend() == "tcgen05"
        want = s.sum(-2) if per_head else s.sum(-2).view(B, Hk, H // Hk, S).sum(2)
        ok, viol = orc.check_sum(got.cpu(), want.float().cpu())
        assert ok, viol
    assert F.device_status() == 0
