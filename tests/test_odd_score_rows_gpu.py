"""Score tensors whose rows do not start on 16-byte boundaries (odd lengths, shifted buffers), which TMA cannot address:
the plain-store forms of the score hook and of the score-only operator against the CPU oracle.  Nothing outside the
tensor may be written: each one lies inside a larger buffer whose margins are checked."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (5, 127), (127, 129), (129, 258), (300, 301), (257, 131), (140, 1030)]


def _inputs(M, N, D, dtype):
    g = torch.Generator().manual_seed(M * 7 + N)
    mk = lambda h, s: torch.randn(1, h, s, D, generator=g).to(dtype)  # noqa: E731
    return mk(4, M), mk(2, N), mk(2, N)


@pytest.mark.parametrize("M,N", SHAPES)
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
@pytest.mark.parametrize("kind", ["fp32", "fp16", "bf16"])
@pytest.mark.parametrize("shift", [0, 1])
def test_scores_in_odd_rows(M, N, causal, kind, shift):
    dtype = torch.bfloat16 if kind == "bf16" else torch.float16
    q, k, v = _inputs(M, N, 64 if M % 2 else 128, dtype)
    sd = torch.float32 if kind == "fp32" else dtype
    ref_out, ref = orc.naive_attention_with_scores(q, k, v, causal, p_seq=N - M)
    n = 4 * M * N
    buf = torch.full((n + 130,), 7.0, device="cuda", dtype=sd)
    lo = 64 + shift
    scores = buf[lo:lo + n].view(1, 4, M, N)
    out, s = F.attention_with_scores(q.cuda(), k.cuda(), v.cuda(), causal, scores_dtype=sd, scores=scores)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    assert bool((buf[:lo] == 7.0).all()) and bool((buf[lo + n:] == 7.0).all())
    slack = orc.bf16_out_slack(ref, v, ref_out) if kind == "bf16" else None
    ok, err = orc.check_out(out.cpu(), ref_out, slack)
    assert ok, err
    got = s.float().cpu()
    hidden = torch.isneginf(ref)
    assert torch.equal(torch.isneginf(got), hidden)
    # a stored 16-bit score is the fp32 one rounded once: half a unit in the last place
    rel = {"fp32": 0.0, "fp16": 2.0 ** -11, "bf16": 2.0 ** -8}[kind]
    x, r = got[~hidden], ref[~hidden]
    assert bool(((x - r).abs() <= (1e-3 + rel) * r.abs() + 1e-4).all())


@pytest.mark.parametrize("M,N", SHAPES)
@pytest.mark.parametrize("kind", ["fp32", "fp16", "bf16"])
def test_scores_only_in_odd_rows(M, N, kind):
    dtype = torch.bfloat16 if kind == "bf16" else torch.float16
    q, k, v = _inputs(M, N, 128, dtype)
    ref = orc.naive_attention_with_scores(q, k, v, False)[1]
    s = F.compute_attention_scores(q.cuda(), k.cuda(), scores_dtype=torch.float32 if kind == "fp32" else None)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    rel = {"fp32": 0.0, "fp16": 2.0 ** -11, "bf16": 2.0 ** -8}[kind]
    assert bool(((s.float().cpu() - ref).abs() <= (1e-3 + rel) * ref.abs() + 1e-4).all())


@pytest.mark.parametrize("M,N", [(5, 127), (129, 258), (257, 131)])
@pytest.mark.parametrize("D", [16, 32])
@pytest.mark.parametrize("kind", ["fp32", "fp16", "bf16"])
def test_scores_in_odd_rows_at_small_head_dims(M, N, D, kind):
    dtype = torch.bfloat16 if kind == "bf16" else torch.float16
    q, k, v = _inputs(M, N, D, dtype)
    ref_out, ref = orc.naive_attention_with_scores(q, k, v, False)
    out, s = F.attention_with_scores(q.cuda(), k.cuda(), v.cuda(), False,
                                     scores_dtype=torch.float32 if kind == "fp32" else dtype)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    slack = orc.bf16_out_slack(ref, v, ref_out) if kind == "bf16" else None
    ok, err = orc.check_out(out.cpu(), ref_out, slack)
    assert ok, err
    rel = {"fp32": 0.0, "fp16": 2.0 ** -11, "bf16": 2.0 ** -8}[kind]
    assert bool(((s.float().cpu() - ref).abs() <= (1e-3 + rel) * ref.abs() + 1e-4).all())


@pytest.mark.parametrize("B,M,N", [(16, 200, 131), (1, 129, 131), (1, 300, 257), (16, 130, 200)])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("kind", ["fp32", "fp16", "bf16"])
def test_scores_only_on_either_side_of_the_family_rule(B, M, N, D, kind):
    """Few tiles of a small head dim go to the CUDA cores, 64 heads to the tcgen05 kernel, odd rows or not."""
    dtype = torch.bfloat16 if kind == "bf16" else torch.float16
    q, k, _ = _inputs(M, N, D, dtype)
    ref = orc.naive_attention_with_scores(q, k, k, False)[1]
    s = F.compute_attention_scores(q.cuda().repeat(B, 1, 1, 1), k.cuda().repeat(B, 1, 1, 1),
                                   scores_dtype=torch.float32 if kind == "fp32" else dtype)
    if B == 16:
        assert F.last_backend() == "tcgen05"
    elif D == 16 or N == 257:
        assert F.last_backend() == "generic"
    rel = {"fp32": 0.0, "fp16": 2.0 ** -11, "bf16": 2.0 ** -8}[kind]
    assert bool(((s.float().cpu() - ref).abs() <= (1e-3 + rel) * ref.abs() + 1e-4).all())
    assert F.device_status() == 0


def test_window_of_odd_rows():
    M, N = 300, 301
    q, k, v = _inputs(M, N, 64, torch.float16)
    ref = orc.naive_attention_with_scores(q, k, v, True, p_seq=N - M)[1]
    scores = torch.full((1, 4, M, N), 7.0, device="cuda")
    F.attention_with_scores(q.cuda(), k.cuda(), v.cuda(), True, q_rows=(128, 271), scores=scores)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    assert bool((scores[:, :, :128] == 7.0).all()) and bool((scores[:, :, 271:] == 7.0).all())
    ok, viol, ok_mask = orc.check_scores(scores[:, :, 128:271].cpu(), ref[:, :, 128:271])
    assert ok and ok_mask, viol


@pytest.mark.parametrize("N", [257, 260])
def test_scores_of_many_heads(N):
    """More 128-row CTAs than SMs: the launches of 256-row CTAs (the shapes above run 128-row ones)."""
    g = torch.Generator().manual_seed(N)
    q, k, v = (torch.randn(1, h, N, 64, generator=g).half() for h in (76, 38, 38))
    ref_out, ref = orc.naive_attention_with_scores(q, k, v, True)
    out, s = F.attention_with_scores(q.cuda(), k.cuda(), v.cuda(), True)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    ok, err = orc.check_out(out.cpu(), ref_out)
    assert ok, err
    ok, viol, ok_mask = orc.check_scores(s.cpu(), ref)
    assert ok and ok_mask, viol
