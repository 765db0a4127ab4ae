"""Split-KV attention (few query rows, keys cut into ranges with a deterministic combine; the
reference's flash.py:68-70,97-134 and split_kv.py) against the CPU oracle and the unsplit kernel."""
import ctypes as C

import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import _lib
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [
    # B, Hq, Hk, M, N, D
    (1, 4, 2, 1, 2048, 128),     # one-token decode
    (2, 8, 2, 16, 4096, 128),
    (1, 2, 1, 128, 1024, 64),
    (1, 2, 2, 200, 1000, 64),    # ragged M and N
    (1, 4, 4, 130, 2048, 128),   # two query tiles, the second nearly empty
]


def _inputs(shape, dtype, seed=0):
    B, Hq, Hk, M, N, D = shape
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, Hq, M, D, generator=g).to(dtype)
    k = torch.randn(B, Hk, N, D, generator=g).to(dtype)
    v = torch.randn(B, Hk, N, D, generator=g).to(dtype)
    return q, k, v


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_split_kv_matches_oracle_and_unsplit(shape, causal, dtype):
    B, Hq, Hk, M, N, D = shape
    q, k, v = _inputs(shape, dtype, seed=13)
    ref_out, ref_scores = orc.naive_attention_with_scores(q, k, v, causal, p_seq=N - M)
    slack = orc.bf16_out_slack(ref_scores, v, ref_out) if dtype == torch.bfloat16 else None
    Lref = orc.log_normalizer(ref_scores)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    one, L1, _, _, _ = F.attention(qd, kd, vd, causal, return_log_normalizer=True, kv_splits=1)
    for splits in (None, 2, 5, (N + 127) // 128):
        out, L, _, _, _ = F.attention(qd, kd, vd, causal, return_log_normalizer=True, kv_splits=splits)
        assert F.last_backend() == "tcgen05"
        ok, err = orc.check_out(out.cpu(), ref_out, slack)
        assert ok, (splits, err)
        fin = torch.isfinite(Lref)
        assert torch.equal(torch.isneginf(L.cpu()), ~fin)
        assert (L.cpu()[fin] - Lref[fin]).abs().max() < 2e-3
        # the sums of the ranges are added in another order, and out may round the other way
        assert (out.float() - one.float()).abs().max() < (4e-3 if dtype == torch.float16 else 3e-2)
        again = F.attention(qd, kd, vd, causal, kv_splits=splits)
        assert torch.equal(again, out), "the combine must be deterministic"
    assert F.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("shape,splits", [((2, 32, 8, 1, 4000, 32), 8), ((1, 8, 8, 40, 2000, 16), 4),
                                          ((4, 32, 8, 16, 1000, 128), 2), ((2, 8, 4, 130, 1500, 64), 12)],
                         ids=lambda x: "x".join(map(str, x)) if isinstance(x, tuple) else str(x))
def test_splitting_the_keys_adds_no_rounding(shape, splits, dtype):
    """Partial results are fp32: the distance of out from fp64 is that of the unsplit call (16-bit partial results made it
    1.22 times as large; 6 % for the sample, 8 k values and more)."""
    q, k, v = (t.cuda() for t in _inputs(shape, dtype, seed=splits))
    G = shape[1] // shape[2]
    s = q.double() @ k.double().repeat_interleave(G, 1).transpose(-1, -2) / shape[5] ** 0.5
    M, N = shape[3], shape[4]
    s = s.masked_fill(torch.ones(M, N, dtype=torch.bool, device="cuda").triu(N - M + 1), float("-inf"))
    ref = s.softmax(-1) @ v.double().repeat_interleave(G, 1)
    one, cut = ((F.attention(q, k, v, True, kv_splits=n).double() - ref).norm().item() for n in (1, splits))
    assert F.last_backend() == "tcgen05"
    assert cut <= 1.06 * one, (cut / ref.norm().item(), one / ref.norm().item())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("interleaved", [False, True], ids=["bhsd", "bshd"])
@pytest.mark.parametrize("shape", [
    (2, 8, 2, 16, 300, 64),      # four heads in half a tile
    (1, 7, 1, 40, 515, 128),     # 280 packed rows: heads across tile edges, a third tile of 24 rows
    (2, 4, 1, 129, 1300, 64),    # 516 packed rows in 5 tiles instead of 8
    (1, 8, 1, 16, 16, 32),       # self-attention, exactly one tile
    (1, 4, 1, 33, 33, 128),      # self-attention, one row more than a tile: two tiles instead of four
    (1, 4, 1, 100, 100, 64),     # self-attention: not packed
    (1, 2, 1, 2, 257, 128),      # a last key tile of one key, hidden from the first row of each head
], ids=lambda s: "x".join(map(str, s)))
def test_few_causal_rows_with_grouped_queries(shape, interleaved, dtype):
    """The heads of a group share a query tile and each row keeps its own causal limit (interleaved heads cannot be
    packed and take the general route)."""
    B, Hq, Hk, M, N, D = shape
    q, k, v = _inputs(shape, dtype, seed=M)
    ref_out, ref_scores = orc.naive_attention_with_scores(q, k, v, True, p_seq=N - M)
    slack = orc.bf16_out_slack(ref_scores, v, ref_out) if dtype == torch.bfloat16 else None
    Lref = orc.log_normalizer(ref_scores)
    if interleaved:
        q = q.transpose(1, 2).contiguous().transpose(1, 2)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    for splits in {None, 1, min(3, (N + 127) // 128), (N + 127) // 128}:
        out, L, _, _, _ = F.attention(qd, kd, vd, True, return_log_normalizer=True, kv_splits=splits)
        assert F.last_backend() == "tcgen05"
        ok, err = orc.check_out(out.cpu(), ref_out, slack)
        assert ok, (splits, err)
        assert (L.cpu() - Lref).abs().max() < 2e-3
    assert F.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("shape,causal", [
    ((16, 28, 4, 40, 515, 64), True),    # 280 packed rows in three tiles, 192 CTAs instead of 448
    ((16, 28, 4, 40, 515, 128), True),
    ((12, 32, 4, 33, 260, 32), True),    # 264 packed rows: the third tile has eight
    ((20, 16, 2, 70, 300, 64), False),   # no mask: 560 packed rows in five tiles instead of eight
], ids=lambda x: "x".join(map(str, x)) if isinstance(x, tuple) else ("causal" if x else "full"))
def test_packed_heads_over_several_tiles(shape, causal, dtype):
    """Shapes whose packed launch is the shorter one; the same call with heads that cannot be packed agrees."""
    B, Hq, Hk, M, N, D = shape
    q, k, v = _inputs(shape, dtype, seed=M)
    ref_out, ref_scores = orc.naive_attention_with_scores(q, k, v, causal, p_seq=N - M)
    slack = orc.bf16_out_slack(ref_scores, v, ref_out) if dtype == torch.bfloat16 else None
    Lref = orc.log_normalizer(ref_scores)
    qd, kd, vd = q.cuda(), k.cuda(), v.cuda()
    apart = torch.empty(B, Hq, M + 8, D, device="cuda", dtype=dtype)[:, :, :M].copy_(qd)
    for x in (qd, apart):
        out, L, _, _, _ = F.attention(x, kd, vd, causal, return_log_normalizer=True)
        assert F.last_backend() == "tcgen05"
        ok, err = orc.check_out(out.cpu(), ref_out, slack)
        assert ok, err
        assert (L.cpu() - Lref).abs().max() < 2e-3
    assert F.device_status() == 0


def test_split_plan_follows_the_occupancy_rule():
    lib = _lib.load()
    q, k, v = (t.cuda() for t in _inputs((1, 4, 2, 16, 16384, 128), torch.float16))
    out = torch.empty_like(q)

    def plan(qq, kk, vv, causal=False, dropout=0.0):
        p = _lib.Problem()
        p.B, p.Hq, p.M, p.D = qq.shape
        p.Hk, p.N = kk.shape[1], kk.shape[2]
        p.dtype, p.causal, p.sm_scale, p.m_end = _lib.FP16, int(causal), 0.088, qq.shape[2]
        t = lambda x: _lib.Tensor(x.data_ptr(), x.stride(0), x.stride(1), x.stride(2))  # noqa: E731
        p.q, p.k, p.v, p.out = t(qq), t(kk), t(vv), t(torch.empty_like(qq))
        p.dropout_p = dropout
        return lib.faws_split_kv_plan(C.byref(p))

    assert plan(q, k, v) > 1                      # 4 CTAs on 148 SMs: split
    assert plan(q, k, v, dropout=0.1) == 1        # never with dropout (flash.py:98)
    big = torch.empty(4, 32, 1024, 128, device="cuda", dtype=torch.float16)
    assert plan(big, big, big) == 1               # 1024 CTAs: enough work already
    del out
    # 96 to 118 CTAs of a few key tiles: the wave rule alone would cut them, for three times the time
    for B, Hq, Hk, M, N, causal in ((4, 16, 4, 200, 1500, True), (2, 12, 12, 500, 512, True), (1, 28, 4, 513, 513, False)):
        qq, kk = (torch.empty(B, h, s, 128, device="cuda", dtype=torch.float16) for h, s in ((Hq, M), (Hk, N)))
        assert plan(qq, kk, kk, causal) == 1, (B, Hq, M, N)
