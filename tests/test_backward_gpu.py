"""attention() under autograd: dq, dk, dv through the C ABI (faws_attention_backward) against the CPU
oracle's torch-autograd gradients of the same fp32 formulas (the reference's FlashAttention.backward,
flash.py:172-261)."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SHAPES = [
    # B, Hq, Hk, M, N, D
    (1, 2, 2, 128, 128, 64),
    (2, 4, 2, 96, 96, 32),
    (1, 4, 1, 100, 100, 128),
    (1, 2, 1, 64, 160, 64),      # M < N
    (1, 2, 2, 160, 64, 16),      # M > N: causal rows without a visible key
    (1, 6, 2, 384, 384, 128),
    (1, 2, 1, 200, 328, 64),
    (2, 2, 2, 640, 640, 128),
]


def _inputs(shape, dtype, seed):
    B, Hq, Hk, M, N, D = shape
    g = torch.Generator().manual_seed(seed)
    q = torch.randn(B, Hq, M, D, generator=g).to(dtype)
    k = torch.randn(B, Hk, N, D, generator=g).to(dtype)
    v = torch.randn(B, Hk, N, D, generator=g).to(dtype)
    do = torch.randn(B, Hq, M, D, generator=g).to(dtype)
    return q, k, v, do


def _run(q, k, v, do, causal, **kw):
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    out = F.attention(qd, kd, vd, causal, **kw)
    assert out.requires_grad and out.grad_fn is not None
    with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's: the backward pass's from here on
        out.backward(do.cuda())
    return out.detach(), qd.grad, kd.grad, vd.grad


def _check(got, ref, what, bf16, slack):
    for name, x, r, sl in zip(("dq", "dk", "dv"), got, ref, slack):
        assert x.shape == r.shape and x.dtype in (torch.float16, torch.bfloat16), (what, name, x.shape, r.shape)
        ok, viol, err = orc.check_grad(x.cpu(), r, bf16, sl)
        assert ok, f"{what} {name}: violation {viol}, max abs err {err}"


@pytest.mark.parametrize("backend", ["generic", "auto", "tcgen05"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_backward_matches_autograd_oracle(shape, causal, dtype, backend):
    B, Hq, Hk, M, N, D = shape
    if backend == "tcgen05" and D not in (64, 128):
        pytest.skip("the tcgen05 kernels take head dims 64 and 128")  # forcing them elsewhere raises (tested below)
    q, k, v, do = _inputs(shape, dtype, seed=7)
    ref = orc.attention_backward(q, k, v, do, causal, p_seq=N - M)
    out, dq, dk, dv = _run(q, k, v, do, causal, backend=backend)
    ref_out, _ = orc.naive_attention_with_scores(q, k, v, causal, p_seq=N - M)
    assert (out.float().cpu() - ref_out).abs().max() < (2e-3 if dtype == torch.float16 else 3e-2)
    bf16 = dtype == torch.bfloat16
    _check((dq, dk, dv), ref, f"{shape} causal={causal} {backend}", bf16,
           orc.grad_slack(q, k, v, do, causal, p_seq=N - M, bf16=bf16))
    assert F.device_status() == 0


def test_backward_one_kv_group_of_cfg3():
    """cfg3's shape restricted to one kv head with its 7 query heads (bf16, S=4096, D=128, causal)."""
    shape = (1, 7, 1, 4096, 4096, 128)
    q, k, v, do = _inputs(shape, torch.bfloat16, seed=3)
    v = (v.float() * 0.5).to(torch.bfloat16)
    ref = orc.attention_backward(q, k, v, do, True)
    out, dq, dk, dv = _run(q, k, v, do, True, backend="tcgen05")
    _check((dq, dk, dv), ref, "cfg3 kv group", True, orc.grad_slack(q, k, v, do, True, bf16=True))
    assert F.device_status() == 0


def test_backward_with_dropout_matches_masked_oracle():
    shape = (1, 4, 2, 192, 192, 64)
    B, Hq, Hk, M, N, D = shape
    q, k, v, do = _inputs(shape, torch.float16, seed=5)
    seed, offset, p_drop = 1234, 64, 0.2
    keep = orc.dropout_keep_mask(seed, offset, B, Hq, M, N, p_drop)
    ref = orc.attention_backward(q, k, v, do, True, keep=keep, dropout_p=p_drop)
    out, dq, dk, dv = _run(q, k, v, do, True, dropout_p=p_drop, philox=(seed, offset))
    _, scores = orc.naive_attention_with_scores(q, k, v, True)
    assert (out.float().cpu() - orc.dropout_out(scores, v, keep, p_drop)).abs().max() < 4e-3
    sl = orc.grad_slack(q, k, v, do, True)
    _check((dq, dk, dv), ref, "dropout", False, tuple(x / (1.0 - p_drop) for x in sl))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=["fp16", "bf16"])
@pytest.mark.parametrize("shape,causal,p_drop,philox", [
    ((2, 2, 2, 128, 128, 64), False, 0.1, (7, 0)),
    ((1, 6, 2, 300, 300, 128), True, 0.3, ((3 << 32) | 5, 2 ** 31 - 70000)),  # linear index passes 2**31
    ((1, 4, 1, 129, 257, 32), True, 0.5, (99, 4)),
    ((2, 3, 3, 257, 130, 16), False, 0.9, (2 ** 63 - 1, 0)),
    ((1, 4, 2, 1, 200, 64), True, 0.2, (5, 8)),
    ((1, 4, 2, 260, 260, 32), True, 0.0, None),
], ids=lambda x: "x".join(map(str, x)) if isinstance(x, tuple) else str(x))
def test_backward_fine_modes(shape, causal, p_drop, philox, dtype):
    """Dropout and small head dims on the tcgen05 kernels: dS in two 16-bit parts, so that nothing is further from
    the oracle than on the CUDA-core kernels, which hold dS in fp32 (2 % for the order of the sums)."""
    B, Hq, Hk, M, N, D = shape
    bf16 = dtype == torch.bfloat16
    q, k, v, do = _inputs(shape, dtype, seed=M + D)
    keep = orc.dropout_keep_mask(*philox, B, Hq, M, N, p_drop) if p_drop else None
    ref = orc.attention_backward(q, k, v, do, causal, p_seq=N - M, keep=keep, dropout_p=p_drop)
    runs = {be: _run(q, k, v, do, causal, dropout_p=p_drop, philox=philox, backend=be)[1:] for be in ("generic", "auto")}
    assert F.last_backend() == "tcgen05"
    sl = tuple(x / (1.0 - p_drop) for x in orc.grad_slack(q, k, v, do, causal, p_seq=N - M, bf16=bf16))
    _check(runs["auto"], ref, "fine", bf16, sl)
    for name, x, y, r in zip(("dq", "dk", "dv"), runs["auto"], runs["generic"], ref):
        ex, ey = ((t.double().cpu() - r.double()).norm() for t in (x, y))
        assert ex <= 1.02 * ey + 1e-6 * r.double().norm(), (name, ex.item(), ey.item())
    assert F.device_status() == 0


@pytest.mark.parametrize("shape,p_drop", [((1, 2, 2, 1024, 1024, 64), 0.1), ((1, 4, 2, 1100, 1100, 32), 0.0),
                                          ((2, 2, 1, 200, 1025, 128), 0.5), ((1, 2, 2, 1030, 1030, 16), 0.0)],
                         ids=lambda x: "x".join(map(str, x)) if isinstance(x, tuple) else str(x))
@pytest.mark.parametrize("size", [1e-5, 1e-4, 1e-3, 5e3])
def test_backward_fine_modes_over_the_size_of_the_gradient(shape, p_drop, size):
    """fp16, gradients of a mean loss and of a scaled one: as close to the oracle as the CUDA-core kernels' fp32 dS.  The
    large ones come with small q and k and large v, so that dS passes fp16's range and the results do not."""
    B, Hq, Hk, M, N, D = shape
    q, k, v, do = _inputs(shape, torch.float16, seed=N + D)
    do = (do.float() * size).half()
    if size > 1:
        q, k, v = q * 0.01, k * 0.01, v * 16
    philox = (17, 8) if p_drop else None
    keep = orc.dropout_keep_mask(*philox, B, Hq, M, N, p_drop) if p_drop else None
    ref = orc.attention_backward(q, k, v, do, True, p_seq=N - M, keep=keep, dropout_p=p_drop)
    runs = {be: _run(q, k, v, do, True, dropout_p=p_drop, philox=philox, backend=be)[1:] for be in ("generic", "auto")}
    assert F.last_backend() == "tcgen05"
    for name, x, y, r in zip(("dq", "dk", "dv"), runs["auto"], runs["generic"], ref):
        assert torch.isfinite(y).all() and torch.isfinite(x).all(), name
        ex, ey = ((t.double().cpu() - r.double()).norm() for t in (x, y))
        assert ex <= 1.02 * ey + 1e-6 * r.double().norm(), (name, ex.item(), ey.item())
    assert F.device_status() == 0


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_backward_fine_modes_keep_infinities_visible(bad):
    q, k, v, do = _inputs((1, 2, 2, 200, 200, 64), torch.float16, seed=2)
    do[0, 1, 77, 5] = bad
    _, dq, dk, dv = _run(q, k, v, do, True, dropout_p=0.1, philox=(3, 0))
    assert not torch.isfinite(dq[0, 1, 77]).any() and not torch.isfinite(dk[0, 1, :70]).all(dim=-1).any()
    assert torch.isfinite(dq[0, 0]).all() and torch.isfinite(dk[0, 0]).all() and torch.isfinite(dv[0, 0]).all()


@pytest.mark.parametrize("M", [100, 129, 128])
def test_backward_with_dropout_close_to_one_and_a_ragged_last_query_tile(M):
    """1 / (1 - p) = 1e5 is beyond fp16: the missing rows of the last query tile must not enter dV with it."""
    q, k, v, do = _inputs((1, 8, 8, M, 2048, 64), torch.float16, seed=M)
    runs = [_run(q, k, v, do, False, dropout_p=0.99999, philox=(5, 0), backend=be) for be in ("generic", "auto")]
    assert F.last_backend() == "tcgen05"
    for x, y in zip(*runs):
        assert torch.isfinite(x).all() and torch.isfinite(y).all()
        assert (x.double() - y.double()).norm() <= 2e-3 * x.double().norm()


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
def test_backward_with_very_negative_scores_and_a_ragged_last_key_tile(D, causal):
    """Every score near -200: exp(0 - L) of the missing keys of the last tile is infinite and must not be used."""
    g = torch.Generator().manual_seed(11)
    M, N = 150, 130 if not causal else 150
    c = (200.0 / D ** 0.5) ** 0.5
    q = (c + 0.02 * torch.randn(1, 2, M, D, generator=g)).half()
    k = (-c + 0.02 * torch.randn(1, 2, N, D, generator=g)).half()
    v, do = (torch.randn(1, 2, n, D, generator=g).half() for n in (N, M))
    ref = orc.attention_backward(q, k, v, do, causal, p_seq=N - M)
    out, dq, dk, dv = _run(q, k, v, do, causal)
    assert F.last_backend() == "tcgen05"
    _check((dq, dk, dv), ref, "negative scores", False, orc.grad_slack(q, k, v, do, causal, p_seq=N - M))


def test_backward_is_deterministic_and_frees_the_caller_from_L():
    q, k, v, do = _inputs((1, 4, 2, 320, 320, 64), torch.float16, seed=9)
    a = _run(q, k, v, do, True)
    b = _run(q, k, v, do, True)
    for x, y in zip(a, b):
        assert torch.equal(x, y)
    # the 5-tuple form is differentiable in its first element too
    qd = q.cuda().requires_grad_(True)
    out, L, tot, _, _ = F.attention(qd, k.cuda(), v.cuda(), True, return_log_normalizer=True,
                                    return_total_attention=True)
    assert not L.requires_grad and not tot.requires_grad
    out.sum().backward()
    assert qd.grad is not None and torch.isfinite(qd.grad.float()).all()
    with pytest.raises(ValueError):
        F.attention(qd, k.cuda(), v.cuda(), True, q_rows=(0, 128))


def test_forcing_the_tcgen05_backward_on_an_unsupported_problem_raises():
    q, k, v, do = _inputs((1, 2, 2, 64, 64, 32), torch.float16, seed=1)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    out = F.attention(qd, kd, vd, True)  # forward on whichever family fits
    with pytest.raises(RuntimeError):
        torch.autograd.grad(F.attention(qd, kd, vd, True, backend="tcgen05"), (qd,), do.cuda())
    del out
