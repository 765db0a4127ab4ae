"""Plain calls, which go from Python to the C entry points in one native step, against the same calls the long way (which a
torch function mode forces): results, layouts, errors, and what is not plain."""
import pytest
import torch
from torch.overrides import TorchFunctionMode

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import _lib

pytestmark = pytest.mark.gpu


class _LongWay(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


OPS = {
    "attention": F.attention, "scores": F.attention_with_scores, "row_sum": F.attention_with_row_sum,
    "col_sum": F.attention_with_col_sum, "sequential": F.attention_with_col_sum_sequential,
    "softmax_col_sum": F.attention_with_softmax_col_sum,
    "col_sum_heads": lambda q, k, v, c: F.attention_with_col_sum(q, k, v, c, per_q_head=True),
    "scaled": lambda q, k, v, c: F.attention_with_scores(q, k, v, c, 0.3),
    "cross_qk": lambda q, k, v, c: F.attention_cross_token_qk_sum(q, k, v, 40, c),
    "cross_softmax": lambda q, k, v, c: F.attention_cross_token_softmax_sum(q, k, v, 40, c),
    "buffered": lambda q, k, v, c: F.attention_cross_token_softmax_sum_buffered(q, k, v, 40, c),
    "scores_only": lambda q, k, v, c: F.compute_attention_scores(q, k),
}


def _inputs(M, N, D, dtype, heads_last):
    g = torch.Generator(device="cuda").manual_seed(M + N)

    def rand(h, s):
        if heads_last:  # (B, S, H, D) in memory
            return torch.randn(2, s, h, D, device="cuda", generator=g).to(dtype).transpose(1, 2)
        return torch.randn(2, h, s, D, device="cuda", generator=g).to(dtype)
    return rand(4, M), rand(2, N), rand(2, N)


@pytest.mark.parametrize("op", OPS)
@pytest.mark.parametrize("M,N,D,dtype,heads_last", [
    (100, 100, 64, torch.float16, False), (129, 200, 128, torch.bfloat16, True), (1, 3000, 128, torch.float16, False),
    (50, 77, 16, torch.bfloat16, False)])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
def test_plain_call_is_the_call(op, M, N, D, dtype, heads_last, causal):
    q, k, v = _inputs(M, N, D, dtype, heads_last)
    native = []
    plain = _lib.plain_call
    try:
        _lib.plain_call = lambda *a: native.append(plain(*a)) or native[-1]
        short = OPS[op](q, k, v, causal)
        assert len(native) == 1 and native[0] is not None
        with _LongWay():
            long = OPS[op](q, k, v, causal)
        assert native[1] is None
    finally:
        _lib.plain_call = plain
    short, long = [x if isinstance(x, tuple) else (x,) for x in (short, long)]
    assert len(short) == len(long)
    for x, y in zip(short, long):
        assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and not x.requires_grad
        assert torch.equal(x, y)
    assert F.device_status() == 0


def test_what_is_not_plain_goes_the_long_way():
    q, k, v = _inputs(64, 64, 64, torch.float16, False)
    call = lambda *t: _lib.plain_call(_lib.OP_ROW_SUM, *t, True, None, 0, False)  # noqa: E731
    assert call(q, k, v) is not None
    wide = torch.empty(2, 4, 64, 72, device="cuda", dtype=q.dtype)
    for other in (wide[..., 1:65], wide[..., :64].transpose(2, 3), q.float(), q.cpu(), q[:, :, :0], q[0], q.bfloat16(), q[..., :32],
                  q[:, :3], torch.nn.Parameter(q).as_subclass(type("T", (torch.Tensor,), {}))):
        assert call(other, k, v) is None
    with pytest.raises(TypeError, match="float16 or bfloat16"):
        F.attention_with_row_sum(q.float(), k.float(), v.float())
    with pytest.raises(AssertionError):
        F.attention_with_row_sum(q[:, :3], k, v)
    out, sums = F.attention_with_row_sum(q.clone().requires_grad_(True), k, v, True)  # not differentiable, as ever
    assert not out.requires_grad and not sums.requires_grad
    with torch.inference_mode():
        assert torch.equal(F.attention(q, k, v, True), F.attention_with_row_sum(q, k, v, True)[0])
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    want = F.attention_with_col_sum(q, k, v, True)
    with torch.cuda.graph(graph, stream=stream):
        got = F.attention_with_col_sum(q, k, v, True)
    graph.replay()
    torch.cuda.synchronize()
    for x, y in zip(got, want):
        assert torch.equal(x, y)


def test_scales_that_only_float_takes():
    q, k, v = _inputs(64, 64, 64, torch.float16, False)
    assert torch.equal(F.attention(q, k, v, True, "0.25"), F.attention(q, k, v, True, 0.25))
    with pytest.raises(ValueError, match="could not convert"):
        F.attention(q, k, v, True, "a quarter")
