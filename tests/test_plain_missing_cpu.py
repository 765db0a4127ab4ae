"""Operators where _plain.so is missing or was built for another torch: the long way, with its results and errors."""
import os
import subprocess
import sys

import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import _lib

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture
def no_plain(monkeypatch):
    monkeypatch.setattr(_lib, "_plain", None)
    monkeypatch.delattr(F, "_plain", raising=False)
    monkeypatch.setitem(sys.modules, "flash_attn_with_score_b200._plain", None)


def test_errors_are_the_long_ways(no_plain):
    q, k = torch.zeros(1, 4, 8, 64, dtype=torch.float16), torch.zeros(1, 2, 8, 64, dtype=torch.float16)
    for op in (F.attention, F.attention_with_scores, F.attention_with_row_sum, F.attention_with_col_sum,
               F.attention_with_softmax_col_sum):
        with pytest.raises(RuntimeError, match="CUDA tensors only"):
            op(q, k, k)
        with pytest.raises(AssertionError, match="feature size"):
            op(q, k[..., :32], k)
    with pytest.raises(RuntimeError, match="CUDA tensors only"):
        F.compute_attention_scores(q, k)
    assert _lib._plain is False


@pytest.mark.gpu
def test_operators_without_the_module(no_plain):
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v = [torch.randn(1, h, 200, 64, device="cuda", generator=g).half() for h in (4, 2, 2)]
    got = F.attention_with_scores(q, k, v, True), F.attention_cross_token_qk_sum(q, k, v, 90, True)
    assert _lib._plain is False and F.last_backend() == "tcgen05"
    _lib._plain = None
    sys.modules.pop("flash_attn_with_score_b200._plain")
    want = F.attention_with_scores(q, k, v, True), F.attention_cross_token_qk_sum(q, k, v, 90, True)
    assert _lib._plain  # the module is there
    for x, y in zip(got, want):
        assert all(torch.equal(a, b) for a, b in zip(x, y))


def test_a_module_for_another_torch_is_not_used():
    child = ("import torch\ntorch.__version__ = '1.0.0'\nfrom flash_attn_with_score_b200 import _lib\n"
             "q = torch.zeros(1, 1, 8, 64)\n"
             "assert _lib.plain_call(_lib.OP_ROW_SUM, q, q, q, True, None, 0, False) is None and _lib._plain is False\n"
             "try:\n    from flash_attn_with_score_b200 import _plain\n"
             "except ImportError as e:\n    assert 'built for torch' in str(e), e\nelse:\n    raise SystemExit('loaded')\n")
    r = subprocess.run([sys.executable, "-c", child], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
