"""Odd score rows: which row count a launch of fewer than two 256-row CTAs per SM takes on either side of its lines (148
SMs), the scores it leaves, and windows of query rows in launches of 256-row CTAs."""
import json
import os
import subprocess
import sys

import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# B, H, Hk, M, N, D, causal, type of the scores, row count of a CTA
CHOICES = [
    (1, 83, 83, 257, 257, 64, True, "float32", 256), (1, 82, 82, 257, 257, 64, True, "float32", 128),   # 249, 246 CTAs of 128 rows
    (2, 42, 14, 300, 413, 128, True, "float32", 256), (2, 41, 41, 300, 413, 128, True, "float32", 128),
    (1, 74, 37, 257, 301, 64, False, "float32", 256), (1, 75, 25, 257, 301, 64, False, "float32", 128),  # 148, 150 CTAs of 256 rows
    (2, 24, 6, 700, 515, 128, False, "float32", 256), (2, 28, 4, 700, 515, 128, False, "float32", 128),
    (1, 44, 11, 515, 515, 64, True, "input", 256), (1, 29, 29, 515, 515, 64, True, "input", 128)]

CHILD = """
import hashlib, json, sys
sys.path.insert(0, sys.argv[1])
import torch
import flash_attn_with_score_b200 as F
shas = []
for B, H, Hk, M, N, D, causal, kind, *_ in json.loads(sys.argv[2]):
    dt = getattr(torch, sys.argv[3])
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q, k, v = [torch.randn(B, h, s, D, device="cuda", generator=g).to(dt) for h, s in ((H, M), (Hk, N), (Hk, N))]
    out, scores = F.attention_with_scores(q, k, v, causal, scores_dtype=torch.float32 if kind == "float32" else dt)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    want = (q.float() @ k.float().repeat_interleave(H // Hk, 1).mT) * D ** -0.5
    seen = torch.ones(M, N, dtype=torch.bool, device="cuda")
    if causal:
        seen = seen.tril(N - M)
    assert bool((scores[:, :, ~seen] == float("-inf")).all())
    # fp32 as the oracle bounds scores; 16 bits: half a unit in the last place more (2^-11 fp16, 2^-8 bf16)
    rel = 1e-3 + (0.0 if kind == "float32" else 2.0 ** -11 if dt == torch.float16 else 2.0 ** -8)
    assert bool(((scores.float() - want).abs() <= rel * want.abs() + 1e-4)[:, :, seen].all())
    shas.append(hashlib.sha256(out.view(torch.uint8).cpu().numpy().tobytes()).hexdigest())
print(json.dumps(shas))
"""


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_the_row_count_that_runs(dtype):
    """As for the other launches: the running maxima that a row's weights are rounded against differ with the row count, and
    with them the bits of the output."""
    got = {}
    for forced in ("0", "1", None):  # FAWS_SPLIT_KV is read once per process
        env = {x: y for x, y in os.environ.items() if x != "FAWS_SPLIT_KV"}
        if forced is not None:
            env["FAWS_SPLIT_KV"] = forced
        r = subprocess.run([sys.executable, "-c", CHILD, ROOT, json.dumps(CHOICES), dtype], env=env, capture_output=True,
                           text=True, timeout=600, cwd=ROOT)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
        got[forced] = json.loads(r.stdout.splitlines()[-1])
    for x, shape in enumerate(CHOICES):
        assert got["0"][x] != got["1"][x], shape
        assert got[None][x] == got["0" if shape[-1] == 256 else "1"][x], shape


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("lo,hi", [(128, 271), (0, 257), (256, 300)])
@pytest.mark.parametrize("N", [301, 302, 303])
def test_window_of_odd_rows_of_many_heads(N, lo, hi, dtype):
    B, H, M, D = 2, 150, 300, 64  # 300 CTAs of 256 rows or more
    g = torch.Generator(device="cuda").manual_seed(N + lo)
    q, k, v = [torch.randn(B, h, s, D, device="cuda", generator=g).to(dtype) for h, s in ((H, M), (H // 3, N), (H // 3, N))]
    scores = torch.full((B, H, M, N), 7.0, device="cuda")
    F.attention_with_scores(q, k, v, True, q_rows=(lo, hi), scores=scores)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    assert bool((scores[:, :, :lo] == 7.0).all()) and bool((scores[:, :, hi:] == 7.0).all())
    want = (q.float() @ k.float().repeat_interleave(3, 1).mT) * D ** -0.5
    want = want.masked_fill(~torch.ones(M, N, dtype=torch.bool, device="cuda").tril(N - M), float("-inf"))
    ok, viol, ok_mask = orc.check_scores(scores[:, :, lo:hi].cpu(), want[:, :, lo:hi].cpu())
    assert ok and ok_mask, viol
