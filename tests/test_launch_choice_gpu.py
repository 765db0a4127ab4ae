"""Launches of fewer than two 256-row CTAs per SM: both row counts of a CTA, on either side of the choice between them."""
import json
import os
import subprocess
import sys

import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hk,M,N,D,causal", [
    (40, 40, 512, 512, 64, False), (32, 32, 512, 512, 64, False), (144, 36, 300, 300, 64, True),
    (32, 8, 513, 1025, 128, True), (48, 12, 700, 700, 128, True), (20, 20, 1030, 1030, 64, True),
    (147, 49, 257, 129, 32, False), (150, 50, 257, 129, 32, False)])
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


ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
# H, Hk, M, N, D, causal, then the row count of a CTA expected for the plain output, row sums, column sums.  75 to 295
# CTAs of 256 rows; the larger ones among those that take them walk a work list.
ROWS = [
    (40, 8, 1531, 1531, 128, True, 256, 256, 256), (144, 48, 512, 512, 64, False, 256, 256, 256),
    (32, 32, 2048, 2048, 128, True, 256, 256, 256), (147, 147, 257, 129, 32, False, 256, 256, 256),
    (40, 40, 512, 512, 64, False, 256, 256, 256), (28, 4, 1531, 1531, 128, True, 128, 128, 128),
    (28, 28, 2048, 700, 64, True, 128, 128, 128), (40, 40, 512, 512, 64, True, 128, 128, 128)]

CHILD = """
import hashlib, json, sys
sys.path.insert(0, sys.argv[1])
import torch
import flash_attn_with_score_b200 as F
shas = []
for H, Hk, M, N, D, causal, *_ in json.loads(sys.argv[2]):
    g = torch.Generator(device="cuda").manual_seed(H + M)
    q, k, v = [torch.randn(1, h, s, D, device="cuda", generator=g).to(getattr(torch, sys.argv[3]))
               for h, s in ((H, M), (Hk, N), (Hk, N))]
    for out in (F.attention(q, k, v, causal, kv_splits=1), F.attention_with_row_sum(q, k, v, causal)[0],
                F.attention_with_col_sum(q, k, v, causal)[0]):
        assert F.last_backend() == "tcgen05" and F.device_status() == 0
        shas.append(hashlib.sha256(out.view(torch.uint8).cpu().numpy().tobytes()).hexdigest())
print(json.dumps(shas))
"""


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_the_row_count_that_runs(dtype):
    """The weights of a row are rounded against one running maximum with 256 rows and against two with 128, which shows in
    the bits of the output: those of a free launch are those of a launch whose row count is forced."""
    got = {}
    for forced in ("0", "1", None):  # FAWS_SPLIT_KV is read once per process
        env = {x: y for x, y in os.environ.items() if x != "FAWS_SPLIT_KV"}
        if forced is not None:
            env["FAWS_SPLIT_KV"] = forced
        r = subprocess.run([sys.executable, "-c", CHILD, ROOT, json.dumps(ROWS), dtype], env=env, capture_output=True,
                           text=True, timeout=600, cwd=ROOT)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
        got[forced] = json.loads(r.stdout.splitlines()[-1])
    ran = [rows for shape in ROWS for rows in shape[6:]]
    for x, rows in enumerate(ran):
        what = (ROWS[x // 3], ("plain", "row sums", "column sums")[x % 3])
        assert got["0"][x] != got["1"][x], what
        assert got[None][x] == got["0" if rows == 256 else "1"][x], what
