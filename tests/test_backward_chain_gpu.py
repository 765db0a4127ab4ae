"""The backward pass's launches overlap (each may begin while the one before it drains).  On grids of several waves, with
another operator on the same memory right behind them, they give the bits of launches that run one after the other."""
import hashlib
import os
import subprocess
import sys

import pytest
import torch

import flash_attn_with_score_b200 as F

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = [  # B, Hq, Hk, S, D, dropout
    (2, 32, 8, 1030, 128, 0.0),
    (2, 32, 32, 1024, 64, 0.0),
    (2, 16, 4, 1100, 64, 0.1),
    (2, 32, 8, 900, 32, 0.0),
]


def digests():
    got = []
    for B, Hq, Hk, S, D, p in CASES:
        g = torch.Generator(device="cuda").manual_seed(S)
        q, k, v, do = (torch.randn(B, h, S, D, device="cuda", generator=g).half() for h in (Hq, Hk, Hk, Hq))
        for t in (q, k, v):
            t.requires_grad_(True)
        for _ in range(3):
            out = F.attention(q, k, v, True, dropout_p=p, philox=(5, 0) if p else None)
            grads = torch.autograd.grad(out, (q, k, v), do)
            # its scratch is the backward pass's: the caching allocator hands the freed block on at once
            sums = F.attention_with_softmax_col_sum(q.detach(), k.detach(), v.detach(), True)
            h = hashlib.sha256()
            for t in (out, *grads, *sums):
                h.update(t.detach().float().cpu().numpy().tobytes())
            got.append(h.hexdigest())
    assert F.device_status() == 0
    return got


def test_overlapped_launches_give_the_bits_of_serial_ones():
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", PYTHONPATH=os.pathsep.join([ROOT, os.path.join(ROOT, "tests")]))
    run = subprocess.run([sys.executable, "-c", "import test_backward_chain_gpu as t; print(*t.digests())"], env=env, cwd=ROOT,
                         capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    assert digests() == run.stdout.split()[-3 * len(CASES):]
