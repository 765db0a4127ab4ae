"""Odd score rows in launches of 256-row CTAs, whose whole key tiles go out 16 bytes a lane: every distance of a row's start
from a 16-byte boundary, one to four whole tiles and a remainder of none, one, a few and all but one key.  Nothing outside
the tensor may be written: it lies inside a larger buffer whose margins are checked."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(300, 301), (257, 258), (270, 131), (256, 129), (300, 255), (290, 256), (130, 515), (256, 128)])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_scores_in_odd_rows_of_whole_tiles(M, N, causal, shift):
    H, D = 300 if M <= 256 else 160, 64 if M % 2 else 128  # at least 296 CTAs of 256 rows
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    q, k, v = [torch.randn(1, h, s, D, device="cuda", generator=g).half() for h, s in ((H, M), (H // 4, N), (H // 4, N))]
    n = H * M * N
    buf = torch.full((n + 130,), 7.0, device="cuda")
    lo = 64 + shift
    scores = buf[lo:lo + n].view(1, H, M, N)
    out, _ = F.attention_with_scores(q, k, v, causal, scores=scores)
    assert F.last_backend() == "tcgen05" and F.device_status() == 0
    assert bool((buf[:lo] == 7.0).all()) and bool((buf[lo + n:] == 7.0).all())
    want = (q.float() @ k.float().repeat_interleave(4, 1).mT) * D ** -0.5
    seen = torch.ones(M, N, dtype=torch.bool, device="cuda")
    if causal:
        seen = seen.tril(N - M)
    # the hidden set bit for bit; the others as orc.check_scores bounds them
    assert bool((scores[:, :, ~seen] == float("-inf")).all())
    assert bool(((scores - want).abs() <= 1e-3 * want.abs() + 1e-4)[:, :, seen].all())
    rows = seen.any(-1)
    ref = want.masked_fill(~seen, float("-inf"))[:, :, rows].softmax(-1) @ v.float().repeat_interleave(4, 1)
    ok, err = orc.check_out(out[:, :, rows].cpu(), ref.cpu())
    assert ok, err
