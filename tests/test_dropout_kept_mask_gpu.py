"""Training with dropout where the forward pass leaves the mask to the backward pass: bit for bit what the passes compute
that each draw it themselves, under saved-tensor hooks and repeated backward passes as well."""
import pytest
import torch

import flash_attn_with_score_b200 as F
from flash_attn_with_score_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hk,M,N,D,causal,dtype", [
    (4, 8, 8, 512, 512, 32, True, torch.float16),         # 1 MB, as much as the queries: the smallest and the longest kept
    (1, 32, 8, 1000, 700, 64, True, torch.bfloat16),      # rows that see no key
    (2, 16, 4, 900, 1700, 128, True, torch.float16),
    (1, 64, 64, 300, 260, 128, False, torch.bfloat16),
    (1, 96, 32, 257, 129, 64, False, torch.float16)])
def test_kept_mask(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    q, k, v, do = [torch.randn(B, h, s, D, device="cuda", generator=g).to(dtype)
                   for h, s in ((Hq, M), (Hk, N), (Hk, N), (Hq, M))]
    for t in (q, k, v):
        t.requires_grad_(True)
    lib, sizes = _lib.load(), []
    size_of = lib.faws_dropout_mask_bytes

    def step(keep, moved=False):
        def mask_bytes(p):
            sizes.append(size_of(p))
            return sizes[-1] if keep else 0
        monkeypatch.setattr(lib, "faws_dropout_mask_bytes", mask_bytes)
        pack = (lambda t: t.cpu()) if moved else (lambda t: t)
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
            out = F.attention(q, k, v, causal, dropout_p=0.3, philox=(11, 8))
        assert F.last_backend() == "tcgen05"
        return (out, *torch.autograd.grad(out, (q, k, v), do, retain_graph=True), *torch.autograd.grad(out, (q, k, v), do))

    drawn = step(False)
    tiles = -(-M // 128) * -(-N // 128)
    assert sizes == [B * Hq * tiles * 2048]
    for kept in (step(True), step(True, moved=True)):
        for x, y in zip(kept, drawn):
            assert torch.equal(x, y)
    with torch.no_grad():
        assert torch.equal(F.attention(q, k, v, causal, dropout_p=0.3, philox=(11, 8)), drawn[0])
    assert F.device_status() == 0


def test_saved_tensors_that_come_back_elsewhere():
    """Hooks that give the tensors back at addresses that TMA cannot read: the CUDA-core kernels, which draw the mask."""
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = [torch.randn(1, 64, 300, 128, device="cuda", generator=g).half() for _ in range(4)]
    for t in (q, k, v):
        t.requires_grad_(True)

    def elsewhere(t):
        return torch.empty(t.numel() + 1, device="cuda", dtype=t.dtype)[1:].view(t.shape).copy_(t)
    grads = []
    for unpack in (lambda t: t, elsewhere):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            out = F.attention(q, k, v, True, dropout_p=0.3, philox=(11, 8))
        assert out.grad_fn.saved_tensors[5] is not None
        with torch.autograd.set_multithreading_enabled(False):  # last_backend() is this thread's
            grads.append(torch.autograd.grad(out, (q, k, v), do))
        assert F.last_backend() == ("tcgen05" if len(grads) == 1 else "generic")
    for x, y in zip(*grads):  # 16-bit weights and results on both families
        assert (x.double() - y.double()).norm() <= 2e-3 * y.double().norm()


def test_what_keeps_no_mask():
    """Larger than the queries, smaller than 1 MB, no gradient wanted, rows that TMA cannot read: the plain calls."""
    for M, N, D, H, off in ((512, 1100, 64, 16, 0), (256, 256, 64, 8, 0), (1024, 1024, 64, 16, 1)):
        q, k, v = [torch.randn(1, H, s, D + 8, device="cuda").half()[..., off:off + D].requires_grad_(True) for s in (M, N, N)]
        out = F.attention(q, k, v, True, dropout_p=0.2, philox=(1, 2))
        assert out.grad_fn.saved_tensors[5] is None
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), torch.ones_like(out))
        assert bool(torch.isfinite(dq).all() and torch.isfinite(dk).all() and torch.isfinite(dv).all())


@pytest.mark.parametrize("B,Hq,Hk,M,N,D,causal,dtype", [
    (1, 16, 16, 1000, 1023, 64, True, torch.float16),  # the last key tile of a kept mask
    (1, 32, 8, 400, 500, 32, False, torch.bfloat16),
    (1, 8, 8, 1930, 2000, 128, True, torch.float16)])
def test_kept_mask_of_lengths_between_whole_tiles(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype):
    test_kept_mask(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype)


def test_which_masks_are_kept():
    """Up to 16 D keys; among causal rows that see no key, in bytes no larger than the queries."""
    for M, N, causal, kept in ((1000, 1024, True, True), (1000, 1025, True, False), (1025, 1000, True, False),
                               (1025, 1000, False, True), (1152, 1000, True, True)):
        q, k, v = [torch.randn(1, 16, s, 64, device="cuda").half().requires_grad_(True) for s in (M, N, N)]
        out = F.attention(q, k, v, causal, dropout_p=0.2, philox=(1, 2))
        assert (out.grad_fn.saved_tensors[5] is not None) == kept


@pytest.mark.parametrize("B,Hq,Hk,M,N,D,causal,dtype", [
    (3, 64, 16, 333, 300, 64, True, torch.bfloat16),  # rows that see no key
    (1, 128, 32, 520, 650, 128, True, torch.float16),
    (2, 74, 74, 250, 515, 128, False, torch.float16),
    (8, 16, 4, 768, 400, 32, True, torch.bfloat16)])
def test_mask_that_the_forward_kernel_leaves(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype):
    test_kept_mask(monkeypatch, B, Hq, Hk, M, N, D, causal, dtype)


@pytest.mark.parametrize("H,M,causal,launches", [
    (186, 256, True, 1), (184, 256, True, 2), (148, 256, False, 1), (150, 256, False, 2), (148, 300, False, 2), (254, 129, False, 1)])
def test_where_the_mask_is_drawn(H, M, causal, launches):
    """In the forward kernel where its CTAs fill the SMs, so that a forward pass is not slower for what it leaves; else by a
    launch of its own.  (148 SMs.)"""
    q, k, v = [torch.randn(1, H, s, 64, device="cuda").half().requires_grad_(True) for s in (M, 256, 256)]
    before = F.launch_count()
    out = F.attention(q, k, v, causal, dropout_p=0.2, philox=(1, 2))
    assert F.launch_count() - before == launches
    assert out.grad_fn.saved_tensors[5] is not None
