"""The workloads whose speed is looked after: what users of the operators run, from the smallest call to the largest.

A case is a dict of plain values:
  op       the operator (a key of ``_OPS``), or "train": ``attention`` forward and backward
  dtype    "float16" or "bfloat16"
  B, Hq, Hk, M, N, D   batch, query heads, key/value heads, query rows, keys, head dimension
  causal   bottom-right aligned mask
  split    the cross-token operators' split position (0 for the other operators)
  dropout  dropout probability (0 = off)

The ranges the listed cases stand for, and that ``draw`` spreads its cases over:
  * B 1 to 16; query heads 4 to 32, multi-head or grouped (up to 7 query heads to a kv head); head dimension 32, 64 or 128
  * self-attention (M = N) over 128 to 8192 tokens for every operator, up to 16384 for the ones that keep no score
    tensor; lengths are whatever the text is, so odd ones are as common as round ones
  * continuing a sequence: 1 to 512 new rows against 256 to 32768 cached keys
  * causal and full; fp16 and bf16; dropout where a model trains with it
"""
import math

import torch

import flash_attn_with_score_b200 as F

_HEADS = [(4, 4), (8, 8), (12, 12), (16, 16), (32, 32), (32, 8), (28, 4), (16, 4), (16, 8)]

_SUMS = ("row_sum", "col_sum", "col_sum_sequential", "softmax_col_sum")
_CROSS = ("cross_qk_sum", "cross_softmax_sum", "cross_softmax_sum_buffered")

_OPS = {
    "attention": F.attention,
    "scores": F.attention_with_scores,
    "scores_only": F.compute_attention_scores,
    "row_sum": F.attention_with_row_sum,
    "col_sum": F.attention_with_col_sum,
    "col_sum_sequential": F.attention_with_col_sum_sequential,
    "softmax_col_sum": F.attention_with_softmax_col_sum,
    "cross_qk_sum": F.attention_cross_token_qk_sum,
    "cross_softmax_sum": F.attention_cross_token_softmax_sum,
    "cross_softmax_sum_buffered": F.attention_cross_token_softmax_sum_buffered,
}


def _case(op, dtype, B, Hq, Hk, M, N, D, causal, split=0, dropout=0.0, name=None):
    c = dict(op=op, dtype=dtype, B=B, Hq=Hq, Hk=Hk, M=M, N=N, D=D, causal=causal, split=split, dropout=dropout)
    return c if name is None else dict(c, name=name)


def listed():
    return [
        # The smallest call: one short prompt whose attention map is inspected.  Launch and host time count.
        _case("scores", "float16", 1, 8, 8, 512, 512, 64, True, name="scores_s512"),
        # The headline workload: output and the whole fp32 score tensor of a 32-head layer, a page of text.
        _case("scores", "float16", 1, 32, 32, 1024, 1024, 128, True, name="scores_s1024"),
        # The same question about a text of whatever length it has, on a grouped-query bf16 model.
        _case("scores", "bfloat16", 1, 28, 4, 1531, 1531, 128, True, name="scores_ragged"),
        # Per-query statistics of a grouped-query prefill.
        _case("row_sum", "bfloat16", 1, 28, 4, 4096, 4096, 128, True, name="row_sum_gqa"),
        # Per-key statistics of a long prefill, as used to rank cached tokens.
        _case("col_sum", "float16", 1, 32, 32, 8192, 8192, 128, True, name="col_sum_s8192"),
        # The largest: softmax mass per key over a long bidirectional batch.
        _case("softmax_col_sum", "bfloat16", 4, 32, 8, 16384, 16384, 128, False, name="softmax_col_sum_long"),
        # Small heads on image patches, an odd number of them: key importance for token pruning.
        _case("softmax_col_sum", "float16", 16, 8, 8, 785, 785, 32, False, name="softmax_col_sum_d32"),
        # What the last quarter of a prompt (the question) asks of the rest (the context).
        _case("cross_qk_sum", "float16", 2, 32, 8, 4096, 4096, 128, True, split=3072, name="cross_qk_sum"),
        # The same as softmax mass, the operator that trades scratch memory for a second pass.
        _case("cross_softmax_sum_buffered", "float16", 1, 32, 32, 2048, 2048, 128, True, split=768,
              name="cross_softmax_buffered"),
        # A training step of a grouped-query layer: output and the three gradients.
        _case("train", "bfloat16", 1, 28, 4, 4096, 4096, 128, True, name="train_gqa"),
        # A training step of a smaller model that uses attention dropout.
        _case("train", "float16", 4, 16, 16, 1024, 1024, 64, True, dropout=0.1, name="train_dropout"),
        # Decoding: one new row per sequence against a cache of whatever length it has reached.
        _case("attention", "bfloat16", 8, 32, 8, 1, 9001, 128, True, name="decode"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _length(rng, lo, hi):
    """A sequence length, log-uniform: half of them as they come, half rounded to a whole number of 64."""
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.5 else max(lo, min(hi, (n + 32) // 64 * 64))


def draw(rng):
    op = rng.choice(["scores", "scores", "scores_only", "row_sum", "col_sum", "col_sum_sequential", "softmax_col_sum",
                     "cross_qk_sum", "cross_softmax_sum", "cross_softmax_sum_buffered", "attention", "train", "train",
                     "decode", "decode"])
    dtype = rng.choice(["float16", "bfloat16"])
    Hq, Hk = rng.choice(_HEADS)
    B = _log_int(rng, 1, 16)
    if op == "decode":
        M = 1 if rng.random() < 0.5 else _log_int(rng, 1, 512)
        return _case("attention", dtype, B, Hq, Hk, M, _length(rng, max(256, M), 32768), rng.choice([64, 128, 128]), True)
    D = rng.choice([32, 64, 64, 128, 128, 128])
    dropout = 0.1 if op == "train" and rng.random() < 0.4 else 0.0
    stores = op in ("scores", "scores_only", "cross_softmax_sum_buffered")
    S = _length(rng, 128, 8192 if stores else 16384)
    causal = op != "scores_only" and rng.random() < 0.7
    # what the case may cost: score tensors of at most 1 GB, and for small heads, dropout and odd score rows 6e10
    # multiply-adds, so that no drawn case takes longer than the largest listed one on any of the kernel families
    cost = 3.5 if op == "train" else 1.5
    most = 6e10 if D == 32 or dropout or (stores and S % 4) else 4e12
    while S > 128 and (2 * B * Hq * D * cost * S * S > most or (stores and 4 * B * Hq * S * S > 1e9)):
        if B > 1:
            B -= 1
        else:
            S = max(128, S - (64 if S % 64 == 0 else 62))
    split = max(1, min(S - 1, int(S * rng.uniform(0.1, 0.9)))) if op in _CROSS else 0
    if split and rng.random() < 0.5:
        split = max(32, split // 32 * 32)
    return _case(op, dtype, B, Hq, Hk, S, S, D, causal, split, dropout)


def _dtype(case):
    return torch.float16 if case["dtype"] == "float16" else torch.bfloat16


def prepare(case, seed):
    """Queries, keys and values as they leave a model's projections, and the gradient that comes back in training."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    dt = _dtype(case)

    def rand(h, s):
        t = torch.empty((case["B"], h, s, case["D"]), device="cuda", dtype=dt)
        return t.normal_(generator=g)

    q, k, v = rand(case["Hq"], case["M"]), rand(case["Hk"], case["N"]), rand(case["Hk"], case["N"])
    state = {"case": dict(case), "q": q, "k": k, "v": v}
    if case["op"] == "train":
        for t in (q, k, v):
            t.requires_grad_(True)
        state["dout"] = rand(case["Hq"], case["M"])
        # the mask's random numbers come from a pair that the training step keeps, so that the step can be repeated
        state["philox"] = (int(seed) + 1, 0) if case["dropout"] else None
    return state


def run(state):
    c, q, k, v = state["case"], state["q"], state["k"], state["v"]
    if c["op"] == "train":
        out = F.attention(q, k, v, c["causal"], dropout_p=c["dropout"], philox=state["philox"])
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["dout"])
        return {"out": out, "dq": dq, "dk": dk, "dv": dv}
    fn = _OPS[c["op"]]
    if c["op"] == "scores_only":
        return fn(q, k)
    if c["op"] in _CROSS:
        return fn(q, k, v, c["split"], c["causal"])
    return fn(q, k, v, c["causal"])


def _pairs(case, i_begin=0, j_end=None):
    """Visible (query, key) pairs per head with query >= i_begin and key < j_end."""
    M, N = case["M"], case["N"]
    j_end, i_begin = N if j_end is None else j_end, min(i_begin, M)
    if not case["causal"]:
        return (M - i_begin) * j_end
    first, last = i_begin + N - M + 1, N  # keys that the first and the last row see
    full_from = max(first, j_end)         # rows from here on see all of the keys below j_end
    n_full = max(0, last - full_from + 1)
    n_part = (last - first + 1) - n_full
    return n_full * j_end + n_part * (first + first + n_part - 1) // 2


def work(case):
    """Two multiply-adds per pair and head dimension for q.k^T and P.v; a second q.k^T over the summed region where the
    weights have to be known before they can be added up; five contractions in a backward pass.  Every input read once,
    every output written once."""
    B, Hq, Hk, M, N, D = (case[x] for x in ("B", "Hq", "Hk", "M", "N", "D"))
    op, pairs = case["op"], _pairs(case)
    q, kv = B * Hq * M * D * 2, B * Hk * N * D * 2
    if op == "scores_only":
        return {"bytes": q + kv + B * Hq * M * N * 2, "flops": 2 * D * B * Hq * M * N}
    flops, size = 4 * pairs, 2 * q + 2 * kv
    if op == "train":
        flops += 10 * pairs
        size += 2 * q + 2 * kv  # dout, dq; dk, dv
    elif op == "scores":
        size += B * Hq * M * N * 4
    elif op == "row_sum":
        size += B * Hq * M * 4
    elif op in _SUMS:
        size += B * Hk * N * 4
    elif op in _CROSS:
        size += B * Hk * case["split"] * 4
    if op == "softmax_col_sum":
        flops += 2 * pairs
    elif op in ("cross_softmax_sum", "cross_softmax_sum_buffered"):
        flops += 2 * _pairs(case, case["split"], case["split"])
    return {"bytes": size, "flops": flops * D * B * Hq}


def tolerance(case):
    """Four times what the operators differ by from the same formulas in fp64: up to 2.8e-4 (fp16) and 2.9e-3 (bf16), the
    16-bit rounding of the results and of the weights that enter P.v; in training, where the operands of the gradients
    are rounded as well, up to 3.8e-4 and 2.9e-3."""
    if case["dtype"] == "bfloat16":
        return {"rel": 1.2e-2}
    return {"rel": 1.6e-3 if case["op"] == "train" else 1.2e-3}
