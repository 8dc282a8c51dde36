"""Workloads for timing the library through its public entry points.

Every case is one call that a program using this library makes over and over:

    forward  the registered attention function in inference, as each decoder layer calls it
             (``raw``: at the layer that also returns the raw logits of the last rows)
    scores   the fused per-document score epilogue of the scoring layer
    train    the registered attention function under autograd, forward and backward
             (``raw``: the layer whose raw logits feed the auxiliary ranking loss)
    rank     the early-exit ranker on host tensors: token ids in, document logits out

A prompt is an instruction block, ``docs`` documents of ``doc_lo``..``doc_hi`` tokens (drawn from
``shape_seed``) and a query block.  ``layout`` is "grid" (the block collator's left-padded (M, H) grid,
what a Hugging Face model is called with) or "packed" (the padding-free layout).
"""
import random

import torch

from blockrank_b200 import (BlockSpans, cuda_blockrank_attention_forward, cuda_blockrank_attention_mask, ops,
                            packed_block_collate_fn)
from blockrank_b200.runner import MistralPrefillRanker, RankerConfig

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
RAW_ROWS = 16  # the attention function's default ``num_last_queries``
SIGNAL_ROWS = 2


def _op(name, kind, prompts, docs, doc_lo, doc_hi, layout, heads=32, kv_heads=8, head_dim=128, dtype="bf16", raw=False,
        instr=64, query=48, shape_seed=5):
    return {"name": name, "kind": kind, "prompts": prompts, "docs": docs, "doc_lo": doc_lo, "doc_hi": doc_hi,
            "instr": instr, "query": query, "layout": layout, "heads": heads, "kv_heads": kv_heads, "head_dim": head_dim,
            "dtype": dtype, "raw": raw, "shape_seed": shape_seed}


def _rank(name, model, prompts, docs, doc_lo, doc_hi, instr=64, query=48, shape_seed=5):
    return {"name": name, "kind": "rank", "model": model, "prompts": prompts, "docs": docs, "doc_lo": doc_lo,
            "doc_hi": doc_hi, "instr": instr, "query": query, "shape_seed": shape_seed}


def listed():
    return [
        # one short request: a handful of passages, where launches and the host path are most of the time
        _op("forward_5docs", "forward", 1, 5, 35, 90, "packed", instr=27, query=19),
        # a batch of short ranking lists on the padded grid a Hugging Face model is called with
        _op("forward_20docs_grid", "forward", 4, 20, 160, 160, "grid"),
        # the benchmark's forward pass: 4 prompts of 100 documents, padding-free
        _op("forward_100docs", "forward", 4, 100, 160, 160, "packed"),
        # the longest lists: 500 documents of very different lengths in one prompt (about 72,000 tokens)
        _op("forward_500docs_ragged", "forward", 1, 500, 32, 256, "packed"),
        # evaluation through a Hugging Face model: the scoring layer returns the raw logits of the last 16 slots
        _op("forward_raw_100docs", "forward", 1, 100, 160, 160, "grid", raw=True),
        # the same in 32 bits, as parity runs and models kept in float32 use it
        _op("forward_raw_20docs_f32", "forward", 1, 20, 120, 160, "grid", dtype="f32", raw=True),
        # the ranker's scoring layer: document scores of a batch
        _op("scores_100docs", "scores", 4, 100, 160, 160, "packed"),
        # fine-tuning, the layer with the auxiliary ranking loss
        _op("train_raw_20docs", "train", 4, 20, 160, 160, "grid", raw=True),
        # fine-tuning, every other layer, long lists of documents of different lengths
        _op("train_100docs_ragged", "train", 1, 100, 32, 256, "grid"),
        # fine-tuning a small model: head_dim 64, two query heads per key head, short ragged documents
        _op("train_raw_12docs_d64", "train", 2, 12, 17, 120, "grid", heads=16, kv_heads=8, head_dim=64, raw=True),
        # one ranking request end to end on the small model: latency
        _rank("rank_small_10docs", "tiny", 1, 10, 40, 120),
        # one ranking request end to end on the 7B architecture, the benchmark's prompt
        _rank("rank_7b_100docs", "7b", 1, 100, 160, 160),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "scores", "train", "train", "rank"])
    doc_hi = _log_int(rng, 24, 256)
    doc_lo = doc_hi if rng.random() < 0.3 else rng.randint(max(8, doc_hi // 8), doc_hi)
    instr, query = rng.randint(9, 130), rng.randint(17, 70)
    seed = rng.randrange(1 << 20)
    if kind == "rank":
        model = "7b" if rng.random() < 0.3 else "tiny"
        budget = 16000 if model == "7b" else 32000  # tokens of one call
        docs = _log_int(rng, 4, min(100, budget // doc_hi))
        prompts = _log_int(rng, 1, max(1, min(8, budget // (docs * doc_hi + instr + query))))
        case = _rank("", model, prompts, docs, doc_lo, doc_hi, instr, query, seed)
    else:
        dtype = "f32" if kind != "scores" and rng.random() < 0.2 else "bf16"
        heads, kv_heads, head_dim = rng.choice([(32, 8, 128)] * 4 + [(16, 8, 64), (8, 2, 64), (16, 8, 128)])
        budget = 6000 if dtype == "f32" else 20000 if kind == "train" else 66000
        docs = _log_int(rng, 3, min(500, budget // doc_hi))
        prompts = _log_int(rng, 1, max(1, min(8, budget // (docs * doc_hi + instr + query))))
        layout = "grid" if kind == "train" else rng.choice(["grid", "packed"])
        case = _op("", kind, prompts, docs, doc_lo, doc_hi, layout, heads, kv_heads, head_dim, dtype,
                   kind != "scores" and rng.random() < 0.4, instr, query, seed)
    del case["name"]
    return case


def _block_lengths(case):
    """One list [instruction, documents..., query] per prompt."""
    rng = random.Random(case["shape_seed"])
    return [[case["instr"]] + [rng.randint(case["doc_lo"], case["doc_hi"]) for _ in range(case["docs"])] + [case["query"]]
            for _ in range(case["prompts"])]


def _slots(case, lens):
    """(slots per prompt, H of the grid or None)."""
    if case["layout"] == "grid":
        h = -(-max(max(bl) for bl in lens) // 16) * 16
        return len(lens[0]) * h, h
    return -(-max(sum(bl) for bl in lens) // 8) * 8, None


class _Layer:
    """What the attention function reads of the attention module that calls it."""

    def __init__(self, training):
        self.layer_idx, self.training = 0, training


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    lens = _block_lengths(case)
    if case["kind"] == "rank":
        cfg = RankerConfig.mistral_7b() if case["model"] == "7b" else RankerConfig.tiny()
        ranker = MistralPrefillRanker(cfg, "cuda").init_random(seed=seed)
        cpu = torch.Generator().manual_seed(int(seed))
        items = [{"input_ids": torch.randint(3, cfg.vocab_size, (sum(bl),), generator=cpu),
                  "block_lengths": bl[:-1] + [bl[-1] - 4, 4]} for bl in lens]  # the completion is the query block's last 4 tokens
        batch = packed_block_collate_fn(items)
        batch = {k: v.pin_memory() if torch.is_tensor(v) else v for k, v in batch.items()}
        return {"kind": "rank", "ranker": ranker, "batch": batch}

    dev, dt = torch.device("cuda"), DTYPES[case["dtype"]]
    B, N, Nk, D = case["prompts"], case["heads"], case["kv_heads"], case["head_dim"]
    S, H = _slots(case, lens)
    ln = torch.tensor(lens, dtype=torch.int32)
    if H is not None:
        slot = torch.arange(H)
        mask = slot[None, None, :] >= (H - ln)[:, :, None]
        spans = cuda_blockrank_attention_mask(attention_mask=mask.to(dev))
        last = torch.full((B,), S)
    else:
        start = torch.zeros_like(ln)
        start[:, 1:] = ln.cumsum(1)[:, :-1]
        spans = BlockSpans.make(start.to(dev), ln.to(dev), int(ln.max()), max_query_len=int(ln[:, -1].max()))
        last = ln.sum(1)

    def normal(rows, heads):
        """Activations in the model's memory layout (B, rows, heads, D)."""
        return torch.randn(B, rows, heads, D, generator=gen, device=dev, dtype=torch.float32).to(dt)

    state = {"kind": case["kind"], "spans": spans, "scale": D ** -0.5}
    if case["kind"] == "scores":
        # the scoring layer projects the queries of the signal rows only
        state["q"], state["k"] = normal(SIGNAL_ROWS, N).transpose(1, 2), normal(S, Nk).transpose(1, 2)
        state["rows"] = torch.arange(SIGNAL_ROWS, dtype=torch.int32, device=dev).expand(B, SIGNAL_ROWS).contiguous()
        return state
    leaves = [normal(S, h) for h in (N, Nk, Nk)]
    train = case["kind"] == "train"
    state["layer"] = _Layer(train)
    state["wanted"] = {"layers_to_return_scores": [0] if case["raw"] else []}
    if train:
        state["leaves"] = [t.requires_grad_(True) for t in leaves]
        state["grads"] = [normal(S, N)]
        if case["raw"]:
            rows = min(RAW_ROWS, S if H is None else H)
            g = torch.randn(B, N, rows, S, generator=gen, device=dev, dtype=torch.float32)
            state["grads"].append((g * 1e-2).to(dt))
    state["qkv"] = [t.transpose(1, 2) for t in leaves]
    return state


def run(state):
    kind = state["kind"]
    if kind == "rank":
        # The document order is left out of what is compared: with random weights neighbouring documents score
        # closer together than bf16 layers resolve.  The logits it is taken from are all here.
        logits, _ = state["ranker"].rank_host(state["batch"])
        return logits
    spans, scale = state["spans"], state["scale"]
    if kind == "scores":
        return ops.doc_scores(state["q"], state["k"], spans[0], spans[1], state["rows"], scale)
    if kind == "forward":
        with torch.no_grad():
            out, raw = cuda_blockrank_attention_forward(state["layer"], *state["qkv"], spans, scale, **state["wanted"])
        return out if raw is None else (out, raw)
    out, raw = cuda_blockrank_attention_forward(state["layer"], *state["qkv"], spans, scale, **state["wanted"])
    outs = [out] if raw is None else [out, raw]
    return outs + list(torch.autograd.grad(outs, state["leaves"], state["grads"]))


def _pairs(bl):
    """Visible (query, key) pairs of one prompt and one head."""
    tri = lambda x: x * (x + 1) // 2
    before = sum(bl[:-1])
    return tri(bl[0]) + sum(n * bl[0] + tri(n) for n in bl[1:-1]) + bl[-1] * before + tri(bl[-1])


def work(case):
    lens = _block_lengths(case)
    tokens = sum(sum(bl) for bl in lens)
    pairs = sum(_pairs(bl) for bl in lens)
    doc_tokens = sum(sum(bl[1:-1]) for bl in lens)
    B = case["prompts"]
    if case["kind"] == "rank":
        c = RankerConfig.mistral_7b() if case["model"] == "7b" else RankerConfig.tiny()
        N, Nk, D, hid, inter = c.num_attention_heads, c.num_key_value_heads, c.head_dim, c.hidden_size, c.intermediate_size
        layer = hid * (N + 2 * Nk) * D + N * D * hid + 3 * hid * inter
        last = hid * Nk * D
        flops = c.score_layer * (2 * tokens * layer + 4 * D * N * pairs) + 2 * tokens * last
        flops += 2 * B * SIGNAL_ROWS * hid * N * D + 2 * D * N * SIGNAL_ROWS * doc_tokens
        weights = c.score_layer * layer + last + hid * N * D
        return {"bytes": 2 * weights + 2 * tokens * hid + 16 * tokens + 4 * B * case["docs"], "flops": flops}
    N, Nk, D, e = case["heads"], case["kv_heads"], case["head_dim"], 2 if case["dtype"] == "bf16" else 4
    if case["kind"] == "scores":
        nbytes = e * D * (doc_tokens * Nk + B * SIGNAL_ROWS * N) + 4 * B * case["docs"] * (N * SIGNAL_ROWS + 1)
        return {"bytes": nbytes, "flops": 2 * D * N * SIGNAL_ROWS * doc_tokens}
    S, H = _slots(case, lens)
    rows = min(RAW_ROWS, S if H is None else H)
    out_rows = B * S  # padding rows of the output are written too (as zeros)
    nbytes = e * D * (tokens * (N + 2 * Nk) + out_rows * N)
    flops = 4 * D * N * pairs
    raw_bytes, raw_flops = e * B * N * rows * S, 2 * D * N * rows * tokens
    if case["kind"] == "train":
        nbytes += e * D * (tokens * N + out_rows * (N + 2 * Nk))
        flops += 10 * D * N * pairs
        raw_bytes, raw_flops = 2 * raw_bytes, 3 * raw_flops
    if case["raw"]:
        nbytes, flops = nbytes + raw_bytes, flops + raw_flops
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "rank":
        return {"rel": 2e-2}  # bf16 rounding of every activation through all layers (20 on the 7B architecture)
    if case["kind"] == "scores":
        return {"rel": 1e-4}  # bf16 products are exact in the 32-bit sums; exponentials of the sums
    if case["dtype"] == "f32":
        return {"rel": 2e-5}
    return {"rel": 1e-2}
