"""Early-exit Mistral-architecture prefill ranker: what scripts/eval_attn.py does, minus the waste.

The reference scores documents by running the HF model with every layer after
the scoring layer ``l*`` patched to identity (scripts/eval_attn.py:121-130) and
reducing that layer's raw attention logits (src/blockrank/losses.py:37-78).
Layer ``l*`` itself still runs completely there.  This runner computes the same
scores with the minimal work: layers 0..l*-1 in full, and at layer ``l*`` only
the input RMSNorm, ``k_proj`` for every token, ``q_proj`` for the signal rows,
RoPE and the fused score epilogue.

Dense projections are cuBLAS GEMMs on PyTorch's handle; RMSNorm, RoPE,
SiLU*up, the block-sparse attention and the scorer are this package's CUDA
kernels.  Weights use the HF parameter names, so a real checkpoint's state
dict loads directly.
"""
from __future__ import annotations

from dataclasses import dataclass
from typing import Dict, Optional

import torch

from . import ops, _lib


@dataclass
class RankerConfig:
    vocab_size: int = 32768
    hidden_size: int = 4096
    intermediate_size: int = 14336
    num_hidden_layers: int = 32
    num_attention_heads: int = 32
    num_key_value_heads: int = 8
    head_dim: int = 128
    rope_theta: float = 1e6
    rms_norm_eps: float = 1e-5
    score_layer: int = 20
    temperature: float = 0.05

    @staticmethod
    def mistral_7b(score_layer: int = 20) -> "RankerConfig":
        return RankerConfig(score_layer=score_layer)

    @staticmethod
    def tiny(score_layer: int = 2) -> "RankerConfig":
        return RankerConfig(vocab_size=32768, hidden_size=256, intermediate_size=688, num_hidden_layers=4,
                            num_attention_heads=4, num_key_value_heads=2, head_dim=64, score_layer=score_layer)


_STEPS = ("decoder_layer", "hidden_before_score_layer", "score", "score_from_hidden")  # methods that rank_host stands on
_LAYER_WEIGHTS = ("ln1", "wqkv", "wo", "ln2", "wgu", "wd")  # of a full layer


@dataclass
class _CapturedScore:
    graph: "torch.cuda.CUDAGraph"
    static: list   # input buffers the graph reads
    out: tuple     # (logits, doc_mass) the graph writes


class MistralPrefillRanker:
    """Holds the fused weights of layers 0..score_layer on one GPU and ranks prompts."""

    def __init__(self, cfg: RankerConfig, device, dtype=torch.bfloat16):
        if cfg.score_layer >= cfg.num_hidden_layers:
            raise ValueError("score_layer must index an existing layer")
        _lib.lib()  # no CUDA library, no runner
        self.cfg, self.device, self.dtype = cfg, torch.device(device), dtype
        self.embed: Optional[torch.Tensor] = None
        self.layers = []  # dicts: ln1, wqkv, wo, ln2, wgu, wd   (scoring layer: ln1, wq, wk)
        inv = 1.0 / (cfg.rope_theta ** (torch.arange(0, cfg.head_dim, 2, dtype=torch.int64).float() / cfg.head_dim))
        self.inv_freq = inv.to(self.device)
        self.algo = _lib.ALGO_AUTO
        self.events = None  # set to {"attn": [], "score": []} to collect (start, end) CUDA events per launch
        self.use_graphs = False  # rank_host replays one captured CUDA graph per batch geometry instead of launching eagerly
        self._graphs: Dict[tuple, "_CapturedScore"] = {}

    # ---- weights ---------------------------------------------------------------
    def load_state_dict(self, sd: Dict[str, torch.Tensor]) -> "MistralPrefillRanker":
        """Take HF-named tensors (model.embed_tokens.weight, model.layers.{i}.self_attn.q_proj.weight, ...)."""
        c, dev, dt = self.cfg, self.device, self.dtype
        g = lambda name: sd[name].detach().to(device=dev, dtype=dt)
        self.embed = g("model.embed_tokens.weight")
        self.layers = []
        for i in range(c.score_layer + 1):
            p = f"model.layers.{i}."
            L = {"ln1": g(p + "input_layernorm.weight")}
            if i < c.score_layer:
                L["wqkv"] = torch.cat([g(p + "self_attn.q_proj.weight"), g(p + "self_attn.k_proj.weight"),
                                       g(p + "self_attn.v_proj.weight")], 0).contiguous()
                L["wo"] = g(p + "self_attn.o_proj.weight")
                L["ln2"] = g(p + "post_attention_layernorm.weight")
                L["wgu"] = torch.cat([g(p + "mlp.gate_proj.weight"), g(p + "mlp.up_proj.weight")], 0).contiguous()
                L["wd"] = g(p + "mlp.down_proj.weight")
            else:
                L["wq"] = g(p + "self_attn.q_proj.weight")
                L["wk"] = g(p + "self_attn.k_proj.weight")
            self.layers.append(L)
        return self

    def init_random(self, seed: int = 3, std: float = 0.02) -> "MistralPrefillRanker":
        """Random weights N(0, std) drawn on the device (norm weights 1); only layers 0..score_layer exist."""
        c, dev, dt = self.cfg, self.device, self.dtype
        gen = torch.Generator(device=dev).manual_seed(seed)
        rnd = lambda *shape: (torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32) * std).to(dt)
        ones = lambda n: torch.ones(n, device=dev, dtype=dt)
        qd, kd = c.num_attention_heads * c.head_dim, c.num_key_value_heads * c.head_dim
        self.embed = rnd(c.vocab_size, c.hidden_size)
        self.layers = []
        for i in range(c.score_layer + 1):
            L = {"ln1": ones(c.hidden_size)}
            if i < c.score_layer:
                L["wqkv"] = rnd(qd + 2 * kd, c.hidden_size)
                L["wo"] = rnd(c.hidden_size, qd)
                L["ln2"] = ones(c.hidden_size)
                L["wgu"] = rnd(2 * c.intermediate_size, c.hidden_size)
                L["wd"] = rnd(c.hidden_size, c.intermediate_size)
            else:
                L["wq"] = rnd(qd, c.hidden_size)
                L["wk"] = rnd(kd, c.hidden_size)
            self.layers.append(L)
        return self

    # ---- forward ---------------------------------------------------------------
    @torch.no_grad()
    def decoder_layer(self, i, h, pos, B, S, blk_start, blk_len, max_block_len, max_query_len=0):
        """One full decoder layer ``i < score_layer`` applied in place to the residual stream ``h`` (B*S, hidden).

        Both residual additions happen in the epilogue of the GEMM that produces the branch
        (C = C + A·B, added in fp32 before the rounding), so the branch output is never
        written to memory and the RMSNorm that follows reads one tensor instead of two."""
        c, L, host = self.cfg, self.layers[i], _lib.host()
        N, Nk, D = c.num_attention_heads, c.num_key_value_heads, c.head_dim
        qkv = host.layer_qkv(h, L["ln1"], L["wqkv"], pos, self.inv_freq, N, Nk, D, c.rms_norm_eps)
        ev = self._tick("attn")
        attn = host.layer_attention(qkv, blk_start, blk_len, B, S, N, Nk, D, max_block_len, max_query_len, self.algo)
        self._tock(ev)
        host.layer_rest(h, attn, L["wo"], L["ln2"], L["wgu"], L["wd"], c.rms_norm_eps)
        return h

    @torch.no_grad()
    def hidden_before_score_layer(self, input_ids, position_ids, blk_start, blk_len, max_block_len, max_query_len=0):
        """Run layers 0..l*-1; returns the residual stream entering layer l*, shape (B*S, hidden)."""
        B, S = input_ids.shape
        c = self.cfg
        pos = position_ids.reshape(B * S).to(torch.int32)
        if self.events is None and not self._overridden("decoder_layer"):  # the layers in one native call
            return _lib.host().hidden_states(
                self.embed, input_ids, self._full_layers(), pos, self.inv_freq,
                blk_start, blk_len, max_block_len, max_query_len, c.num_attention_heads, c.num_key_value_heads, c.head_dim,
                c.rms_norm_eps, self.algo)
        h = torch.embedding(self.embed, input_ids.reshape(B * S))
        for i in range(c.score_layer):
            self.decoder_layer(i, h, pos, B, S, blk_start, blk_len, max_block_len, max_query_len)
        return h

    @torch.no_grad()
    def score(self, input_ids, position_ids, blk_start, blk_len, max_block_len, signal_rows, max_query_len=0):
        """input_ids/position_ids (B, S) on the device, spans int32 (B, M), signal_rows int32 (B, R), or (1, R) for
        the same rows of every prompt;
        ``max_query_len`` (optional) bounds the query block's length (smaller attention scratch).

        Returns (logits (B, num_docs) fp32, doc_mass (B, N, R, num_docs) fp32).  Device-side problems
        (malformed spans, a kernel wait that gave up) are raised by ``ops.check_status()``, which
        :meth:`rank_host` calls after copying the scores back.
        """
        h = self.hidden_before_score_layer(input_ids, position_ids, blk_start, blk_len, max_block_len, max_query_len)
        return self.score_from_hidden(h, position_ids, blk_start, blk_len, signal_rows)

    @torch.no_grad()
    def score_from_hidden(self, h, position_ids, blk_start, blk_len, signal_rows):
        """The scoring layer's share of the work, from the residual stream ``h`` (B*S, hidden) entering it:
        input RMSNorm, ``k_proj`` of every token, ``q_proj`` of the signal rows, RoPE, fused score epilogue."""
        c = self.cfg
        L = self.layers[c.score_layer]
        pos = position_ids.to(torch.int32).contiguous()
        q, k, rows = _lib.host().score_qk(h, pos, signal_rows.to(torch.int32), L["ln1"], L["wq"], L["wk"], self.inv_freq,
                                          c.num_attention_heads, c.num_key_value_heads, c.head_dim, c.rms_norm_eps)
        ev = self._tick("score")
        mass, logits = ops.doc_scores(q, k, blk_start, blk_len, rows, c.head_dim ** -0.5, c.temperature)
        self._tock(ev)
        return logits, mass

    # ---- CUDA graphs -----------------------------------------------------------
    @torch.no_grad()
    def score_graphed(self, input_ids, position_ids, blk_start, blk_len, max_block_len, signal_rows, max_query_len=0):
        """Same contract as :meth:`score`, but the whole launch sequence (about 440 kernels for the 7B
        architecture) is captured once per batch geometry ``(B, S, M, R, max_block_len)`` and replayed.

        Inputs are copied into the graph's static buffers; the returned tensors are the graph's static
        outputs and are overwritten by the next call with the same geometry.  The first call for a
        geometry runs eagerly twice (library initialisation, allocator warm-up) before capturing.
        """
        key = (tuple(input_ids.shape), tuple(blk_start.shape), tuple(signal_rows.shape), int(max_block_len),
               int(max_query_len))
        cap = self._graphs.get(key)
        if cap is None:
            if self.events is not None:
                raise RuntimeError("per-launch events cannot be collected while capturing a CUDA graph")
            static = [t.clone() for t in (input_ids, position_ids, blk_start, blk_len, signal_rows)]
            side = torch.cuda.Stream(device=self.device)
            side.wait_stream(torch.cuda.current_stream(self.device))
            with torch.cuda.stream(side):
                for _ in range(2):
                    self.score(static[0], static[1], static[2], static[3], int(max_block_len), static[4], int(max_query_len))
            torch.cuda.current_stream(self.device).wait_stream(side)
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                out = self.score(static[0], static[1], static[2], static[3], int(max_block_len), static[4], int(max_query_len))
            cap = self._graphs[key] = _CapturedScore(graph, static, out)
        for dst, src in zip(cap.static, (input_ids, position_ids, blk_start, blk_len, signal_rows)):
            dst.copy_(src, non_blocking=True)
        cap.graph.replay()
        return cap.out

    def _tick(self, kind):
        if self.events is None:
            return None
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        self.events[kind].append((a, b))
        a.record()
        return b

    @staticmethod
    def _tock(ev):
        if ev is not None:
            ev.record()

    @torch.no_grad()
    def rank_host(self, batch: dict, k: int = 10):
        """End-to-end call on HOST tensors: ``batch`` holds pinned ``input_ids``/``position_ids`` (B, S) int64,
        ``block_spans`` int32 (2, B, M), ``signal_rows`` int32 (B, R) and ``max_block_len``.  Copies them to the
        device, scores, and returns (logits, top-k document indices) on the host."""
        c, host = self.cfg, _lib.host()
        if not self.use_graphs and self.events is None and not self._overridden(*_STEPS):
            last = self.layers[c.score_layer]
            return host.rank(self.embed, self._full_layers(), [last["ln1"], last["wq"], last["wk"]], self.inv_freq,
                             batch["input_ids"], batch["position_ids"], batch["block_spans"], batch["signal_rows"],
                             int(batch["max_block_len"]), c.num_attention_heads, c.num_key_value_heads, c.head_dim,
                             c.rms_norm_eps, self.algo, c.temperature, k)
        ids, pos, start, length, rows, max_query_len = host.upload(
            batch["input_ids"], batch["position_ids"], batch["block_spans"], batch["signal_rows"], self.embed.device)
        run = self.score_graphed if self.use_graphs else self.score
        logits, _ = run(ids, pos, start, length, int(batch["max_block_len"]), rows, max_query_len)
        # (raises if a kernel reported malformed spans or a wait that gave up)
        return host.download(logits, k)

    def _overridden(self, *steps) -> bool:
        """Has a subclass, or somebody on this object, put another method in the place of one of ``steps``?"""
        return any(s in self.__dict__ or getattr(type(self), s) is not getattr(MistralPrefillRanker, s) for s in steps)

    def _full_layers(self):
        return [[L[n] for n in _LAYER_WEIGHTS] for L in self.layers[:self.cfg.score_layer]]

    def weight_bytes(self) -> int:
        n = self.embed.numel() * self.embed.element_size()
        for L in self.layers:
            n += sum(t.numel() * t.element_size() for t in L.values())
        return n
