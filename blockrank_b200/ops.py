"""Torch-facing functions over the C ABI: tensors in, tensors out, current stream.

PyTorch is used for device memory, streams and the dense projections only; all
BlockRank-specific compute happens in libblockrank_b200.so.  The work of each
call (checks, allocation, parameter structs) is done by csrc/torch_host.cpp.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import _lib


def __getattr__(name: str):
    if name == "launch_count":  # kernels of the library enqueued in this process so far
        return _lib.host().launch_count()
    raise AttributeError(f"module {__name__!r} has no attribute {name!r}")


def _view(t: torch.Tensor) -> _lib.View:
    """(B, heads, S, D) tensor (any strides, innermost contiguous) -> brk_view, for callers of the ctypes ABI."""
    if t.dim() != 4 or t.stride(-1) != 1:
        raise ValueError("expected a (B, heads, S, D) tensor with contiguous head_dim")
    return _lib.View(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


def spans_from_mask(mask_bmh: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """(B, M, H) bool left-padded block mask (collator output) -> int32 (B, M) start, length."""
    return _lib.host().spans_from_mask(mask_bmh)


def status_word(device) -> torch.Tensor:
    """The device's int32 status word, zeroed when created.  Every attention call passes it; the kernels set
    it (the first code written stays) when a bounded wait gives up or the block spans are malformed, and check_status()
    turns it into an exception at the caller's next synchronisation point."""
    device = torch.device(device)
    return _lib.host().status_word(device.index if device.index is not None else torch.cuda.current_device())


def check_status(device=None) -> None:
    """Synchronise the current stream of ``device`` and raise if a kernel reported a problem since the last
    check: BlockRankLibraryError (BRK_E_TIMEOUT) after a device-side wait gave up, ValueError (BRK_E_ARG)
    after malformed block spans.  The word is cleared, so the next call starts clean."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    w = status_word(device)
    with torch.cuda.device(w.device):
        _lib.check(_lib.lib().brk_status_poll(w.data_ptr(), torch.cuda.current_stream(w.device).cuda_stream),
                   "brk_status_poll")


def attention(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, blk_start: torch.Tensor, blk_len: torch.Tensor,
              scale: float, max_block_len: int, out: Optional[torch.Tensor] = None, return_lse: bool = False,
              algo: int = _lib.ALGO_AUTO, max_query_len: int = 0, lse: Optional[torch.Tensor] = None):
    """BlockRank attention forward.

    q (B,N,S,D), k/v (B,Nk,S,D) views of any stride (head_dim contiguous);
    blk_start/blk_len int32 (B,M) on the device.  Returns out (B,S,N,D)
    [and lse (B,N,S)].  Padding slots of ``out`` are zero.  ``max_query_len``
    (optional) bounds the last block's length and shrinks the scratch of the
    tensor-core path.  Device-side problems (malformed spans, a wait that gave
    up) surface at the next :func:`check_status`.
    """
    res = _lib.host().attention(q, k, v, blk_start, blk_len, scale, int(max_block_len), out, return_lse, algo,
                                int(max_query_len), lse)
    return res if (return_lse or lse is not None) else res[0]


def attention_bwd(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, d_out: torch.Tensor,
                  lse: torch.Tensor, blk_start: torch.Tensor, blk_len: torch.Tensor, scale: float, max_block_len: int):
    """Gradients of :func:`attention` (what autograd derives from the reference's eager / SDPA paths,
    src/blockrank/blockrank_std_attention.py:96-262, 472-650).

    q (B,N,S,D), k/v (B,Nk,S,D) as given to the forward; out / d_out (B,S,N,D); lse (B,N,S) fp32 from the
    forward.  Returns (dq (B,N,S,D), dk, dv (B,Nk,S,D)) in the input dtype; slots outside every block get zeros.
    """
    return _lib.host().attention_bwd(q, k, v, out, d_out, lse, blk_start, blk_len, scale, int(max_block_len))


def doc_scores(q: torch.Tensor, k: torch.Tensor, blk_start: torch.Tensor, blk_len: torch.Tensor, rows: torch.Tensor,
               scale: float, temperature: float = 0.05):
    """Fused score epilogue.

    rows: int32 (B, R) slot indices of the signal rows.  Returns
    (doc_mass (B,N,R,num_docs) fp32, logits (B,num_docs) fp32) where logits is
    the mean over heads and rows divided by ``temperature`` -- what the
    reference's compute_auxiliary_attention_loss(return_logits=True) yields.
    """
    return _lib.host().doc_scores(q, k, blk_start, blk_len, rows, scale, temperature)


def raw_scores(q: torch.Tensor, k: torch.Tensor, blk_start: torch.Tensor, blk_len: torch.Tensor, scale: float,
               num_last: int = 16, grid_h: Optional[int] = None) -> torch.Tensor:
    """Reference-compatible second return value: (B, N, R, S) masked logits of the last R slots.

    R = min(num_last, grid_h): on the reference's (M, H) grid the window never reaches past the last
    block's H slots (src/blockrank/blockrank_std_attention.py:256-262); without a grid (padding-free
    layout) R = min(num_last, S)."""
    return _lib.host().raw_scores(q, k, blk_start, blk_len, scale, int(num_last), -1 if grid_h is None else int(grid_h))


def raw_scores_bwd(q: torch.Tensor, k: torch.Tensor, d_raw: torch.Tensor, blk_start: torch.Tensor, blk_len: torch.Tensor,
                   scale: float, dq: Optional[torch.Tensor] = None, dk: Optional[torch.Tensor] = None):
    """Gradient of :func:`raw_scores`: d_raw (B,N,R,S) -> (dq (B,N,S,D), dk (B,Nk,S,D)).

    With dq and dk given (both, e.g. what :func:`attention_bwd` returned) it is added to them in place; otherwise new
    tensors are returned, dq zero outside the last R rows."""
    return _lib.host().raw_scores_bwd(q, k, d_raw, blk_start, blk_len, scale, dq, dk)


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float, residual: Optional[torch.Tensor] = None,
            out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """RMSNorm over the last dim.  With ``residual`` given: residual += x (in place), norm of the sum."""
    return _lib.host().rmsnorm(x, weight, eps, residual, out)


def rope_(q: Optional[torch.Tensor], k: Optional[torch.Tensor], pos: torch.Tensor, inv_freq: torch.Tensor) -> None:
    """In-place rotate-half RoPE.  q (T, N, D) and/or k (T, Nk, D) may be strided views with
    contiguous (heads, D); either may be None; pos int32 (T,), inv_freq fp32 (D/2,)."""
    _lib.host().rope_(q, k, pos, inv_freq)


def silu_mul(gate_up: torch.Tensor, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """(rows, 2*I) [gate | up] -> (rows, I) silu(gate) * up."""
    return _lib.host().silu_mul(gate_up, out)
