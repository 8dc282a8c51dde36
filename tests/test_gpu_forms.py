"""Calls of every form that the entry points take -- layouts, options, orders of use -- and the precision that they promise."""
import pytest
import torch

from tests import helpers as H_

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from blockrank_b200 import BlockSpans, _lib, cuda_blockrank_attention_forward, ops

    class Layer:
        layer_idx, training = 0, True


def packed(lens, N, Nk, D, dtype, seed=0):
    """(spans, q, k, v) of packed prompts on the GPU, (B, heads, S, D) views of (B, S, heads, D) tensors."""
    start, ln, S, longest = H_.packed_spans(lens)
    g = torch.Generator().manual_seed(seed)
    spans = BlockSpans.make(start.cuda(), ln.cuda(), longest, max_query_len=int(ln[:, -1].max()))
    return (spans, *(torch.randn(len(lens), S, h, D, generator=g).to(dtype).cuda().transpose(1, 2) for h in (N, Nk, Nk)))


def test_forward_of_a_prompt_does_not_depend_on_its_batch():
    """The query block's context of a long prompt is cut into the same chunks alone and in a batch: the same bits."""
    lens = [[64] + [100] * 100 + [48]] * 4
    spans, q, k, v = packed(lens, 32, 8, 128, torch.bfloat16)
    batch = ops.attention(q, k, v, spans[0], spans[1], 128 ** -0.5, spans.max_block_len, max_query_len=spans.max_query_len)
    alone = ops.attention(q[:1], k[:1], v[:1], spans[0][:1], spans[1][:1], 128 ** -0.5, spans.max_block_len,
                          max_query_len=spans.max_query_len)
    assert torch.equal(batch[:1], alone)
