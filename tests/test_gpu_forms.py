"""Calls of every form that the entry points take -- layouts, options, orders of use -- and the precision that they promise."""
import pytest
import torch

from oracle import blockrank_oracle as orc
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


@pytest.mark.parametrize("q_scale", [1, 32], ids=["", "rescaled"])  # 32: the running maximum jumps, also inside a 128-key tile
@pytest.mark.parametrize("N,Nk,D,M,H", [
    (16, 8, 64, 7, 160), (8, 1, 64, 5, 96), (4, 4, 64, 3, 130), (8, 2, 64, 1, 200),   # every group size, one block
    (4, 2, 64, 30, 96), (4, 2, 64, 3, 700),          # key chunks of the query block; blocks too long to stay resident
    (16, 8, 128, 7, 160), (8, 1, 128, 12, 64), (2, 2, 128, 2, 300)])
def test_default_bf16_forward_rounds_the_output_only(N, Nk, D, M, H, q_scale):
    """Off head_dim 128 with four heads per KV head, probabilities are not rounded to bf16: the error against 64 bits is that
    of the rounded output (1 % for the sums in 32 bits; with P in bf16 it is 28 % more)."""
    lens = H_.random_lens(2, M, H, 7 * M + D)
    mask = H_.ragged_mask(2, M, H, lens)
    q, k, v = H_.qkv(2, N, Nk, M * H, D, M, torch.bfloat16)
    q = (q.float() * q_scale).bfloat16()
    ref, _ = orc.attention_dense(q, k, v, mask, D ** -0.5)
    start, ln = ops.spans_from_mask(mask.cuda())
    out = ops.attention(*(H_.to_cuda_view(x) for x in (q, k, v)), start, ln, D ** -0.5, H)
    rows = mask.reshape(2, -1)
    ref = ref[rows]
    assert (out.cpu()[rows].double() - ref).norm() <= 1.01 * (ref.bfloat16().double() - ref).norm()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N,Nk,R", [(8, 2, 16), (5, 1, 13), (8, 1, 16), (16, 4, 64), (4, 1, 64)])  # 64, 65, 128, 256 pairs
def test_raw_score_gradient_rounds_dk_once(N, Nk, R, D):
    """dk of more (head, row) pairs than a pass holds is summed in fp32 over the passes: its error against 64 bits is that of
    one rounding to bf16 (1.66e-3; 2.4e-3 and 3.1e-3 with a rounding after each of two and four passes)."""
    g = torch.Generator().manual_seed(N + R)
    B, S, scale = 2, 5 * 130, D ** -0.5
    rb = lambda *s: torch.randn(*s, generator=g).bfloat16()
    q, k, d_raw = rb(B, N, S, D), rb(B, Nk, S, D), rb(B, N, R, S)
    start, ln = ops.spans_from_mask(torch.ones(B, 5, 130, dtype=torch.bool).cuda())
    _, dk = ops.raw_scores_bwd(q.cuda(), k.cuda(), d_raw.cuda(), start, ln, scale)
    rk = ((d_raw.double() * scale).transpose(-1, -2) @ q[:, :, S - R:].double()).view(B, Nk, N // Nk, S, D).sum(2)
    assert (dk.cpu().double() - rk).norm() <= 1.01 * (rk.bfloat16().double() - rk).norm()


@pytest.mark.parametrize("shift", [1, 4, 8])
def test_raw_scores_into_a_buffer_of_any_alignment(shift):
    """The C entry takes any `out` that is aligned for its elements, also where a row is whole 16-byte pieces."""
    import ctypes as C
    spans, q, k, _ = packed([[9, 30, 41, 24]], 4, 2, 128, torch.bfloat16, seed=3)
    B, N, S, D, R = 1, 4, q.shape[2], 128, 16
    assert S % 8 == 0
    ref = ops.raw_scores(q, k, spans[0], spans[1], D ** -0.5, R)
    start, ln = spans[0].contiguous(), spans[1].contiguous()
    p = _lib.ScoreParams()
    p.dtype, p.B, p.N, p.Nk, p.D, p.S, p.M, p.R, p.scale, p.temperature = _lib.BRK_BF16, B, N, 2, D, S, 4, R, D ** -0.5, 1.0
    p.q, p.k, p.blk_start, p.blk_len = ops._view(q), ops._view(k), start.data_ptr(), ln.data_ptr()
    buf = torch.full((ref.numel() + 16,), 7.0, dtype=torch.bfloat16, device="cuda")
    rc = _lib.lib().brk_raw_scores(C.byref(p), buf.data_ptr() + 2 * shift, torch.cuda.current_stream().cuda_stream)
    assert rc == 0, _lib.lib().brk_last_error()
    assert torch.equal(buf[shift:shift + ref.numel()], ref.flatten())
    assert (buf[:shift] == 7).all() and (buf[shift + ref.numel():] == 7).all()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs a device that is not the current one")
def test_ranker_layers_run_on_their_own_device():
    """decoder_layer, and the whole forward when launches are timed, on a device that is not the current one."""
    from blockrank_b200 import packed_block_collate_fn
    from blockrank_b200.runner import MistralPrefillRanker, RankerConfig
    cfg = RankerConfig.tiny()
    bl = [30, 40, 50, 20, 4]
    items = [{"input_ids": torch.arange(3, 3 + sum(bl)), "block_lengths": bl}]
    batch = packed_block_collate_fn(items)
    ref = MistralPrefillRanker(cfg, "cuda:0").init_random(seed=1).rank_host(batch)[0]
    other = MistralPrefillRanker(cfg, "cuda:1").init_random(seed=1)
    other.events = {"attn": [], "score": []}
    with torch.cuda.device(0):
        assert torch.equal(other.rank_host(batch)[0], ref)


@pytest.mark.parametrize("switch", ["none", "bf16_reduction", "cublaslt", "deterministic"])
def test_ranker_products_follow_pytorchs_switches(switch, monkeypatch):
    """The products of a layer are torch.addmm's, bit for bit, whatever PyTorch's switches say."""
    monkeypatch.setenv("CUBLAS_WORKSPACE_CONFIG", ":4096:8")
    matmul, blas = torch.backends.cuda.matmul, torch.backends.cuda.preferred_blas_library()
    monkeypatch.setattr(matmul, "allow_bf16_reduced_precision_reduction", switch != "bf16_reduction")
    if switch == "cublaslt":
        torch.backends.cuda.preferred_blas_library("cublaslt")
    torch.use_deterministic_algorithms(switch == "deterministic")
    try:
        gen = torch.Generator(device="cuda").manual_seed(2)
        for dtype in (torch.bfloat16, torch.float32):
            for T, K, n in [(16, 14336, 4096), (64, 4096, 1024), (2, 4096, 4096), (40, 8192, 256)]:
                x = torch.randn(T, K, generator=gen, device="cuda").to(dtype)
                w = (torch.randn(n, K, generator=gen, device="cuda") / K ** 0.5).to(dtype)
                h = torch.randn(T, n, generator=gen, device="cuda").to(dtype)
                ref = h.clone().addmm_(x, w.t())
                zero = lambda *s: torch.zeros(*s, dtype=dtype, device="cuda")
                _lib.host().layer_rest(h, x, w, zero(n), zero(16, n), zero(n, 8), 1e-5)  # (an MLP that adds nothing)
                assert torch.equal(h, ref), (dtype, T, K, n)
    finally:
        torch.use_deterministic_algorithms(False)
        torch.backends.cuda.preferred_blas_library(blas)


def _requests(n, lens, dtype=torch.bfloat16):
    """(ranker, batch) of n prompts of the same block lengths on the tiny model."""
    from blockrank_b200 import packed_block_collate_fn
    from blockrank_b200.runner import MistralPrefillRanker, RankerConfig
    cfg = RankerConfig.tiny()
    g = torch.Generator().manual_seed(n)
    items = [{"input_ids": torch.randint(3, cfg.vocab_size, (sum(lens),), generator=g), "block_lengths": lens} for _ in range(n)]
    return MistralPrefillRanker(cfg, "cuda", dtype).init_random(seed=1), packed_block_collate_fn(items)


def test_one_set_of_signal_rows_serves_every_prompt():
    """signal_rows of shape (1, R) are the rows of every prompt: host request, device call, captured graph."""
    rk, batch = _requests(3, [30, 40, 50, 60, 20, 4])
    full = rk.rank_host(batch)[0]
    one = dict(batch, signal_rows=batch["signal_rows"][:1])
    assert torch.equal(rk.rank_host(one)[0], full)
    spans = batch["block_spans"].cuda()
    args = (batch["input_ids"].cuda(), batch["position_ids"].cuda(), spans[0], spans[1], int(batch["max_block_len"]))
    assert torch.equal(rk.score(*args, one["signal_rows"].cuda())[0].cpu(), full)
    rk.use_graphs = True
    assert torch.equal(rk.rank_host(one)[0], full)


def test_request_shapes_that_do_not_belong_together_are_refused():
    rk, batch = _requests(3, [30, 40, 50, 20, 4])
    for bad in (dict(batch, signal_rows=batch["signal_rows"][:2]), dict(batch, position_ids=batch["position_ids"].flatten()),
                dict(batch, position_ids=batch["position_ids"][:, :-1].contiguous())):
        with pytest.raises((ValueError, RuntimeError)):
            rk.rank_host(bad)


def test_error_messages_carry_their_numbers():
    spans, q, k, v = packed([[9, 30, 41, 24]], 4, 2, 64, torch.bfloat16)
    with pytest.raises(ValueError, match=r"shape mismatch q\[1, 4, 104, 64\]"):
        ops.attention(q, k[:, :, :-8], v, spans[0], spans[1], 0.125, spans.max_block_len)


def test_spans_of_one_prompt_and_parts_of_spans():
    """(2, M) spans serve one prompt; a slice of spans is refused, not read as a block mask; too few spans are refused."""
    spans, q, k, v = packed([[9, 30, 41, 24]] * 2, 4, 2, 64, torch.bfloat16)
    run = lambda n, sp: cuda_blockrank_attention_forward(Layer(), q[:n], k[:n], v[:n], sp, 0.125)[0]
    full = run(2, spans)
    assert torch.equal(run(1, BlockSpans.make(spans[0][0], spans[1][0], spans.max_block_len)), full[:1])
    with pytest.raises(AttributeError):
        run(1, spans[:, :1])
    for call in (lambda: run(2, BlockSpans.make(spans[0][0], spans[1][0], spans.max_block_len)),
                 lambda: ops.raw_scores(q, k, spans[0][:1], spans[1][:1], 0.125),
                 lambda: ops.doc_scores(q, k, spans[0][:1], spans[1][:1], torch.zeros(2, 2, dtype=torch.int32, device="cuda"), 0.125)):
        with pytest.raises(ValueError, match="too few"):
            call()


def _train(dtype, lens=((20, 30, 40, 24),) * 2, N=4, Nk=2, D=64):
    """(leaves, call): call() is a forward with raw logits under autograd on fresh graph nodes."""
    spans, q, k, v = packed([list(x) for x in lens], N, Nk, D, dtype, seed=5)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    return leaves, lambda: cuda_blockrank_attention_forward(Layer(), *leaves, spans, D ** -0.5, layers_to_return_scores=[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_outputs_can_be_differentiated_in_passes_of_their_own(dtype):
    """The attention output and the raw logits, in one pass, in two passes of either order, and no output twice."""
    leaves, call = _train(dtype)
    out, raw = call()
    g = torch.Generator(device="cuda").manual_seed(1)
    go, gr = (torch.randn(t.shape, generator=g, device="cuda").to(dtype) for t in (out, raw))
    both = torch.autograd.grad([out, raw], leaves, [go, gr], retain_graph=True)
    a = torch.autograd.grad(out, leaves, go)
    r = torch.autograd.grad(raw, leaves, gr, allow_unused=True)
    assert r[2] is None
    tol = 1e-2 if dtype == torch.bfloat16 else 1e-5
    for x, y, z in zip(both[:2], a, r):
        assert (x.double() - (y.double() + z.double())).norm() <= tol * x.double().norm()
    out, raw = call()  # the other order
    r2 = torch.autograd.grad(raw, leaves[:2], gr)
    a2 = torch.autograd.grad(out, leaves, go)
    for x, y in zip((*a, *r[:2]), (*a2, *r2)):
        assert (x.double() - y.double()).norm() <= 1e-4 * x.double().norm()  # (sums of the prefix in another order)
    for t, gt in ((out, go), (raw, gr)):
        with pytest.raises(RuntimeError, match="second time"):
            torch.autograd.grad(t, leaves[:2], gt)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_raw_logits_can_be_differentiated_twice(dtype):
    """A penalty on the gradient of the raw logits: its gradient against 64 bits."""
    leaves, call = _train(dtype)
    _, raw = call()
    g = torch.randn(raw.shape, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(dtype) * 0.1
    dq, dk = torch.autograd.grad(raw, leaves[:2], g, create_graph=True)
    got = torch.autograd.grad(dq.float().square().sum() + dk.float().square().sum(), leaves[:2])
    q, k = (t.detach().double().requires_grad_(True) for t in leaves[:2])
    R, S = raw.shape[2:]
    ref = (q[:, :, S - R:] * 0.125) @ k.repeat_interleave(2, 1).transpose(-1, -2)
    rq, rk = torch.autograd.grad(ref, (q, k), g.double(), create_graph=True)
    want = torch.autograd.grad(rq.square().sum() + rk.square().sum(), (q, k))
    for x, y in zip(got, want):
        assert (x.double() - y).norm() <= (1e-2 if dtype == torch.bfloat16 else 1e-5) * y.norm()


def test_autograd_forms_that_are_refused_or_hooked():
    leaves, call = _train(torch.bfloat16)
    kept = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(t) or t.cpu(), lambda t: t.cuda()):
        out, raw = call()
    assert len(kept) == 7
    hooked = torch.autograd.grad([out, raw], leaves, [torch.ones_like(out), torch.ones_like(raw)])
    out, raw = call()
    plain = torch.autograd.grad([out, raw], leaves, [torch.ones_like(out), torch.ones_like(raw)])
    for x, y in zip(hooked, plain):
        assert (x.double() - y.double()).norm() <= 1e-4 * y.double().norm()
    spans, q, k, v = packed([[20, 30, 40, 24]], 4, 2, 64, torch.bfloat16)
    y = q.clone().requires_grad_(True) * 1
    out, _ = cuda_blockrank_attention_forward(Layer(), y, k, v, spans, 0.125)
    with torch.no_grad():
        y.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.float().sum().backward()
    import torch.autograd.forward_ad as fa
    with fa.dual_level(), pytest.raises(NotImplementedError):
        dual = fa.make_dual(q.clone().requires_grad_(True), torch.ones_like(q))
        cuda_blockrank_attention_forward(Layer(), dual, k, v, spans, 0.125)
    for transform in (lambda f: torch.func.grad(lambda x: f(x).float().sum())(q), lambda f: torch.vmap(f)(torch.stack([q, q]))):
        with pytest.raises(RuntimeError):
            transform(lambda x: cuda_blockrank_attention_forward(Layer(), x, k, v, spans, 0.125)[0])


def test_other_threads_run_while_calls_are_enqueued():
    """A call that blocks on the full queue of a busy device does not hold Python's lock."""
    import threading
    import time
    spans, q, k, v = packed([[64] + [100] * 10 + [48]], 32, 8, 128, torch.bfloat16)
    call = lambda: cuda_blockrank_attention_forward(Layer(), q, k, v, spans, 0.1)
    call()
    torch.cuda.synchronize()
    gap, stop = [0.0], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gap[0], last = max(gap[0], now - last), now

    thread = threading.Thread(target=tick)
    thread.start()
    torch.cuda._sleep(1_500_000_000)  # about 0.8 s of an idle kernel; the queue holds about a thousand launches
    for _ in range(1200):
        call()
    torch.cuda.synchronize()
    stop.set()
    thread.join()
    assert gap[0] < 0.3


def test_calls_of_several_threads_on_streams_of_their_own():
    import threading
    spans, q, k, v = packed([[30, 90, 70, 50, 24]] * 2, 8, 2, 128, torch.bfloat16)
    ref, raw = cuda_blockrank_attention_forward(Layer(), q, k, v, spans, 0.1, layers_to_return_scores=[0])
    torch.cuda.synchronize()
    bad = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                o, r = cuda_blockrank_attention_forward(Layer(), q, k, v, spans, 0.1, layers_to_return_scores=[0])
                bad.append(not (torch.equal(o, ref) and torch.equal(r, raw)))

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(bad) == 200 and not any(bad)


def test_sizes_may_be_any_number():
    spans, q, k, v = packed([[9, 30, 41, 24]], 4, 2, 64, torch.bfloat16)
    ref = ops.attention(q, k, v, spans[0], spans[1], 0.125, spans.max_block_len)
    for size in (float(spans.max_block_len), torch.tensor(spans.max_block_len)):
        assert torch.equal(ops.attention(q, k, v, spans[0], spans[1], torch.tensor(0.125), size), ref)


def test_overridden_steps_of_the_ranker_are_used():
    from blockrank_b200.runner import MistralPrefillRanker
    rk, batch = _requests(2, [30, 40, 50, 20, 4])
    full = rk.rank_host(batch)[0]

    class Halved(MistralPrefillRanker):
        def decoder_layer(self, i, h, *args, **kwargs):
            self.seen = getattr(self, "seen", 0) + 1
            return super().decoder_layer(i, h, *args, **kwargs)

    sub = Halved(rk.cfg, "cuda").init_random(seed=1)
    assert torch.equal(sub.rank_host(batch)[0], full) and sub.seen == rk.cfg.score_layer
    score = rk.score_from_hidden
    rk.score_from_hidden = lambda *a, **kw: (score(*a, **kw)[0] + 1, None)
    assert torch.equal(rk.rank_host(batch)[0], full + 1)


@pytest.mark.parametrize("dtype,D,lens", [(torch.float32, 128, [512, 4096]), (torch.bfloat16, 64, [512, 8192])])
def test_long_query_block_within_the_scratch_limit(dtype, D, lens):
    """Partials of all chunks would exceed the limit: fewer chunks, the same result (heads of three KV heads against 64 bits)."""
    N, Nk = 32, 8
    spans, q, k, v = packed([lens], N, Nk, D, dtype)
    out, lse = ops.attention(q, k, v, spans[0], spans[1], D ** -0.5, spans.max_block_len, return_lse=True)
    for n in (0, 13, 31):
        s = (q[0, n].double() @ k[0, n // 4].double().t()) * D ** -0.5
        s = s.masked_fill(torch.ones_like(s, dtype=torch.bool).triu(1), float("-inf"))
        ref = s.softmax(-1) @ v[0, n // 4].double()
        assert (out[0, :, n].double() - ref).norm() <= (1e-6 if dtype == torch.float32 else 1.7e-3) * ref.norm()
        assert (lse[0, n].double() - s.logsumexp(-1)).abs().max() < 1e-5


def test_scales_that_are_not_positive():
    """Refused where the tcgen05 kernel alone serves a shape, computed on CUDA cores elsewhere."""
    for N, Nk, D, dtype, refused in ((8, 2, 128, torch.bfloat16, True), (8, 2, 64, torch.bfloat16, False), (8, 2, 128, torch.float32, False)):
        spans, q, k, v = packed([[9, 30, 41, 24]], N, Nk, D, dtype)
        call = lambda s: ops.attention(q, k, v, spans[0], spans[1], s, spans.max_block_len)
        if refused:
            with pytest.raises(ValueError, match="scale must be positive"):
                call(-0.1)
        else:  # the same logits with the sign on the queries
            ref = ops.attention(-q, k, v, spans[0], spans[1], 0.1, spans.max_block_len)
            assert (call(-0.1).double() - ref.double()).norm() <= 1e-3 * ref.double().norm()


@pytest.mark.parametrize("N,Nk,D,lens", [(8, 1, 64, [[64] + [140] * 20 + [48]]), (8, 2, 128, [[64, 700, 650, 48]]), (8, 8, 128, [[64, 30, 35, 28, 48]] * 2)])
def test_fp32_gradients_stay_close_to_64_bits(N, Nk, D, lens):
    """Sums of hundreds of rows in fp32, each product rounded once: errors of the gradients, and of the output, against fp64
    autograd.  Bounds: 10 % above those of sums taken in parts of D / 4 and of 64 rows (one long sum: up to 1.4e-6)."""
    spans, q, k, v = packed(lens, N, Nk, D, torch.float32, seed=5)
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out, _ = cuda_blockrank_attention_forward(Layer(), *leaves, spans, D ** -0.5)
    go = torch.randn(out.shape, generator=torch.Generator(device="cuda").manual_seed(9), device="cuda")
    exact = [t.detach().double().requires_grad_(True) for t in leaves]
    start, ln = spans[0].tolist(), spans[1].tolist()
    S, M = q.shape[2], len(lens[0])
    ok = torch.zeros(len(lens), S, S, dtype=torch.bool, device="cuda")
    for b in range(len(lens)):
        for m in range(M):
            s, e = start[b][m], start[b][m] + ln[b][m]
            ok[b, s:e, s:e] = torch.ones(e - s, e - s, dtype=torch.bool, device="cuda").tril()
            if m > 0:
                ok[b, s:e, :ln[b][0] if m < M - 1 else s] = True
    logits = (exact[0] @ exact[1].repeat_interleave(N // Nk, 1).transpose(-1, -2)) * D ** -0.5
    p = logits.masked_fill(~ok[:, None], float("-inf")).softmax(-1).nan_to_num(0.0)
    ref = (p @ exact[2].repeat_interleave(N // Nk, 1)).transpose(1, 2)
    assert (out.detach().double() - ref.detach()).norm() <= 3e-7 * ref.detach().norm()
    for got, want, bound in zip(torch.autograd.grad(out, leaves, go), torch.autograd.grad(ref, exact, go.double()), (3.95e-7, 4.05e-7, 3.8e-7)):
        assert (got.double() - want).norm() <= bound * want.norm()


def test_launches_are_counted_where_they_happen():
    """One prompt of five short documents is one kernel; a call of more than one wave has a kernel in front, chunks one behind."""
    def count(call):
        before = ops.launch_count
        call()
        return ops.launch_count - before

    def attend(lens, N, Nk, D, dtype, raw=False, **kw):
        spans, q, k, v = packed(lens, N, Nk, D, dtype)
        return lambda: cuda_blockrank_attention_forward(Layer(), q, k, v, spans, 0.1, layers_to_return_scores=[0] if raw else [], **kw)

    short, long = [[27] + [60] * 5 + [19]], [[64] + [160] * 20 + [48]] * 4
    assert count(attend(short, 32, 8, 128, torch.bfloat16)) == 1
    assert count(attend(short, 32, 8, 128, torch.bfloat16, raw=True)) == 2
    assert count(attend(long, 32, 8, 128, torch.bfloat16)) == 3
    assert count(attend(short, 32, 8, 128, torch.float32)) == 2
    assert count(attend(long, 32, 8, 128, torch.float32)) == 3
    assert count(attend(short, 32, 8, 128, torch.bfloat16, blockrank_algo=_lib.ALGO_SIMT)) == 2
    for dtype, one, two in ((torch.bfloat16, 2, 3), (torch.float32, 2, 2)):  # backward of one block, of several
        for lens, n in (([[100]], one), (short, two)):
            spans, q, k, v = packed(lens, 32, 8, 128, dtype)
            leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
            out, _ = cuda_blockrank_attention_forward(Layer(), *leaves, spans, 0.1)
            assert count(lambda: torch.autograd.grad(out, leaves, torch.ones_like(out))) == n


@pytest.mark.parametrize("N,Nk,D", [(8, 2, 128), (8, 1, 64), (4, 4, 64)])
def test_fp32_chunked_query_block_on_a_padded_grid(N, Nk, D):
    """fp32 with a query block in several key chunks: padding between documents, a run of empty documents longer than a chunk,
    a prompt with one document only; output, lse and gradients against fp64 autograd."""
    M, H = 30, 48                                     # 1,440 slots: three chunks of 512
    lens = H_.random_lens(3, M, H, 9)
    lens[0][3:16] = [0] * 13                          # 624 empty slots
    lens[1] = [0] + [0] * (M - 3) + [40, H]           # empty prefix, everything in the last chunk
    mask = H_.ragged_mask(3, M, H, lens)
    q, k, v = H_.qkv(3, N, Nk, M * H, D, 5, torch.float32)
    start, ln = ops.spans_from_mask(mask.cuda())
    qd, kd, vd = (H_.to_cuda_view(t) for t in (q, k, v))
    out, lse = ops.attention(qd, kd, vd, start, ln, D ** -0.5, H, return_lse=True)
    exact = [t.double().requires_grad_(True) for t in (q, k, v)]
    ref, ref_lse = orc.attention_dense(*exact, mask, D ** -0.5)
    rows = mask.reshape(3, -1)
    assert (out.cpu().double() - ref.detach())[rows].norm() <= 1e-6 * ref.detach()[rows].norm()
    assert out.cpu()[~rows].abs().max() == 0
    live = rows[:, None].expand(3, N, M * H)
    assert (lse.cpu().double() - ref_lse.detach())[live].abs().max() < 1e-5
    g = torch.randn(ref.shape, generator=torch.Generator().manual_seed(1)) * rows[..., None, None]
    grads = ops.attention_bwd(qd, kd, vd, out, g.cuda(), lse, start, ln, D ** -0.5, H)
    for got, want in zip(grads, torch.autograd.grad(ref[rows], exact, g.double()[rows])):
        assert (got.cpu().double() - want).norm() <= 2e-6 * want.norm()


@pytest.mark.parametrize("nd,k", [(1, 1), (5, 5), (300, 10), (2048, 2048), (2048, 7), (2049, 12)])  # 2,049: the general path
def test_best_documents_with_ties_and_nan(nd, k):
    """Indices of the k best: best first, NaN in front, equal scores in document order (up to 2,048 documents)."""
    g = torch.Generator().manual_seed(nd)
    logits = torch.randint(-3, 4, (3, nd), generator=g).float() if nd <= 2048 else torch.randperm(3 * nd, generator=g).view(3, nd).float()
    logits[0, nd // 2] = float("nan")
    logits[1, 0], logits[1, -1] = float("-inf"), float("inf")
    got, top = _lib.host().download(logits.cuda(), k)
    assert torch.equal(got.nan_to_num(9.0), logits.nan_to_num(9.0)) and top.shape == (3, k) and top.dtype == torch.int64
    for b in range(3):
        key = [(0, 0.0) if x != x else (1, -x) for x in logits[b].tolist()]
        assert top[b].tolist() == sorted(range(nd), key=lambda i: (key[i], i))[:k]


def test_requests_of_other_types_and_layouts():
    """Tensors that cannot travel in one packed copy give the same scores: other integer types, strides, device tensors."""
    rk, batch = _requests(3, [30, 40, 50, 20, 4])
    full, order = rk.rank_host(batch, k=2)
    for name, f in (("input_ids", lambda t: t.int()), ("input_ids", lambda t: t.t().contiguous().t()), ("position_ids", lambda t: t.int()),
                    ("position_ids", lambda t: t.float()), ("signal_rows", lambda t: t.long()), ("signal_rows", lambda t: t.cuda()),
                    ("block_spans", lambda t: t.cuda())):
        logits, top = rk.rank_host(dict(batch, **{name: f(batch[name])}), k=2)
        assert torch.equal(logits, full) and torch.equal(top, order)


@pytest.mark.parametrize("row", [-1, "S"])
def test_signal_row_outside_the_prompt_is_reported(row):
    rk, batch = _requests(2, [30, 40, 50, 20, 4])
    rows = batch["signal_rows"].clone()
    rows[1, 0] = batch["input_ids"].shape[1] if row == "S" else row
    with pytest.raises(ValueError, match="signal row"):
        rk.rank_host(dict(batch, signal_rows=rows))
    assert torch.isfinite(rk.rank_host(batch)[0]).all()  # (the word is clear again)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_raw_score_gradient_with_infinite_keys_and_queries(dtype):
    """An infinity in the last slot's key or the last pair's query reaches what it multiplies, as an infinity."""
    g = torch.Generator().manual_seed(6)
    B, N, Nk, S, D, R = 1, 5, 1, 3 * 30, 64, 13          # 65 pairs and 90 slots: remainders of both tiles
    rb = lambda *s: (torch.rand(*s, generator=g) + 0.5).to(dtype)
    q, k, d_raw = rb(B, N, S, D), rb(B, Nk, S, D), rb(B, N, R, S)
    k[0, 0, S - 1, 3] = float("inf")
    q[0, N - 1, S - 1, 5] = float("inf")
    start, ln = ops.spans_from_mask(torch.ones(B, 3, 30, dtype=torch.bool).cuda())
    dq, dk = ops.raw_scores_bwd(q.cuda(), k.cuda(), d_raw.cuda(), start, ln, 0.5)
    want_q = torch.zeros(B, N, S, D)
    want_q[0, :, S - R:, 3] = float("inf")
    want_k = torch.zeros(B, Nk, S, D)
    want_k[..., 5] = float("inf")
    for got, want in ((dq, want_q), (dk, want_k)):
        assert not got.isnan().any() and torch.equal(got.float().cpu().isinf(), want.isinf()) and (got >= 0).all()


@pytest.mark.parametrize("B,N,Nk,R,docs", [(1, 4, 4, 1, 1), (2, 8, 2, 3, 40), (1, 40, 40, 2, 33), (1, 8, 2, 5, 257), (2, 32, 8, 2, 300),
                                              # one SM's last size, then clusters: all KV heads shared out evenly, one or none left
                                              # for the last CTA, too few to share, more documents than threads
                                              (1, 32, 8, 2, 256), (1, 40, 40, 2, 205), (2, 12, 3, 16, 86), (1, 48, 6, 8, 43),
                                              (1, 4, 1, 64, 65), (2, 32, 8, 8, 600)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_document_scores_merge(B, N, Nk, R, docs, dtype):
    """One document, rows that do not fill a warp's turn, more documents than a lane holds, more (document, group) pairs than
    threads: masses and logits against fp64.  Products of bf16 (and sums of 64 fp32 products) are good to 1e-6; the exponentials
    of logits up to 10 in magnitude take that to 1e-5."""
    gen = torch.Generator().manual_seed(N + docs)
    lens = torch.randint(1, 12, (B, docs + 2), generator=gen, dtype=torch.int32)
    start = torch.zeros_like(lens)
    start[:, 1:] = lens.cumsum(1)[:, :-1]
    S, D = int(lens.sum(1).max()), 64
    q, k = (torch.randn(B, s, h, D, generator=gen).to(dtype).cuda().transpose(1, 2) for s, h in ((R, N), (S, Nk)))
    rows = torch.arange(R, dtype=torch.int32).expand(B, R).contiguous()
    mass, logits = ops.doc_scores(q, k, start.cuda(), lens.cuda(), rows.cuda(), D ** -0.5)
    z = (q.double() @ k.double().repeat_interleave(N // Nk, 1).transpose(2, 3) * D ** -0.5).cpu()
    for b in range(B):
        lo, hi = int(start[b, 1]), int(start[b, -1])
        p = torch.softmax(z[b, :, :, lo:hi], -1)
        want = torch.stack([p[..., s - lo:s - lo + n].sum(-1) for s, n in zip(start[b, 1:-1].tolist(), lens[b, 1:-1].tolist())], -1)
        assert (mass[b].cpu().double() - want).norm() <= 1e-5 * want.norm()
        mean = want.mean((0, 1))
        assert (logits[b].cpu().double() * 0.05 - mean).norm() <= 1e-5 * mean.norm()  # (the default temperature)


def test_merge_of_one_long_list_is_spread_over_sms():
    """The same documents and signal rows as one prompt and as four: keys and products are the same, the merge has eight SMs or four
    times eight.  Measured: 257 and 179 us, a ratio of 1.44; with one SM per prompt 597 and 270 us, 2.21.  The bound lies between."""
    def call(B, docs, N=32, Nk=8, R=16, D=128, L=32):
        lens = torch.full((B, docs + 2), L, dtype=torch.int32)
        start = torch.arange(docs + 2, dtype=torch.int32).mul(L).expand(B, docs + 2).contiguous()
        q, k = (torch.randn(B, s, h, D, device="cuda").bfloat16().transpose(1, 2) for s, h in ((R, N), ((docs + 2) * L, Nk)))
        rows = torch.arange(R, dtype=torch.int32, device="cuda").expand(B, R).contiguous()
        start, lens = start.cuda(), lens.cuda()
        return lambda: ops.doc_scores(q, k, start, lens, rows, D ** -0.5)

    def best(f):
        times = []
        for _ in range(12):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            f()
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b))
        return min(times[2:])

    one, four = best(call(1, 2000)), best(call(4, 500))
    assert one < 1.8 * four, (one, four)
