"""Training-path kernels of the recurrent cells, Conv2d and expert-choice routing against the same modules on the CPU
reference backend in fp32 (parameters and inputs rounded to bf16 on both sides)."""
import pytest
import torch

from rustral_b200.core import CpuBackend, ForwardCtx
from rustral_b200.nn import Conv2d, Conv2dConfig, ExpertChoiceConfig, ExpertChoiceRouter, GruCell, LstmCell
from rustral_b200.nn.expert_choice import ec_select, ec_table
from tolerances import assert_close

pytestmark = pytest.mark.gpu
BE = CpuBackend()


def _to_cuda_bf16(cell):
    for name in ("wx", "wh", "b", "weight", "bias", "router"):
        p = getattr(cell, name, None)
        if p is not None:
            p.tensor = p.tensor.detach().bfloat16().cuda().requires_grad_()
    return cell


def _round_params(cell):
    for name in ("wx", "wh", "b", "weight", "bias", "router"):
        p = getattr(cell, name, None)
        if p is not None:
            p.tensor = p.tensor.detach().bfloat16().float().requires_grad_()
    return cell


@pytest.mark.parametrize("cls", [LstmCell, GruCell])
@pytest.mark.parametrize("T,B,I,H", [(6, 4, 32, 64), (3, 5, 24, 40)])
def test_recurrent_cells_train_on_the_gate_kernels(cls, T, B, I, H, cuda_status):
    ref, dev = _round_params(cls.new(BE, I, H, seed=3)), _to_cuda_bf16(cls.new(BE, I, H, seed=3))
    g = torch.Generator().manual_seed(T * 100 + B)
    xs = torch.randn(T, B, I, generator=g).bfloat16()
    w = torch.randn(T, B, H, generator=g).bfloat16()
    ctx = ForwardCtx.train(BE)
    xr = xs.float().requires_grad_()
    out_r, _ = ref.forward_sequence(xr, ctx)
    (out_r * w.float()).sum().backward()
    xd = xs.cuda().requires_grad_()
    out_d, _ = dev.forward_sequence(xd, ctx)
    (out_d.float() * w.cuda().float()).sum().backward()
    assert out_d.dtype == torch.bfloat16
    assert_close(out_d, out_r, "norm", "hidden states")
    assert_close(xd.grad, xr.grad, "attention_grad", "dx")
    for name in ("wx", "wh", "b"):
        assert_close(getattr(dev, name).tensor.grad, getattr(ref, name).tensor.grad, "attention_grad", f"d{name}")


@pytest.mark.parametrize("N,C,H,W,O,k,stride,nopad", [(2, 3, 16, 16, 8, 3, 1, False), (2, 3, 17, 23, 13, 3, 2, False),
                                                      (1, 8, 12, 12, 16, 5, 1, True), (3, 1, 28, 28, 6, 3, 1, False)])
def test_conv2d_trains_on_im2col_gemm_col2im_kernels(N, C, H, W, O, k, stride, nopad, cuda_status):
    conv = Conv2d.new(BE, Conv2dConfig(O, k, k, stride=stride, no_padding=nopad, in_channels=C), seed=5)
    g = torch.Generator().manual_seed(N * 10 + C)
    with torch.no_grad():
        conv.bias.tensor.copy_(torch.randn(O, generator=g) * 0.1)
    x = torch.randn(N, C, H, W, generator=g).bfloat16()
    wt, bs = conv.weight.tensor.detach().bfloat16(), conv.bias.tensor.detach().bfloat16()
    pad = 0 if nopad else k // 2
    xr, wr, br = x.float().requires_grad_(), wt.float().requires_grad_(), bs.float().requires_grad_()
    yr = torch.nn.functional.conv2d(xr, wr, br, stride=stride, padding=pad)
    dy = torch.randn(yr.shape, generator=g).bfloat16()
    yr.backward(dy.float())
    _to_cuda_bf16(conv)
    xd = x.cuda().requires_grad_()
    yd = conv(xd, ForwardCtx.train(BE))
    assert yd.shape == yr.shape and yd.dtype == torch.bfloat16
    yd.backward(dy.cuda())
    assert_close(yd, yr, "gemm_bf16", "conv output")
    assert_close(xd.grad, xr.grad, "attention_grad", "conv dx")
    assert_close(conv.weight.tensor.grad, wr.grad, "attention_grad", "conv dW")
    assert_close(conv.bias.tensor.grad, br.grad, "attention_grad", "conv db")
    # the same call twice gives the same bits (no atomics in col2im or in the reductions)
    xd2 = x.cuda().requires_grad_()
    conv.weight.tensor.grad = None
    conv(xd2, ForwardCtx.train(BE)).backward(dy.cuda())
    assert torch.equal(xd2.grad, xd.grad)


@pytest.mark.parametrize("T,E,cap", [(64, 4, 8), (1000, 8, 100), (4096, 16, 256), (33, 3, 33)])
def test_expert_choice_selection_and_table(T, E, cap, cuda_status):
    g = torch.Generator().manual_seed(T + E)
    probs = torch.softmax(torch.randn(T, E, generator=g), -1)
    probs[::7] = probs[0]                                    # exact ties across tokens
    idx_r, gate_r = ec_select(probs, cap)
    idx_d, gate_d = ec_select(probs.cuda(), cap)
    assert torch.equal(idx_d.cpu(), idx_r) and torch.equal(gate_d.cpu(), gate_r)
    assert torch.equal(ec_table(idx_d, T).cpu(), ec_table(idx_r, T))


def test_expert_choice_router_trains_on_native_kernels(cuda_status):
    d, E, T = 64, 4, 96
    cfg = ExpertChoiceConfig(d, E, 128, tokens_per_expert=24)
    ref, dev = _round_params(ExpertChoiceRouter.new(BE, cfg, seed=9)), _to_cuda_bf16(ExpertChoiceRouter.new(BE, cfg, seed=9))
    g = torch.Generator().manual_seed(1)
    with torch.no_grad():
        big = (torch.randn(E, d, generator=g) * 0.5).bfloat16()
        ref.router.tensor.copy_(big.float()); dev.router.tensor.copy_(big.cuda())
    ws = [(torch.randn(d, d, generator=g) * 0.1).bfloat16() for _ in range(E)]
    x = torch.randn(T, d, generator=g).bfloat16()
    dy = torch.randn(T, d, generator=g).bfloat16()
    xr = x.float().requires_grad_()
    wr = [w.float().requires_grad_() for w in ws]
    yr = ref.forward(xr, lambda e, rows: rows @ wr[e].t(), ForwardCtx.train(BE))
    yr.backward(dy.float())
    from rustral_b200 import ops
    xd = x.cuda().requires_grad_()
    wd = [w.cuda().requires_grad_() for w in ws]
    yd = dev.forward(xd, lambda e, rows: ops.linear(rows, wd[e]), ForwardCtx.train(BE))
    yd.backward(dy.cuda())
    assert dev.last_stats.unrouted_tokens == ref.last_stats.unrouted_tokens
    assert_close(yd, yr, "attention", "expert-choice output")
    assert_close(xd.grad, xr.grad, "attention_grad", "dx")
    assert_close(dev.router.tensor.grad, ref.router.tensor.grad, "attention_grad", "drouter")
    for e in range(E):
        assert_close(wd[e].grad, wr[e].grad, "attention_grad", f"dW{e}")


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,W,k,stride", [(8, 8, 2, 2), (9, 11, 3, 2), (7, 7, 3, 1), (6, 6, 6, 6)])
def test_max_pool2d_forward_and_backward(H, W, k, stride, dtype, cuda_status):
    from rustral_b200.nn.conv import global_max_pool2d, max_pool2d
    g = torch.Generator().manual_seed(H * 10 + k)
    x = torch.randn(3, 4, H, W, generator=g).to(dtype)
    xr = x.float().clone().requires_grad_()            # a copy: for fp32 `x.float()` is x itself
    yr = torch.nn.functional.max_pool2d(xr, k, stride)
    dy = torch.randn(yr.shape, generator=g).to(dtype)
    yr.backward(dy.float())
    xd = x.detach().cuda().requires_grad_()
    yd = max_pool2d(xd, k, stride)
    yd.backward(dy.cuda())
    assert torch.equal(yd.float().cpu(), yr.detach().to(dtype).float())
    assert torch.allclose(xd.grad.float().cpu(), xr.grad, atol=2e-2 if dtype is torch.bfloat16 else 1e-6)
    if H == W:
        assert torch.equal(global_max_pool2d(x.cuda()).float().cpu(), x.float().amax((2, 3)))


def test_a_captured_graph_owns_its_scratch(cuda_status):
    """Scratch that a graph names must not be in the grow-only buffers: those are freed when a later call needs more, and the graph would
    read and write what is not its own any more."""
    from rustral_b200 import ops
    from rustral_b200.ops import elementwise, embed, norm, optim
    a = torch.randn(500, 256, device="cuda").bfloat16()
    wide = torch.randn(64, 40000, device="cuda").bfloat16()
    want, want_wide = ops.sum_dim0(a), ops.sum_dim0(wide)
    caches = [m._scratch for m in (elementwise, embed, norm, optim)]
    before = [{k: v.data_ptr() for k, v in c.items()} for c in caches]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got, total = ops.sum_dim0(a), ops.sum_all(a)
        got_wide = ops.sum_dim0(wide)
    assert [{k: v.data_ptr() for k, v in c.items()} for c in caches] == before
    torch.cuda.empty_cache()
    graph.replay()
    assert torch.equal(got, want) and torch.equal(got_wide, want_wide) and torch.isfinite(total)


@pytest.mark.parametrize("splits", [0, 3])
def test_a_captured_graph_owns_its_split_products_scratch(splits, cuda_status):
    """Two graphs whose products split their contraction, replayed side by side on two streams: each has slabs of its own, and the buffer of
    the streams' direct calls is not among them."""
    from rustral_b200.ops import matmul
    from rustral_b200.ops.matmul import gemm
    g = torch.Generator(device="cuda").manual_seed(splits)
    a, b = ([torch.randn(16384, n, device="cuda", generator=g).bfloat16() for _ in range(2)] for n in (256, 384))
    want = [gemm(x, y, a_mn=True, b_mn=True, out_dtype=torch.float32, splits=splits) for x, y in zip(a, b)]
    before = {k: v.data_ptr() for k, v in matmul._workspaces.items()}
    graphs, got = [], []
    for x, y in zip(a, b):
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            got.append(gemm(x, y, a_mn=True, b_mn=True, out_dtype=torch.float32, splits=splits))
    assert {k: v.data_ptr() for k, v in matmul._workspaces.items()} == before
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    for _ in range(5):
        for t in got:
            t.zero_()
        torch.cuda.synchronize()
        for s, graph in zip(streams, graphs):
            with torch.cuda.stream(s):
                for _ in range(10):
                    graph.replay()
        torch.cuda.synchronize()
        for t, w in zip(got, want):
            assert torch.equal(t, w)


def test_routing_gradient_takes_a_number_under_capture(cuda_status):
    """The scale of the balancing loss as a number, as a tensor and as nothing, directly and captured."""
    from rustral_b200.ops import moe
    g = torch.Generator(device="cuda").manual_seed(1)
    logits, dw = torch.randn(40, 8, device="cuda", generator=g), torch.randn(40, 2, device="cuda", generator=g)
    idx, w, probs = moe.route(logits, 2, True)
    counts = torch.bincount(idx.reshape(-1).long(), minlength=8).int()
    call = lambda s: moe.route_backward(probs, idx, w, dw, counts, True, s)  # noqa: E731
    want = [call(torch.tensor(s, device="cuda")) for s in (0.25, 0.0)]
    cpu = moe.route_backward(probs.cpu(), idx.cpu(), w.cpu(), dw.cpu(), counts.cpu(), True, 0.25)
    assert torch.allclose(want[0].cpu(), cpu, rtol=1e-4, atol=1e-6)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [call(0.25), call(0.0)]
    graph.replay()
    for a, b, c in zip(want, got, (0.25, 0.0)):
        assert torch.equal(a, b) and torch.equal(a, call(c))


@pytest.mark.parametrize("tokens,out,inp,splits,block", [
    (64, 64, 64, 0, 0), (1998, 1152, 384, 0, 0), (2100, 384, 1536, 3, 0), (4096, 2304, 768, 0, 0), (4096, 768, 768, 4, 256), (1024, 264, 520, 1, 128),
    (333, 136, 200, 1, 192), (70, 8, 24, 1, 64), (32768, 256, 256, 0, 0), (8192, 3072, 768, 2, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_bias_gradient_inside_the_weight_gradient(tokens, out, inp, splits, block, accumulate, cuda_status):
    """Column sums of the first operand beside the product: one- and two-CTA tiles of every width, ragged tiles and contractions, slabs of splits, added to
    what is there.  Bound: fp32 sums of at most `tokens` bf16 numbers (2^-24 of the sum of magnitudes per addition, about tokens / 64 + 16 of them in
    a row); twice the same bits; the product is the one without sums."""
    from rustral_b200.ops import matmul
    g = torch.Generator(device="cuda").manual_seed(tokens + out)
    dy = (torch.randn(tokens, out + 8, device="cuda", generator=g) + 0.5).bfloat16()[:, :out]
    x = torch.randn(tokens, inp, device="cuda", generator=g).bfloat16()
    w0, b0 = torch.randn(out, inp, device="cuda", generator=g), torch.randn(out, device="cuda", generator=g)
    runs = []
    for _ in range(2):
        w, b = w0.clone(), b0.clone()
        matmul.gemm(dy, x, a_mn=True, b_mn=True, out=w, accumulate=accumulate, splits=splits, block_n=block, col_sum=b)
        runs.append((w, b))
    plain = w0.clone()
    matmul.gemm(dy, x, a_mn=True, b_mn=True, out=plain, accumulate=accumulate, splits=splits, block_n=block)
    want = dy.double().sum(0) + (b0.double() if accumulate else 0)
    bound = 2.0 ** -24 * (tokens / 64 + 16) * dy.double().abs().sum(0) + 2.0 ** -23 * want.abs()
    assert torch.equal(runs[0][1], runs[1][1]) and torch.equal(runs[0][0], plain)
    assert ((runs[0][1].double() - want).abs() <= bound).all()


@pytest.mark.parametrize("vocab,tokens", [(1, 5), (31, 100), (512, 3000), (16384, 5000), (16385, 4000), (50257, 9000)])
def test_embedding_gradient_for_vocabularies_around_a_scan_round(vocab, tokens, cuda_status):
    """The bucket offsets of the ids at the edges of a warp's, a block's and a round's share, with ids that occur often, never and out of range."""
    from rustral_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(vocab)
    ids = torch.randint(0, vocab, (tokens,), device="cuda", generator=g)
    ids[::7], ids[1] = vocab - 1, 0
    dy = torch.randn(tokens, 64, device="cuda", generator=g).bfloat16()
    got = torch.zeros(vocab, 64, device="cuda")
    ops.embedding_backward(ids, dy, got, None, tokens)
    want = torch.zeros(vocab, 64, dtype=torch.float64, device="cuda").index_add(0, ids, dy.double())
    often = torch.zeros(vocab, 64, dtype=torch.float64, device="cuda").index_add(0, ids, dy.double().abs())
    count = torch.bincount(ids, minlength=vocab)[:, None]
    assert ((got.double() - want).abs() <= 2.0 ** -24 * (count + 1) * often).all()


@pytest.mark.parametrize("hook", [False, True])
@pytest.mark.parametrize("captured", [False, True])
def test_a_split_that_fills_the_scratch_takes_column_sums_too(hook, captured, cuda_status):
    """Eight parts of 4096 x 1024 are exactly the scratch of split contractions: asked for directly or by a plan table, they are taken with column sums
    as without.  The product is the one without sums; the sums' bound as above."""
    from rustral_b200.ops import matmul
    tokens, out, inp = 8192, 4096, 1024
    assert 8 * out * inp * 4 == matmul.WORKSPACE_BYTES
    g = torch.Generator(device="cuda").manual_seed(5)
    dy = torch.randn(tokens, out, device="cuda", generator=g).bfloat16()
    x = torch.randn(tokens, inp, device="cuda", generator=g).bfloat16()
    w, b, plain = torch.empty(out, inp, device="cuda"), torch.empty(out, device="cuda"), torch.empty(out, inp, device="cuda")
    call = lambda dst, splits, sums: matmul.gemm(dy, x, a_mn=True, b_mn=True, out=dst, splits=splits, col_sum=sums)  # noqa: E731
    call(plain, 8, None)
    matmul._PLAN_HOOK = (lambda *a: {"block_n": 0, "splits": 8, "group_m": 0}) if hook else None
    try:
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                call(w, 0 if hook else 8, b)
            graph.replay()
        else:
            call(w, 0 if hook else 8, b)
    finally:
        matmul._PLAN_HOOK = None
    assert torch.equal(w, plain)
    want = dy.double().sum(0)
    assert ((b.double() - want).abs() <= 2.0 ** -24 * (tokens / 64 + 16) * dy.double().abs().sum(0) + 2.0 ** -23 * want.abs()).all()


@pytest.mark.parametrize("tokens,out,inp,splits,inside", [
    (1, 64, 64, 0, False), (64, 64, 64, 0, True), (70, 8, 24, 0, False), (127, 136, 64, 0, True), (1024, 256, 256, 0, True), (1998, 1152, 384, 0, False),
    (4096, 2304, 768, 0, True), (6144, 776, 768, 3, True), (6144, 780, 256, 0, False), (8192, 3072, 768, 2, True), (8200, 264, 256, 12, False),
    (8256, 256, 256, 0, False), (16384, 768, 768, 0, True), (32768, 2304, 768, 0, True), (32768, 256, 520, 3, True), (32767, 200, 768, 6, True)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_bias_gradient_has_the_bits_of_a_column_sum(tokens, out, inp, splits, inside, accumulate, cuda_status):
    """Inside the weight gradient's product where the slabs of `sum_dim0` are whole k-blocks: one and several blocks to a slab, slabs that reach into the next
    part of the contraction, a last one that is cut short, ragged columns; in launches of its own elsewhere."""
    from rustral_b200 import _native as N
    from rustral_b200.ops import matmul, sum_dim0
    g = torch.Generator(device="cuda").manual_seed(tokens + out)
    dy = (torch.randn(tokens, out + 8 - out % 8, device="cuda", generator=g) * 3 + 0.1).bfloat16()[:, :out]
    x = torch.randn(tokens, inp, device="cuda", generator=g).bfloat16()
    b0 = torch.randn(out, device="cuda", generator=g)
    w, b, plain, want = torch.zeros(out, inp, device="cuda"), b0.clone(), torch.zeros(out, inp, device="cuda"), b0.clone()
    call = lambda d, **kw: matmul.gemm(dy, x, a_mn=True, b_mn=True, out=d, accumulate=accumulate, splits=splits, **kw)  # noqa: E731
    before = N.launch_count
    call(plain)
    product = N.launch_count - before
    call(w, col_sum=b)
    assert (N.launch_count - before - 2 * product == 1) == inside
    sum_dim0(dy, out=want, accumulate=accumulate)
    assert torch.equal(b, want) and torch.equal(w, plain)


@pytest.mark.parametrize("vocab,tokens", [(31, 100), (16385, 4000), (50257, 9000)])
def test_embedding_gradient_leaves_out_ids_out_of_range(vocab, tokens, cuda_status):
    """Negative ids and ids behind the table add to no row."""
    from rustral_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(tokens)
    ids = torch.randint(0, vocab, (tokens,), device="cuda", generator=g)
    ids[::5], ids[1::5], ids[2], ids[3] = -1, vocab, vocab + 12345, -(1 << 40)
    dy = torch.randn(tokens, 64, device="cuda", generator=g).bfloat16()
    got = torch.zeros(vocab, 64, device="cuda")
    ops.embedding_backward(ids, dy, got, None, tokens)
    real = (ids >= 0) & (ids < vocab)
    want, often = (torch.zeros(vocab, 64, dtype=torch.float64, device="cuda").index_add(0, ids[real], v[real]) for v in (dy.double(), dy.double().abs()))
    assert ((got.double() - want).abs() <= 2.0 ** -24 * (torch.bincount(ids[real], minlength=vocab)[:, None] + 1) * often).all()
