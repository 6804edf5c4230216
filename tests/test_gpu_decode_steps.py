"""Decoding kernels at the edges of their work splits: rotation with append, slices of the cached tokens."""
import pytest
import torch

from rustral_b200 import _native as N
from rustral_b200.ops import paged
from rustral_b200.ops import rotary

pytestmark = pytest.mark.gpu


def _rotated(x, pos, heads, dim, inverse):
    """x [rows, heads * dim] in 64 bits, turned by its positions; the bound: a bf16 result, fp32 angles up to 20000 (2^-24 of them)."""
    freq = 10000.0 ** (-torch.arange(dim // 2, device="cuda").double() * 2 / dim)
    a = pos.double()[:, None, None] * freq * (-1 if inverse else 1)
    u, v = x.double().view(x.shape[0], heads, dim).split(dim // 2, -1)
    want = torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], -1)
    return want, 2.0 ** -8 * want.abs() + 20000 * 2.0 ** -22 * (u.abs() + v.abs()).repeat(1, 1, 2)


@pytest.mark.parametrize("tokens,heads,kv,dim", [(1, 4, 1, 64), (7, 6, 2, 80), (33, 16, 4, 128), (3000, 30, 5, 64)])
def test_rope_append_is_rope_and_append(tokens, heads, kv, dim, cuda_status):
    """The one launch against the two, bit for bit; skipped tokens; wide rows."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    cols = (heads + 2 * kv) * dim
    qkv = torch.randn(tokens, cols + 8, device="cuda", generator=g).bfloat16()[:, :cols]
    other = qkv.clone()
    pos = torch.randint(0, 20000, (tokens,), device="cuda", generator=g)
    slots = torch.randperm(tokens + 32, device="cuda", generator=g)[:tokens]
    slots[::5] = -1
    kc, vc = (torch.zeros((tokens + 47) // 16, 16, kv, dim, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    kc2, vc2 = kc.clone(), vc.clone()
    before = N.launch_count
    rotary.rope_append_(qkv, heads, kv, dim, pos, 10000.0, kc, vc, slots)
    assert N.launch_count == before + 1                       # none of these is long enough for two launches
    rotary.rope_(other, heads + kv, dim, positions=pos, theta=10000.0)
    paged.kv_append(other[:, heads * dim:(heads + kv) * dim], other[:, (heads + kv) * dim:], kc2, vc2, slots)
    assert torch.equal(qkv, other) and torch.equal(kc, kc2) and torch.equal(vc, vc2)


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("tokens,heads,dim", [(7, 6, 80), (12000, 30, 64), (6000, 29, 128)])
def test_rotation_against_64_bit(tokens, heads, dim, inverse, cuda_status):
    """One head per thread, and four where that leaves a thread for every lane of the GPU (the two long ones), with counts of heads that four
    does not divide."""
    assert (tokens * ((heads + 3) // 4) * (dim // 16) >= 148 * 2048) == (tokens > 1000)
    g = torch.Generator(device="cuda").manual_seed(tokens)
    pos = torch.randint(0, 20000, (tokens,), device="cuda", generator=g)
    x = torch.randn(tokens, heads * dim + 8, device="cuda", generator=g).bfloat16()
    want, bound = _rotated(x[:, :heads * dim].contiguous(), pos, heads, dim, inverse)
    got = x.clone()
    rotary.rope_(got, heads, dim, positions=pos, theta=10000.0, inverse=inverse)
    assert torch.equal(got[:, heads * dim:], x[:, heads * dim:])
    assert ((got[:, :heads * dim].double().view(tokens, heads, dim) - want).abs() <= bound).all()


@pytest.mark.parametrize("tokens", [3, 9000])
def test_rope_append_refuses_what_it_cannot_address(tokens, cuda_status):
    """The one launch and the two refuse the same: caches of other heads or types, slots of another type or number."""
    heads, kv, dim = 30, 5, 64
    qkv = torch.zeros(tokens, (heads + 2 * kv) * dim, device="cuda").bfloat16()
    pos, slots = torch.arange(tokens, device="cuda"), torch.full((tokens,), -1, device="cuda")
    cache = torch.zeros(2, 16, kv, dim, device="cuda").bfloat16()
    rotary.rope_append_(qkv, heads, kv, dim, pos.int(), 10000.0, cache, cache.clone(), slots)
    for bad in (dict(k=cache.view(2, 16, 1, kv * dim), v=cache.view(2, 16, 1, kv * dim)), dict(v=cache.float()), dict(k=cache.cpu()),
                dict(slots=slots.int()), dict(slots=slots[1:]), dict(slots=torch.stack([slots, slots], 1)[:, 0]), dict(pos=pos[1:])):
        with pytest.raises(TypeError):
            rotary.rope_append_(qkv, heads, kv, dim, bad.get("pos", pos), 10000.0, bad.get("k", cache), bad.get("v", cache), bad.get("slots", slots))


@pytest.mark.parametrize("batch,heads,kv,dim,longest,width", [(1, 8, 2, 128, 2500, 400), (64, 8, 4, 128, 1300, 1024), (120, 32, 16, 64, 700, 64),
                                                             (3, 4, 4, 64, 257, 1024)])
def test_slices_of_the_context(batch, heads, kv, dim, longest, width, cuda_status):
    """Several slices per CTA and fewer slices than CTAs, up to four warps' worth of sequences; lengths from 1 to the longest."""
    g = torch.Generator(device="cuda").manual_seed(batch)
    need = (longest + 15) // 16
    blocks = batch * need
    kc, vc = (torch.randn(blocks, 16, kv, dim, device="cuda", generator=g).bfloat16() for _ in range(2))
    table = torch.zeros(batch, width, dtype=torch.int32, device="cuda")
    table[:, :need] = torch.randperm(blocks, device="cuda", generator=g).view(batch, need).int()
    ctx = torch.randint(1, longest + 1, (batch,), device="cuda", generator=g, dtype=torch.int32)
    ctx[0], ctx[-1] = longest, 1 if batch > 1 else longest
    q = torch.randn(batch, heads * dim, device="cuda", generator=g).bfloat16()
    got = paged.paged_attention_decode(q, kc, vc, table, ctx).view(batch, heads, dim).double()
    for b in {0, 1 % batch, batch // 2, batch - 1}:
        n = int(ctx[b])
        rows = table[b, :need].long()
        k, v = (c[rows].reshape(-1, kv, dim)[:n].repeat_interleave(heads // kv, 1).double() for c in (kc, vc))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double().view(heads, dim), k) * dim ** -0.5, -1)
        want = torch.einsum("hn,nhd->hd", p, v)
        # weights rounded to bf16 (2^-9 each, against the unrounded sum) and a bf16 result
        assert ((got[b] - want).abs() <= 2.0 ** -8 * torch.einsum("hn,nhd->hd", p, v.abs()) + 1e-3).all(), b


@pytest.mark.parametrize("rule", [None, dict(chunk=300), dict(window=500, keep_first=7, sink=True, softcap=20.0)])
@pytest.mark.parametrize("heads,kv,dim", [(8, 2, 128), (40, 2, 64)])
def test_a_sequence_has_the_same_bits_alone_and_beside_others(heads, kv, dim, rule, cuda_status):
    """Slices are cut by a sequence's own length: neither the batch, nor the others' lengths (among them none and a very long one), nor the
    width of the tables changes a bit.  40 heads on 2 take two passes of 16 and one of 8."""
    from rustral_b200.ops.attention import ScoreRule
    rule = ScoreRule(**rule) if rule else None
    g = torch.Generator(device="cuda").manual_seed(dim)
    lens = [1, 255, 256, 257, 9000, 0, 2049, 2048] + [33 * i % 700 + 1 for i in range(62)]
    need = [(n + 15) // 16 for n in lens]
    kc, vc = (torch.randn(sum(need), 16, kv, dim, device="cuda", generator=g).bfloat16() for _ in range(2))
    pages = torch.randperm(sum(need), device="cuda", generator=g).int()
    table = torch.zeros(len(lens), 1024, dtype=torch.int32, device="cuda")
    for i, n in enumerate(need):
        table[i, :n] = pages[sum(need[:i]):sum(need[:i + 1])]
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    q = torch.randn(len(lens), heads * dim, device="cuda", generator=g).bfloat16()
    run = lambda rows, width: paged.paged_attention_decode(q[rows], kc, vc, table[rows, :width].contiguous(), ctx[rows], rule=rule)  # noqa: E731
    together = run(list(range(len(lens))), 1024)
    for i in (4, 6, 7):                                       # 36, 9 and 8 slices: both forms of the merge (without a rule: all are seen)
        rows = table[i, :need[i]].long()
        k, v = (c[rows].reshape(-1, kv, dim)[:lens[i]].repeat_interleave(heads // kv, 1).double() for c in (kc, vc))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].double().view(heads, dim), k) * dim ** -0.5, -1)
        # weights rounded to bf16 (2^-9 each, against the unrounded sum) and a bf16 result
        bound = 2.0 ** -8 * torch.einsum("hn,nhd->hd", p, v.abs()) + 1e-3
        off = (together[i].double().view(heads, dim) - torch.einsum("hn,nhd->hd", p, v)).abs()
        assert rule is not None or (off <= bound).all(), i
    for i in (0, 1, 2, 3, 4, 6, 7, 40, 69):
        assert torch.equal(run([i], 1024)[0], together[i]), i
        if need[i] > 16:
            assert torch.equal(run([i], need[i])[0], together[i]), i
    some = [3, 4, 69, 6]
    assert torch.equal(run(some, 700), together[some])


@pytest.mark.parametrize("batch,heads,kv,dim,longest,width,theta", [
    (1, 8, 2, 128, 2500, 400, 10000.0), (36, 8, 4, 128, 1300, 96, 500000.0), (10, 32, 16, 64, 700, 64, 10000.0), (3, 4, 4, 64, 257, 1024, 0.0),
    (5, 16, 1, 128, 20000, 1250, 10000.0), (2, 12, 12, 64, 1, 1, 0.0)])
def test_attention_step_is_rotation_append_and_attention(batch, heads, kv, dim, longest, width, theta, cuda_status):
    """The one launch of a decoding step against the three, for lengths at the edges of tiles and slices, in wide rows, twice in a
    row on the same counters; a table entry out of range keeps its token out of the cache."""
    g = torch.Generator(device="cuda").manual_seed(batch)
    need = (longest + 15) // 16
    blocks = batch * need + 1
    kc, vc = (torch.randn(blocks, 16, kv, dim, device="cuda", generator=g).bfloat16() for _ in range(2))
    table = torch.zeros(batch, width, dtype=torch.int32, device="cuda")
    table[:, :need] = 1 + torch.randperm(blocks - 1, device="cuda", generator=g).view(batch, need).int()
    edges = [n for n in (1, 32, 33, 128, 129, 256, 257, 512, 513, longest) if n <= longest]
    lens = torch.tensor([longest] + [edges[i % len(edges)] for i in range(batch - 1)], dtype=torch.int32, device="cuda")
    cols = (heads + 2 * kv) * dim
    arrived = torch.zeros(batch * kv, dtype=torch.int32, device="cuda")
    pos = (lens - 1).long()
    slots = table.gather(1, (pos // 16)[:, None]).view(-1).long() * 16 + pos % 16
    for turn in range(2):
        qkv = torch.randn(batch, cols + 8, device="cuda", generator=g).bfloat16()[:, :cols]
        other, k2, v2 = qkv.clone(), kc.clone(), vc.clone()
        if theta:
            rotary.rope_append_(other, heads, kv, dim, pos, theta, k2, v2, slots)
        else:
            paged.kv_append(other[:, heads * dim:(heads + kv) * dim], other[:, (heads + kv) * dim:], k2, v2, slots)
        want = paged.paged_attention_decode(other[:, :heads * dim], k2, v2, table, lens, 0.1)
        assert paged.step_supported(qkv, heads, kv, dim, kc, vc, table)
        before = qkv.clone()
        got = paged.attention_step(qkv, heads, kv, dim, theta, kc, vc, table, lens, arrived, 0.1)
        torch.cuda.synchronize()
        assert torch.equal(qkv, before) and torch.equal(kc, k2) and torch.equal(vc, v2) and not arrived.any()
        # the same arithmetic in the same order, but for contractions the compiler chooses: one rounding to bf16
        assert ((got.float() - want.float()).abs() <= 2.0 ** -7 * want.float().abs() + 1e-6).all()
    # an entry out of range: nothing is stored for that sequence
    table[0, pos[0] // 16] = blocks
    k2, v2 = kc.clone(), vc.clone()
    paged.attention_step(torch.full((batch, cols), 3.0, device="cuda").bfloat16(), heads, kv, dim, theta, kc, vc, table, lens, arrived, 0.1)
    own = torch.ones(blocks * 16, dtype=torch.bool, device="cuda")
    own[slots[1:]] = False
    assert torch.equal(kc.view(-1, kv, dim)[own], k2.view(-1, kv, dim)[own]) and torch.equal(vc.view(-1, kv, dim)[own], v2.view(-1, kv, dim)[own])
    N.read_status(clear=True)


@pytest.mark.parametrize("rows,n,k", [(1, 768, 768), (1, 50304, 768), (4, 640, 4096), (8, 528, 2048), (3, 272, 200), (1, 3072, 1032), (2, 28672, 4096),
                                      (9, 256, 256), (5, 256, 4096)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_inside_a_product_with_few_rows(rows, n, k, rms, cuda_status):
    """The norm formed by the product's own blocks against norm and product, at one and several parts of the contraction, with stages that are filled
    again, blocks that end inside 64 columns, and one size too many (rows, numbers): two launches.  Both round the normed rows to bf16; their
    statistics differ in the order of fp32 sums, so a number may round the other way: 2^-8 of sqrt(k) terms beside the result's own rounding."""
    from rustral_b200.ops import matmul, norm as norm_ops
    g = torch.Generator(device="cuda").manual_seed(rows * n)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, w, gamma = rand(rows, k + 8)[:, :k] * 3 + 1, rand(n, k) * 0.05, rand(k)
    beta, bias = (None, None) if rms else (rand(k), rand(n))
    for act, weight in (("none", w), ("gelu", w), ("swiglu", w)):
        b = None if act == "swiglu" else bias
        before = N.launch_count
        got = matmul.norm_gemm(x, gamma, beta, 1e-5, rms, weight, bias=b, act=act, b_constant=True)
        one = rows <= 8 and rows * k <= 16384
        assert (N.launch_count - before == 1) == one
        h = norm_ops.norm_forward(x, gamma, beta, 1e-5, rms)[0]
        want = rotary.swiglu_product(h, weight) if act == "swiglu" else matmul.gemm(h, weight, bias=b, act=act)
        e = (got.float() - want.float()).abs()
        assert (e <= 2.0 ** -7 * want.float().abs() + 2.0 ** -8 * want.float().pow(2).mean().sqrt()).all(), e.max()


@pytest.mark.parametrize("rows,n,k", [(1, 768, 768), (4, 640, 4096), (8, 528, 2048), (7, 272, 1024), (3, 272, 200), (5, 264, 1032), (2, 28672, 4096), (3, 520, 3000)])
@pytest.mark.parametrize("rms", [False, True])
def test_norm_inside_a_product_has_the_bits_of_norm_and_product(rows, n, k, rms, cuda_status):
    """One, two and four warps to a row, rows that leave warps without one, blocks that end inside 64 columns; a row has the same bits beside others."""
    from rustral_b200.ops import matmul, norm as norm_ops
    g = torch.Generator(device="cuda").manual_seed(rows * n)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, w, gamma = rand(rows, k + 8)[:, :k] * 3 + 1, rand(n, k) * 0.05, rand(k)
    beta, bias = (None, None) if rms else (rand(k), rand(n))
    for act in ("none", "gelu", "swiglu") if n % 16 == 0 else ("none", "gelu"):        # swiglu: halves of whole 16-byte pieces
        b = None if act == "swiglu" else bias
        before = N.launch_count
        got = matmul.norm_gemm(x, gamma, beta, 1e-5, rms, w, bias=b, act=act, b_constant=True)
        assert N.launch_count - before == 1
        h = norm_ops.norm_forward(x, gamma, beta, 1e-5, rms)[0]
        assert torch.equal(got, rotary.swiglu_product(h, w) if act == "swiglu" else matmul.gemm(h, w, bias=b, act=act))
        assert torch.equal(got[-1:], matmul.norm_gemm(x[-1:], gamma, beta, 1e-5, rms, w, bias=b, act=act))


@pytest.mark.parametrize("batch,heads,kv,dim,longest,width,theta", [
    (1, 8, 2, 128, 2500, 400, 10000.0), (36, 8, 4, 128, 1300, 96, 500000.0), (10, 32, 16, 64, 700, 64, 10000.0), (3, 4, 4, 64, 257, 1024, 0.0),
    (2, 16, 1, 128, 20000, 1250, 10000.0), (3, 12, 1, 64, 9000, 600, 0.0)])
def test_attention_step_has_the_bits_of_the_three_launches(batch, heads, kv, dim, longest, width, theta, cuda_status):
    """One slice, some and more than 32; both forms of the merge; lengths at the edges of tiles and slices."""
    g = torch.Generator(device="cuda").manual_seed(batch)
    need = (longest + 15) // 16
    kc, vc = (torch.randn(batch * need, 16, kv, dim, device="cuda", generator=g).bfloat16() for _ in range(2))
    table = torch.zeros(batch, width, dtype=torch.int32, device="cuda")
    table[:, :need] = torch.randperm(batch * need, device="cuda", generator=g).view(batch, need).int()
    edges = [n for n in (1, 32, 33, 128, 129, 256, 257, 512, 513, 2048, 2049, longest) if n <= longest]
    lens = torch.tensor([longest] + [edges[i % len(edges)] for i in range(batch - 1)], dtype=torch.int32, device="cuda")
    qkv = torch.randn(batch, (heads + 2 * kv) * dim, device="cuda", generator=g).bfloat16()
    pos = (lens - 1).long()
    slots = table.gather(1, (pos // 16)[:, None]).view(-1).long() * 16 + pos % 16
    other, k2, v2 = qkv.clone(), kc.clone(), vc.clone()
    if theta:
        rotary.rope_append_(other, heads, kv, dim, pos, theta, k2, v2, slots)
    else:
        paged.kv_append(other[:, heads * dim:(heads + kv) * dim], other[:, (heads + kv) * dim:], k2, v2, slots)
    arrived = torch.zeros(batch * kv, dtype=torch.int32, device="cuda")
    for scale in (dim ** -0.5, 0.37):
        want = paged.paged_attention_decode(other[:, :heads * dim], k2, v2, table, lens, scale)
        got = paged.attention_step(qkv, heads, kv, dim, theta, kc, vc, table, lens, arrived, scale)
        assert torch.equal(got, want) and torch.equal(kc, k2) and torch.equal(vc, v2)


@pytest.mark.parametrize("arch,d,heads,kv,blocks", [("gpt2", 768, 12, 12, 1024), ("llama", 2048, 16, 4, 1024), ("llama", 4096, 32, 8, 700)])
def test_a_decoded_sequence_has_the_same_bits_beside_others(arch, d, heads, kv, blocks, cuda_status):
    """Logits, keys and values of one sequence alone and in batches on both sides of every limit: norms inside the products (8 rows, 16384 numbers),
    attention in one launch (slices that the tables have room for), replayed and eager."""
    from rustral_b200.models.config import GPTConfig
    from rustral_b200.serve.model_runner import ModelRunner
    from rustral_b200.serve.weights import InferenceWeights
    cfg = GPTConfig(vocab_size=1000, seq_len=1024 if arch == "gpt2" else 8192, n_layer=2, n_head=heads, n_kv_head=kv, d_model=d, ffn_dim=2 * d, arch=arch)
    weights = InferenceWeights.random_llama(cfg, "cuda", seed=3) if arch == "llama" else None
    r = ModelRunner(cfg, params=weights, device="cuda", num_blocks=blocks, block_size=16, seed=3)
    g = torch.Generator(device="cuda").manual_seed(d)
    lens = [700] + [(97 * i) % 300 + 1 for i in range(33)]
    for i, n in enumerate(lens):
        assert r.cache.allocate(i, n)
    for l in range(2):
        r.cache.k[l].normal_(0.0, 0.9, generator=g)
        r.cache.v[l].normal_(0.0, 0.9, generator=g)
    for graphs in (True, False):
        r.use_graphs = graphs
        alone = r.decode([0], [17], lens[:1]).clone()
        for batch in (2, 3, 4, 5, 8, 9, 16, 34):
            ids = list(range(1, batch)) + [0]
            got = r.decode(ids, [5] * (batch - 1) + [17], [lens[i] for i in ids])
            assert torch.equal(got[-1:], alone), batch


@pytest.mark.parametrize("dim,many", [(128, False), (64, True)])
def test_attention_goes_by_the_slices_that_are_there(dim, many, monkeypatch, cuda_status):
    """In tables of one width: twelve short sequences attend in one launch, twelve long ones with heads of 128 in three, eager and captured, in turn; a short
    one has the same bits beside both."""
    from rustral_b200.models.config import GPTConfig
    from rustral_b200.ops import paged as paged_ops
    from rustral_b200.serve.model_runner import ModelRunner
    from rustral_b200.serve.weights import InferenceWeights
    cfg = GPTConfig(vocab_size=512, seq_len=4096, n_layer=2, n_head=8, n_kv_head=4, d_model=8 * dim, ffn_dim=512, arch="llama")
    r = ModelRunner(cfg, params=InferenceWeights.random_llama(cfg, "cuda", seed=3), device="cuda", num_blocks=12 * 256, block_size=16, seed=3)
    g = torch.Generator(device="cuda").manual_seed(dim)
    for i in range(12):
        assert r.cache.allocate(i, 4096)
    for l in range(2):
        r.cache.k[l].normal_(0.0, 0.9, generator=g)
        r.cache.v[l].normal_(0.0, 0.9, generator=g)
    short, long = [300 + i for i in range(12)], [300] + [4090 - i for i in range(11)]
    calls = []
    real = paged_ops.attention_step
    monkeypatch.setattr(paged_ops, "attention_step", lambda *a: calls.append(1) or real(*a))
    first = []
    for graphs in (False, True):
        r.use_graphs = graphs
        for lens in (short, long, short, long):
            before = len(calls)
            first.append(r.decode(list(range(12)), list(range(12)), lens)[0].clone())
            fresh = not graphs or len(first) <= (5 if many else 6)    # a replay calls nothing; with heads of 64 all share a graph
            assert (len(calls) > before) == (fresh and (lens is short or many)), (graphs, lens)
    assert all(torch.equal(first[0], x) for x in first)


def test_attention_in_one_launch_on_a_tensor_parallel_shard(monkeypatch, cuda_status):
    """A rank's shard (half of the heads, exchanges that return the rank's own part): the decoding step with attention in one launch has the bits of the
    three launches, eager and replayed."""
    from rustral_b200.models.config import GPTConfig
    from rustral_b200.ops import paged as paged_ops
    from rustral_b200.serve.model_runner import ModelRunner

    class Shard:
        world, rank = 2, 1

        def __init__(self):
            self.memory = {}

        def staging(self, rows, cols):
            return self.memory.setdefault((rows, cols), torch.zeros(rows, cols, device="cuda", dtype=torch.bfloat16))

        def all_reduce(self, rows, cols, residual=None):
            return self.staging(rows, cols) + residual

        def all_gather_cols(self, rows, cols):
            return self.staging(rows, cols).clone()

        def end_step(self):
            pass

    cfg = GPTConfig(vocab_size=1024, seq_len=2048, n_layer=2, n_head=16, n_kv_head=8, d_model=1024, ffn_dim=2048, arch="llama")
    lens = [1, 300, 1000]
    got = []
    for one in (True, False):
        if not one:
            monkeypatch.setattr(paged_ops, "step_most_slices", lambda *a: 0)
        r = ModelRunner(cfg, device="cuda", num_blocks=128, block_size=16, seed=3, tp=Shard())
        g = torch.Generator(device="cuda").manual_seed(1)
        for i, n in enumerate(lens):
            assert r.cache.allocate(i, n)
        for l in range(2):
            r.cache.k[l].normal_(0.0, 0.9, generator=g)
            r.cache.v[l].normal_(0.0, 0.9, generator=g)
        assert r.n_kv_head == 4 and r._attends_in_one_launch(lens, 128) == one
        for graphs in (False, True, True):
            r.use_graphs = graphs
            got.append((r.decode([0, 1, 2], [5, 6, 7], lens).clone(), *(c.clone() for c in (*r.cache.k, *r.cache.v))))
    assert torch.isfinite(got[0][0]).all()
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
