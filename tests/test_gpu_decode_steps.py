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
