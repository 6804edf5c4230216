"""Decoding kernels at the edges of their work splits: slices of the cached tokens."""
import pytest
import torch

from rustral_b200.ops import paged

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,heads,kv,dim,longest,width", [(1, 8, 2, 128, 2500, 400), (64, 8, 4, 128, 1300, 1024), (120, 32, 16, 64, 700, 64),
                                                             (3, 4, 4, 64, 257, 1024)])
def test_slices_of_the_context(batch, heads, kv, dim, longest, width, cuda_status):
    """Slices of 256 tokens, of more (many sequences), and one slice for everything; lengths from 1 to the longest."""
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
