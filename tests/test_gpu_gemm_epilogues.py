"""Results of the tile products that leave through shared-memory tiles and TMA, where a CTA writes several tiles one after another."""
import pytest
import torch

from rustral_b200.ops.matmul import gemm

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(s, device="cuda", generator=g).bfloat16() for s in ((M, K), (N, K))]


@pytest.mark.parametrize("block_n", [64, 128, 192, 256])
@pytest.mark.parametrize("M,N", [(5011, 1992), (128 * 74, 2048)])
def test_a_tile_that_is_still_being_stored_is_not_written_again(M, N, block_n, cuda_status):
    """Short contractions and several tiles per CTA: epilogues run back to back, each into result tiles that the one before may still be
    reading out.  128-wide products have one block of 64 columns per warp, so the two tiles have to alternate from output tile to output tile."""
    a, b = _operands(M, N, 64, M)
    want = a.double() @ b.double().T
    bound = 2.0 ** -8 * want.abs() + 64 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T) + 1e-30
    first = gemm(a, b, block_n=block_n)
    assert ((first.double() - want).abs() <= bound).all()
    for _ in range(20):
        assert torch.equal(gemm(a, b, block_n=block_n), first)


def _gelu(x):
    return torch.nn.functional.gelu(x, approximate="tanh")


def _gelu_grad(x):
    x = x.clone().requires_grad_()
    return torch.autograd.grad(_gelu(x).sum(), x)[0]


# what the epilogue reads and writes besides the product; "relu" and "mul" keep the bound at the rounding of the result
FORMS = ("residual", "in place", "mul", "mul + residual", "dgelu + residual", "relu + pre", "relu + pre + residual", "gelu + pre",
         "gelu + pre + residual")


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("block_n,M,N", [(256, 2500, 3016), (256, 100, 38000), (128, 2500, 3016), (192, 300, 392), (64, 300, 200)])
def test_side_inputs_and_second_results(block_n, M, N, form, cuda_status):
    """Several output tiles per CTA, no multiple of a tile; 256-wide products run on the two-CTA kernel with many rows and on the one-CTA
    kernel with one tile per warp with few.  Each form against 64-bit arithmetic, element by element."""
    a, b = _operands(M, N, 72, N)
    g = torch.Generator(device="cuda").manual_seed(M)
    res, aux = (torch.randn(M, N, device="cuda", generator=g).bfloat16() for _ in range(2))
    bias = torch.randn(N, device="cuda", generator=g).bfloat16()
    kw = dict(block_n=block_n, group_m=8)                    # a plan of the tile kernels for few rows too
    pre = a.double() @ b.double().T
    sums = 72 * 2.0 ** -24 * (a.double().abs() @ b.double().abs().T) + 1e-30
    if "pre" in form:
        pre = pre + bias.double()
        act = form.split()[0]
        kept = torch.empty(M, N, device="cuda", dtype=torch.bfloat16)
        got = gemm(a, b, bias=bias, act=act, aux_out=kept, residual=res if "residual" in form else None, **kw)
        # one rounding to bf16; the result from the rounded pre-activation or from the unrounded one (slopes of at most 1.13), then a
        # rounding of its own; tanh.approx is 5e-4 off, relative
        assert ((kept.double() - pre).abs() <= 2.0 ** -8 * pre.abs() + sums).all()
        want = torch.relu(pre) if act == "relu" else _gelu(pre)
        slack = 1.13 * (2.0 ** -8 * pre.abs() + sums) + (0.0 if act == "relu" else 5e-4) * pre.abs()
        if "residual" in form:
            want = want + res.double()
    elif form == "in place":
        got = res.clone()
        assert gemm(a, b, residual=got, out=got, **kw) is got
        want, slack = pre + res.double(), sums
    else:
        act = form.split()[0]
        kind = act if act in ("mul", "dgelu") else "none"
        got = gemm(a, b, act=kind, aux_in=aux if kind != "none" else None, residual=res if "residual" in form else None, **kw)
        f = {"mul": aux.double(), "dgelu": _gelu_grad(aux.double()), "none": 1.0}[kind]
        want = pre * f + (res.double() if "residual" in form else 0.0)
        # tanh.approx and what the gradient makes of it: 1e-3 of the product and an absolute 1e-3 where the gradient crosses zero
        slack = sums * 1.13 + (2e-3 * (pre.abs() + 0.1) if kind == "dgelu" else 1.2e-7 * pre.abs() + sums * aux.double().abs())
    bound = 2.0 ** -8 * (want.abs() + slack) + slack
    assert ((got.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("block_n", [64, 128, 192, 256])
@pytest.mark.parametrize("M,N,K", [(700, 260, 64), (96, 3000, 64)])
def test_accumulation_keeps_subnormal_sums(M, N, K, block_n, cuda_status):
    """d += a b^T in fp32: an entry that nothing is added to keeps its bits, and sums below the smallest normal number are not flushed,
    whichever unit adds them (registers or the TMA reduction)."""
    d = torch.full((M, N), 1e-40, device="cuda")
    d[::3] = 1.5e-38
    a, b = torch.zeros(M, K, device="cuda").bfloat16(), torch.zeros(N, K, device="cuda").bfloat16()
    a[:, 3], b[::2, 3] = 2.0 ** -70, -(2.0 ** -57)           # a product of -2^-127 (5.9e-39, itself subnormal) in every second column
    want = d.double()
    want[:, ::2] -= 2.0 ** -127
    out = gemm(a, b, out=d.clone(), accumulate=True, block_n=block_n, group_m=8)
    assert torch.equal(out[:, 1::2], d[:, 1::2])
    # the tensor core may flush the subnormal product, the addition may not flush its result
    flushed = torch.equal(out, d)
    assert flushed or torch.equal(out.double(), want)
    a[:, 3] = 2.0 ** -68                                     # -2^-125, a normal number; 1.5e-38 - 2^-125 = -8.5e-39 is not
    want = d.double()
    want[:, ::2] -= 2.0 ** -125
    assert torch.equal(gemm(a, b, out=d.clone(), accumulate=True, block_n=block_n, group_m=8).double(), want.float().double())


@pytest.mark.parametrize("rows,N", [(200, 264), (97, 96)])
def test_expert_weight_gradients_in_16_bits(rows, N, cuda_status):
    """Grouped weight gradients whose results are stacked below one another (whole 32-row tiles) and where they are not; an expert without
    tokens gets zeros."""
    from rustral_b200.ops import moe
    E, K, T = 6, 136, 1500
    g = torch.Generator(device="cuda").manual_seed(rows)
    idx = torch.randint(0, E - 1, (T, 1), device="cuda", generator=g, dtype=torch.int32)      # the last expert has none
    pl = moe.plan(idx, E)
    x, dy = (torch.randn(T, n, device="cuda", generator=g).bfloat16() for n in (K, N))
    xp, dyp = moe.gather(x, pl), moe.gather(dy, pl)
    fill = torch.full((E, N, K), float("nan"), device="cuda").bfloat16()
    for out in (moe.grouped_wgrad(dyp, xp, pl, dtype=torch.bfloat16), moe.grouped_wgrad(dyp, xp, pl, out=fill)):
        for e in range(E):
            m = idx[:, 0] == e
            want = dy[m].double().T @ x[m].double()
            bound = 2.0 ** -8 * want.abs() + 2048 * 2.0 ** -24 * (dy[m].double().abs().T @ x[m].double().abs()) + 1e-30
            assert ((out[e].double() - want).abs() <= bound).all(), e


@pytest.mark.parametrize("N", [800, 808])
@pytest.mark.parametrize("form", ["bf16", "fp32", "fp32 added", "bf16 added"])
def test_expert_weight_gradients_in_wide_tiles(N, form, cuda_status):
    """256-wide tiles: on CTA pairs where the experts' results are stacked in whole 32-row tiles (800 rows, the last pair with a tile and a
    half of nothing), on single CTAs where they are not; experts with few rows, one k-block's worth and none."""
    from rustral_b200.ops import moe
    E, K = 6, 760
    counts = (1, 64, 65, 700, 0, 333)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).int()
    g = torch.Generator(device="cuda").manual_seed(N)
    idx = idx[torch.randperm(len(idx), generator=torch.Generator().manual_seed(1))].cuda()[:, None].contiguous()
    pl = moe.plan(idx, E)
    x, dy = (torch.randn(idx.shape[0], n, device="cuda", generator=g).bfloat16() for n in (K, N))
    xp, dyp = moe.gather(x, pl), moe.gather(dy, pl)
    dtype = torch.float32 if form.startswith("fp32") else torch.bfloat16
    base = torch.randn(E, N, K, device="cuda", generator=g).to(dtype)
    out = moe.grouped_wgrad(dyp, xp, pl, out=base.clone(), accumulate=True) if form.endswith("added") else moe.grouped_wgrad(dyp, xp, pl, dtype=dtype)
    for e in range(E):
        m = idx[:, 0] == e
        want = dy[m].double().T @ x[m].double() + (base[e].double() if form.endswith("added") else 0)
        size = dy[m].double().abs().T @ x[m].double().abs() + base[e].double().abs()
        # sums of at most 701 terms in 32 bits, any order; a result of 16 bits rounded once
        bound = 1024 * 2.0 ** -24 * size + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0) + 1e-30
        assert ((out[e].double() - want).abs() <= bound).all(), (e, counts[e])
