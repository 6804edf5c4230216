"""The product kernel for few rows (gemm_rows.cu) at the edges of its tiles, parts and rule, against 64-bit arithmetic and the tile kernel."""
import pytest
import torch

from rustral_b200.ops.matmul import gemm

pytestmark = pytest.mark.gpu

# (N, K): one tile and less, ragged columns, a last K block of 8, one block only, parts of unequal length, more tiles than SMs
SIZES = [(8, 64), (128, 8), (130, 72), (520, 200), (768, 768), (1000, 1016), (2048, 8192), (19200, 136)]


def _operands(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    ld = (K + 15) // 8 * 8                                             # rows that do not follow each other
    return rnd(M, ld)[:, :K], rnd(N, ld)[:, :K], rnd(N), rnd(M, (N + 15) // 8 * 8)[:, :N]


@pytest.mark.parametrize("M", [1, 15, 16, 17, 48, 49, 96, 97])
@pytest.mark.parametrize("N,K", SIZES)
def test_matches_64_bit_and_the_tile_kernel(M, N, K, cuda_status):
    x, w, bias, res = _operands(M, N, K)
    ref = x.double() @ w.double().T
    # fp32 sums of K products in any order: K * 2^-24 of the sum of magnitudes
    bound = K * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-6
    y = torch.empty(M, (N + 7) // 4 * 4, device="cuda")[:, :N]
    gemm(x, w, out=y)
    assert ((y.double() - ref).abs() <= bound).all()
    assert ((gemm(x, w, out=torch.empty_like(y, memory_format=torch.preserve_format), group_m=8).double() - ref).abs() <= bound).all()
    if N % 8 == 0:
        for act, f in (("none", lambda t: t), ("relu2", lambda t: torch.relu(t) ** 2), ("silu", torch.nn.functional.silu),
                       ("gelu", lambda t: torch.nn.functional.gelu(t, approximate="tanh"))):
            got = gemm(x, w, bias=bias, act=act, residual=res, alpha=0.5)
            want = f(0.5 * ref + bias.double()) + res.double()
            # bf16 result (2^-8), fp32 sums, tanh.approx of gelu (5e-4 relative)
            assert ((got.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-3 * (want - res.double()).abs() + 1e-2 * bound + 1e-3).all(), act
            assert torch.equal(got, gemm(x, w, bias=bias, act=act, residual=res, alpha=0.5))


def test_residual_in_place_and_graph_replay(cuda_status):
    """The result may replace the residual; a captured chain of dependent products gives what the eager one gives."""
    x, w, _, _ = _operands(5, 256, 256)
    w = (w.float() * 0.05).bfloat16()

    def chain(t, r):
        for _ in range(6):
            gemm(t, w, residual=r, out=r)
            t = gemm(r, w, act="relu")
        return t

    r0 = x.flip(0).contiguous()
    want = chain(x, r0.clone())
    r = r0.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(x, r)
    r.copy_(r0)
    graph.replay()
    assert torch.equal(got, want)


@pytest.mark.parametrize("M", [1, 17, 96, 97, 129, 300, 513])
@pytest.mark.parametrize("F,K", [(8, 64), (64, 72), (72, 768), (200, 2048), (1000, 264), (2504, 72), (3200, 2048)])
def test_swiglu_product(M, F, K, cuda_status):
    """Gates and ups of one result column come from two places of the weight: edges of 64- and 128-column tiles, rows of both kernels and of
    neither, with more than 128 rows few tiles (two launches) and many, and a weight whose rows behind the gates are the ups (a tile that ends in the middle reads into them)."""
    from rustral_b200.ops.rotary import swiglu_product
    x, w, _, _ = _operands(M, 2 * F, K)
    w = (w.float() * K ** -0.5).bfloat16()
    g, u = (x.double() @ w.double().T).split(F, -1)
    want = torch.nn.functional.silu(g) * u
    got = swiglu_product(x, w)
    # bf16 result (2^-8); where the two products are rounded first: 2^-8 of each, the gate's through silu's slope (at most 1.1)
    bound = 2.0 ** -7 * want.abs() + 2.0 ** -7 * 1.1 * (g * u).abs() + 1e-5
    assert ((got.double() - want).abs() <= bound).all()
    assert torch.equal(got, swiglu_product(x, w, b_constant=True))


def test_swiglu_product_refuses_weights_that_are_no_gates_and_ups(cuda_status):
    from rustral_b200.ops.rotary import swiglu_product
    x, w, _, _ = _operands(5, 34, 64)
    for a, b in ((x, w[:33]), (x.cpu(), w[:33].cpu()), (x, w.cpu()), (x, w[:, :56])):
        with pytest.raises(ValueError):
            swiglu_product(a, b)
