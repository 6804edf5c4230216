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
