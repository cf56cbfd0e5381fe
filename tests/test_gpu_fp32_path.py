"""The kernels of the 32-bit path against 64-bit sums, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from kungfu_b200 import ops as o
    return o


# one row more and one less than every row tile (1, 2, 4, 8, 16, 32, 64); features and k around a tile of 128 and of 32;
# k that is no multiple of four (4-byte copies), shorter than a tile, and cut in two, four and eight parts, the last one short
@pytest.mark.parametrize("N,K", [(1, 1), (127, 31), (128, 32), (129, 33), (300, 514), (2304, 2052), (3000, 1031), (17000, 600)])
def test_product_of_32_bit_operands(ops, N, K):
    g = torch.Generator().manual_seed(N + K)
    x = torch.randn(130, K, generator=g).to(DEV)
    w = (torch.randn(N, K, generator=g) * 0.05).to(DEV)
    ref = x.double() @ w.double().T
    # every product and every sum of a chain rounds once: K + 3 terms of 2^-24, on the sum of the products' sizes
    bound = (K + 3) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 1e-30
    whole = torch.full((130, N), float("nan"), device=DEV)
    ops.linear(x, w, whole)
    assert bool(((whole - ref).abs() <= bound).all())
    for T in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65):
        out = torch.full((T + 1, N), float("nan"), device=DEV)
        ops.linear(x[:T], w, out[:T])
        assert torch.equal(out[:T], whole[:T]), T              # a row does not depend on the others, to the bit
        assert bool(out[T].isnan().all()), T                   # and nothing is written behind the last
    half = torch.empty(65, N, dtype=torch.bfloat16, device=DEV)
    ops.linear(x[:65], w, half, softcap=0.7)
    want = 0.7 * torch.tanh(ref[:65] / 0.7)
    assert bool(((half - want).abs() <= 2.0 ** -8 * want.abs() + bound[:65] + 1e-6).all())


def test_product_of_a_column_range_and_unaligned_bases(ops):
    """x as a column range of a wider matrix, at offsets that allow 16-byte copies and ones that do not."""
    g = torch.Generator().manual_seed(5)
    base = torch.randn(37, 400, generator=g).to(DEV)
    buf = torch.randn(200 * 96 + 1, generator=g).to(DEV)
    for col0, w in ((0, buf[:-1].view(200, 96)), (64, buf[:-1].view(200, 96)), (3, buf[:-1].view(200, 96)), (64, buf[1:].view(200, 96))):
        x = base[:, col0:col0 + 96]
        ref = x.double() @ w.double().T
        out = torch.empty(37, 200, device=DEV)
        ops.linear_cols(base, col0, w, out)
        bound = 99 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
        assert bool(((out - ref).abs() <= bound).all()), col0
