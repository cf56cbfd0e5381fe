"""The 32-bit product on the tensor cores against 64-bit sums and, row for row, against itself beside other rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from kungfu_b200 import ops as o
    return o


def _case(N, K, T, seed=1):
    g = torch.Generator(device=DEV).manual_seed(seed)
    x = torch.randn(T, K, generator=g, device=DEV)
    w = torch.randn(N, K, generator=g, device=DEV) * 0.05
    return x, w


# one, two, four and eight parts of K; features around a tile of 128; a k tail of 4, 8 and 60 and a chunk that ends in its first half;
# rows at the edges of the small tile (16), of the tiles beyond (multiples of 16 up to 80) and of two to five of them
@pytest.mark.parametrize("N,K", [(18433, 228), (8000, 600), (16500, 260), (4095, 1084), (2304, 2052), (1100, 4128), (70000, 64)])
def test_rows_against_64_bits_and_alone(ops, N, K):
    assert ops.library().kf_linear_split_supported(0, 0, N, K)
    x, w = _case(N, K, 330)
    ref = x.double() @ w.double().T
    # each product loses at most 2^-21 of itself (the planes left out); at most K / 8 additions of a row are cut off or rounded
    # by 2^-23 of the sum of the products' sizes, which is also above what K / 64 rounded additions lose
    bound = (2.0 ** -21 + (K / 8 + 4) * 2.0 ** -23) * (x.double().abs() @ w.double().abs().T)
    whole = torch.full((330, N), float("nan"), device=DEV)
    ops.linear(x, w, whole)
    assert bool(((whole - ref).abs() <= bound).all())
    # and on the whole no worse than a chain of rounded 32-bit sums of K / 2 terms, whose error grows as sqrt(K / 2) 2^-25
    assert float((whole - ref).norm() / ref.norm()) <= (K / 2) ** 0.5 * 2.0 ** -25 + 2.0 ** -23
    for T in (1, 15, 16, 17, 32, 33, 79, 80, 81, 160, 161, 321):
        out = torch.full((T + 1, N), float("nan"), device=DEV)
        ops.linear(x[:T], w, out[:T])
        assert torch.equal(out[:T], whole[:T]), T                # a row does not depend on the others, to the bit
        assert bool(out[T].isnan().all()), T
    for T in (16, 40):
        half = torch.empty(T, N, dtype=torch.bfloat16, device=DEV)
        ops.linear(x[:T], w, half, softcap=0.7)
        want = 0.7 * torch.tanh(ref[:T] / 0.7)
        assert bool(((half - want).abs() <= 2.0 ** -8 * want.abs() + bound[:T] + 1e-6).all())
    ops.raise_on_device_error()


@pytest.mark.parametrize("T", [3, 70])
def test_infinities_nan_and_tiny_numbers_as_plain_sums_have_them(ops, T):
    N, K = 2304, 2052
    x, w = _case(N, K, T, 2)
    w = w.bfloat16().float()                                     # lower planes of zeros: an infinity times them would be NaN
    x[1, 7], x[2, 2050] = float("inf"), float("nan")
    x[0] *= 2.0 ** -120
    w[5, 9], w[300] = float("-inf"), w[300] * 2.0 ** -115
    out = torch.empty(T, N, device=DEV)
    ops.linear(x, w, out)
    ref = x.double() @ w.double().T
    assert torch.equal(out.isnan(), ref.isnan()) and torch.equal(out.isinf(), ref.isinf())
    assert torch.equal(out[ref.isinf()].double(), ref[ref.isinf()])
    fin = ref.isfinite()
    bound = (K + 3) * 2.0 ** -23 * (x.nan_to_num(0, 0, 0).double().abs() @ w.nan_to_num(0, 0, 0).double().abs().T) + 2.0 ** -140
    assert bool(((out - ref).abs() <= bound)[fin].all())
    ops.raise_on_device_error()
