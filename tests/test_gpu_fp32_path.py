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


# heads per stored head 1, 3, 2, 16 and 20 (two cuts); head sizes at and beside the element counts of the instances
@pytest.mark.parametrize("nh,nkv,d,P,dtype", [(4, 4, 20, 5, torch.float32), (6, 2, 64, 16, torch.float32), (4, 2, 72, 64, torch.float32),
                                              (16, 1, 130, 7, torch.float32), (20, 1, 128, 32, torch.float32), (8, 4, 256, 64, torch.float32),
                                              (3, 1, 512, 16, torch.float32), (2, 1, 300, 16, torch.bfloat16), (6, 2, 40, 8, torch.bfloat16)])
@pytest.mark.parametrize("window,keep,sink", [(0, 0, False), (40, 0, False), (33, 37, True)])
def test_generic_attention(ops, nh, nkv, d, P, dtype, window, keep, sink):
    """Rows of several requests in one launch, alone, and behind a list of rows: the same bits; against 64 bits; and a key
    that a row does not see does not reach it, whatever its value holds."""
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    lens = [1, 200, 31, 33, 64]
    pages, table, ks, vs = _paged_setup(dtype, nh, nkv, d, P, lens, seed=11)
    rows = [(1, p) for p in range(95, 130)] + [(-1, 0)] + [(2, p) for p in range(31)] + [(3, 32), (0, 0), (4, 63), (3, 31), (1, 199)]
    g = torch.Generator().manual_seed(6)
    q = torch.randn(len(rows), nh * d, generator=g).to(dtype).to(DEV)
    dev_pages, dev_table = pages.to(DEV), table.to(DEV)

    def attend(which, p=dev_pages):
        ctx = _Ctx(torch.tensor([rows[i][1] for i in which], dtype=torch.int32, device=DEV),
                   torch.tensor([rows[i][0] for i in which], dtype=torch.int32, device=DEV), dev_table)
        out = torch.full((len(which), nh * d), float("nan"), dtype=dtype, device=DEV)
        ops.paged_attention(q[which], out, ctx, _View(p, P), nh, nkv, d, d ** -0.5, 30.0, window or None, keep_first=keep, sink=sink)
        return out

    whole = attend(list(range(len(rows))))
    assert float(whole[35].abs().max()) == 0.0                        # the padding row
    for which in ([0], [34, 36], list(range(36, 50)), [71, 3]):
        assert torch.equal(attend(which), whole[which])
    for i, (r, p) in enumerate(rows):
        if r < 0:
            continue
        see = torch.tensor([j for j in range(p + 1) if not window or p - j < window or j < keep])
        kd, vd = ks[r][see].double(), vs[r][see].double()
        kd, vd = kd.repeat_interleave(nh // nkv, 1), vd.repeat_interleave(nh // nkv, 1)
        s = torch.einsum("jhd,hd->hj", kd, q[i].cpu().double().view(nh, d)) * d ** -0.5
        s = 30.0 * torch.tanh(s / 30.0)
        e = torch.exp(s - s.amax(1, keepdim=True))
        w = e / (e.sum(1, keepdim=True) + (torch.exp(-s.amax(1, keepdim=True)) if sink else 0.0))
        want = torch.einsum("hj,jhd->hd", w, vd)
        err = (whole[i].cpu().double().view(nh, d) - want).abs().max()
        # scores of size <= 30 err by (d + 4) 2^-24 of |q| |k| scale <= 8 sqrt(d) each; the weights by as much, relatively
        bound = (d + 40) * 2.0 ** -24 * 8 * d ** 0.5 * vd.abs().max() + (2.0 ** -8 * want.abs().max() if dtype == torch.bfloat16 else 0)
        assert float(err) <= float(bound), (i, float(err), float(bound))
    # request 1, position 120: rows 0..24 (positions 95..119) must not see it
    poisoned = pages.clone()
    poisoned[table[1, 120 // P], 1, :, 120 % P] = float("inf")
    got = attend(list(range(len(rows))), poisoned.to(DEV))
    assert torch.equal(got[:25], whole[:25]) and not bool(got[25].isfinite().all())


def test_a_seen_key_counts_the_same_beside_any_other_rows(ops):
    """A key that a row sees with a weight below the smallest number, and whose value is infinite: the row holds what it holds
    alone, also where its block walks rows that do not see the key."""
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    nh, d, P = 16, 32, 16
    pages, table, _, _ = _paged_setup(torch.float32, nh, nh, d, P, [41], seed=3)
    pages[table[0, 0], 0, :, 5] = -30.0                               # q is all ones: a score of -170 at position 5
    pages[table[0, 0], 1, :, 5, 3] = float("inf")
    dev_pages, dev_table = pages.to(DEV), table.to(DEV)
    places = [40 if i % 2 else 4 for i in range(200)]                 # enough rows for blocks of several

    def attend(at):
        ctx = _Ctx(torch.tensor(at, dtype=torch.int32, device=DEV), torch.zeros(len(at), dtype=torch.int32, device=DEV), dev_table)
        out = torch.empty(len(at), nh * d, device=DEV)
        ops.paged_attention(torch.ones(len(at), nh * d, device=DEV), out, ctx, _View(dev_pages, P), nh, nh, d, d ** -0.5, 0.0, None)
        return out.view(len(at), nh, d)

    low, high = attend([4])[0], attend([40])[0]
    assert bool(low.isfinite().all()) and not bool(high[:, 3].isfinite().any()) and bool(high[:, 4:].isfinite().all())
    together = attend(places)
    for i, p in enumerate(places):
        assert torch.equal(together[i].nan_to_num(7.0), (high if p == 40 else low).nan_to_num(7.0)), i
