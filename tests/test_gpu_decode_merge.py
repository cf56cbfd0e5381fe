"""Decode attention whose keys are cut into many splits: the merge through shared memory, and the one for more records than it holds."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# splits: min(64, keys / 256, SMs x blocks / pairs); 20 splits of 2 and of 16 heads of 256 (the latter do not fit), 9, 8 and 40
@pytest.mark.parametrize("nh,nkv,d,n", [(2, 1, 256, 5000), (16, 1, 256, 5000), (4, 2, 256, 2100), (4, 2, 128, 2048), (8, 1, 64, 10200), (3, 1, 16, 4000)])
@pytest.mark.parametrize("sink", [False, True])
def test_many_splits(nh, nkv, d, n, sink):
    from kungfu_b200 import ops
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    pages, table, ks, vs = _paged_setup(torch.bfloat16, nh, nkv, d, 64, [n], seed=n)
    g = torch.Generator().manual_seed(3)
    q = torch.randn(1, nh * d, generator=g).to(torch.bfloat16)
    ctx = _Ctx(torch.tensor([n - 1], dtype=torch.int32, device=DEV), torch.tensor([0], dtype=torch.int32, device=DEV), table.to(DEV), dec_rows=[0])
    out = torch.empty(1, nh * d, dtype=torch.bfloat16, device=DEV)
    for _ in range(2):                                               # the counters are left at zero
        ops.paged_attention(q.to(DEV), out, ctx, _View(pages.to(DEV), 64), nh, nkv, d, 2 * d ** -0.5, 0.0, None, sink=sink)
    s = torch.einsum("jhd,hd->hj", ks[0].double().repeat_interleave(nh // nkv, 1), q.double().view(nh, d)) * 2 * d ** -0.5
    e = torch.exp(s - s.amax(1, keepdim=True))
    w = e / (e.sum(1, keepdim=True) + (torch.exp(-s.amax(1, keepdim=True)) if sink else 0.0))
    v = vs[0].double().repeat_interleave(nh // nkv, 1)
    want = torch.einsum("hj,jhd->hd", w, v)
    # weights rounded to bfloat16 (2^-9 each, on the weighted sizes), the result too
    bound = 2.0 ** -8 * torch.einsum("hj,jhd->hd", w, v.abs()) + 2.0 ** -8 * want.abs() + 1e-4
    assert bool(((out.cpu().double().view(nh, d) - want).abs() <= bound).all())


# more (row, kv head) pairs than SMs hold blocks with at most 512 keys: blocks of four warps; one key, a tile more and less, 512;
# a window, kept first tokens and the sink; and at 513 keys the blocks of eight warps again
@pytest.mark.parametrize("nh,nkv,d,B,most", [(8, 4, 256, 80, 512), (16, 8, 128, 90, 300), (8, 4, 256, 80, 513), (6, 3, 64, 500, 70), (4, 4, 16, 700, 40)])
@pytest.mark.parametrize("window,keep,sink", [(None, 0, False), (33, 5, True)])
def test_many_short_rows(nh, nkv, d, B, most, window, keep, sink):
    from kungfu_b200 import ops
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    lens = [min(n, most) for n in [most, 1, 15, 16, 17, 64, 65] + [1 + (i * 37) % most for i in range(B - 7)]]
    pages, table, ks, vs = _paged_setup(torch.bfloat16, nh, nkv, d, 64, lens, seed=B)
    g = torch.Generator().manual_seed(3)
    q = torch.randn(B, nh * d, generator=g).to(torch.bfloat16)
    ctx = _Ctx(torch.tensor([n - 1 for n in lens], dtype=torch.int32, device=DEV), torch.arange(B, dtype=torch.int32, device=DEV), table.to(DEV),
               dec_rows=list(range(B)))
    out = torch.empty(B, nh * d, dtype=torch.bfloat16, device=DEV)
    ops.paged_attention(q.to(DEV), out, ctx, _View(pages.to(DEV), 64), nh, nkv, d, d ** -0.5, 30.0, window, keep_first=keep, sink=sink)
    for r in list(range(12)) + [B - 1]:
        p = lens[r] - 1
        see = torch.tensor([j for j in range(p + 1) if window is None or p - j < window or j < keep])
        k, v = ks[r][see].double().repeat_interleave(nh // nkv, 1), vs[r][see].double().repeat_interleave(nh // nkv, 1)
        s = torch.einsum("jhd,hd->hj", k, q[r].double().view(nh, d)) * d ** -0.5
        s = 30.0 * torch.tanh(s / 30.0)
        e = torch.exp(s - s.amax(1, keepdim=True))
        w = e / (e.sum(1, keepdim=True) + (torch.exp(-s.amax(1, keepdim=True)) if sink else 0.0))
        want = torch.einsum("hj,jhd->hd", w, v)
        # weights rounded to bfloat16 (2^-9 each, on the weighted sizes), the result too
        bound = 2.0 ** -8 * torch.einsum("hj,jhd->hd", w, v.abs()) + 2.0 ** -8 * want.abs() + 1e-4
        assert bool(((out[r].cpu().double().view(nh, d) - want).abs() <= bound).all()), r
