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
