"""Decode attention in blocks of four warps planned for more keys than there are: rows taken by their rank in length (as many as fill one
block on every SM, up to twice as many, more, and rows of equal length), three parts a pair, rows of no request between the others."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

RAGGED = [1100, 1, 15, 16, 17, 128, 129, 500, 33, 700]


# heads of 256 (148 and 296 blocks on the GPU): 64 rows of 4 heads, 78 of them (more than two a block of every SM), 20 rows in three parts;
# heads of 128 and 16; one head of keys (as many rows ranked as SMs), and few rows, which stay in blocks of eight warps
@pytest.mark.parametrize("nh,nkv,d,lens,most", [(8, 4, 256, [40 + 13 * i for i in range(50)] + [77] * 4, 1900), (8, 4, 256, RAGGED * 7, 1100), (8, 4, 256, RAGGED + [900] * 8, 3000),
                                                (16, 4, 128, [5 + (i * 97) % 600 for i in range(90)], 900), (4, 4, 16, [5, 300] * 130, 2000),
                                                (4, 1, 256, [(i * 31) % 250 + 1 for i in range(200)], 700), (16, 4, 128, RAGGED, 1100)])
@pytest.mark.parametrize("window,keep,sink,sig", [(None, 0, False, False), (200, 21, True, False), (None, 0, False, True)])
def test_rows_of_unequal_length(nh, nkv, d, lens, most, window, keep, sink, sig):
    from kungfu_b200 import ops
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    pages, table, ks, vs = _paged_setup(torch.bfloat16, nh, nkv, d, 64, lens, seed=len(lens))
    reqs = [-1] + [r for i in range(len(lens)) for r in ([i, -1] if i % 4 == 2 else [i])] + [-1]
    g = torch.Generator().manual_seed(3)
    q = torch.randn(len(reqs), nh * d, generator=g).to(torch.bfloat16)
    bias = torch.randn(nh, generator=g)
    ctx = _Ctx(torch.tensor([lens[r] - 1 if r >= 0 else 7 for r in reqs], dtype=torch.int32, device=DEV),
               torch.tensor(reqs, dtype=torch.int32, device=DEV), table.to(DEV), dec_rows=list(range(len(reqs))))
    ctx.max_kv_len = most                                            # what the launch is planned for, as in a replayed step
    view, dev_q = _View(pages.to(DEV), 64), q.to(DEV)
    got = []
    for _ in range(2):                                               # the counters are left at zero
        out = torch.full((len(reqs), nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.paged_attention(dev_q, out, ctx, view, nh, nkv, d, d ** -0.5, 30.0, window, keep_first=keep, sink=sink,
                            sigmoid_bias=bias.to(DEV) if sig else None)
        got.append(out)
    assert torch.equal(got[0], got[1])                               # whatever block merges a pair's parts
    rows = range(len(reqs)) if len(reqs) < 40 else list(range(0, len(reqs), 5)) + [1, 2, 3]
    for i in rows:
        r = reqs[i]
        if r < 0:
            assert float(got[0][i].abs().max()) == 0.0
            continue
        p = lens[r] - 1
        see = torch.tensor([j for j in range(p + 1) if window is None or p - j < window or j < keep])
        k, v = ks[r][see].double().repeat_interleave(nh // nkv, 1), vs[r][see].double().repeat_interleave(nh // nkv, 1)
        s = torch.einsum("jhd,hd->hj", k, q[i].double().view(nh, d)) * d ** -0.5
        s = 30.0 * torch.tanh(s / 30.0)
        if sig:
            w = torch.sigmoid(s + bias.double()[:, None])
        else:
            e = torch.exp(s - s.amax(1, keepdim=True))
            w = e / (e.sum(1, keepdim=True) + (torch.exp(-s.amax(1, keepdim=True)) if sink else 0.0))
        want = torch.einsum("hj,jhd->hd", w, v)
        # weights rounded to bfloat16 (2^-9 each, on the weighted sizes), the result too
        bound = 2.0 ** -8 * torch.einsum("hj,jhd->hd", w, v.abs()) + 2.0 ** -8 * want.abs() + 1e-4
        assert bool(((got[0][i].cpu().double().view(nh, d) - want).abs() <= bound).all()), i
