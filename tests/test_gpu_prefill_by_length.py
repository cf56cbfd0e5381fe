"""Prompt tiles cut by their own keys in a launch planned for a long context: tiles that stay whole beside tiles cut in as many runs
as they are worth, against the same launch uncut."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# Key tiles of 64: 1 to 4 and 11 (whole), 12 and 13 (cut), 21, 47.  A cut into p runs of n key tiles is taken when ceil(n / p) + 9 < n: runs of one
# key tile need n <= 8 and never pay, runs of two or more cost at least 11, so up to 11 key tiles stay whole and 12 in six runs do not.
@pytest.mark.parametrize("nh,nkv,d", [(8, 4, 256), (4, 1, 128), (6, 2, 64)])
@pytest.mark.parametrize("spans", [[(0, 200), (2900, 3000)], [(640, 704)], [(700, 768)], [(700, 832)], [(1200, 1281), (0, 2)]])
@pytest.mark.parametrize("window,keep,sink", [(None, 0, False), (900, 70, True)])
def test_tiles_cut_by_their_own_keys(nh, nkv, d, spans, window, keep, sink):
    from kungfu_b200 import ops
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    pages, table, _, _ = _paged_setup(torch.bfloat16, nh, nkv, d, 64, [z for _, z in spans], seed=9)
    rows = [(r, p) for r, (a, z) in enumerate(spans) for p in range(a, z)]
    g = torch.Generator().manual_seed(4)
    q = torch.randn(len(rows), nh * d, generator=g).to(torch.bfloat16).to(DEV)
    ctx = _Ctx(torch.tensor([p for _, p in rows], dtype=torch.int32, device=DEV), torch.tensor([r for r, _ in rows], dtype=torch.int32, device=DEV),
               table.to(DEV), dec_rows=[], pre_rows=list(range(len(rows))))
    ctx.max_kv_len = 16384
    view = _View(pages.to(DEV), 64)

    def attend():
        out = torch.full((len(rows), nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.paged_attention(q, out, ctx, view, nh, nkv, d, d ** -0.5, 30.0, window, keep_first=keep, sink=sink)
        return out.float()

    cut = attend()
    ops.prefill_plan_override = (1, 0)
    try:
        whole = attend()
    finally:
        ops.prefill_plan_override = None
    # P is rounded to bfloat16 against another maximum (2^-9 of the weighted sizes, which are those of the values) and the result once
    assert float((cut - whole).abs().max()) <= 2.0 ** -7 * float(pages[:, 1].float().abs().max())
    assert float((cut - whole).norm() / whole.norm()) <= 2.0 ** -7
    few = [i for i, (r, p) in enumerate(rows) if spans[r][1] <= 704 and window is None]
    assert torch.equal(cut[few], whole[few])                       # up to eleven key tiles: not cut
