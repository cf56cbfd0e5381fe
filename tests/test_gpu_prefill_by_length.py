"""Prompt tiles cut by their own keys in a launch planned for a long context: which tiles are cut, at the line and around it, that each
holds what its kind of launch gives bit for bit, and the result in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PLANNED = 16384


def _key_tiles(pos0, nrows, window, keep):
    first = max(0, pos0 - window + 1) // 64 * 64 if window else 0
    kept = -(-min(keep, first) // 64) if window else 0
    return kept + (pos0 + nrows - 1 - first) // 64 + 1


def _whole(n, parts, n_tiles, nh, d, capped):
    """What a cut saves against what it costs, in ns (the rule the kernel states)."""
    ns = {256: (940, 980), 128: (620, 850), 64: (580, 830)}[d][capped]
    return (n - -(-n // parts)) * ns <= 2200 + 18 * d + 5 * nh * d // 2 - 260 * n_tiles


def _exact(q, k, v, pos, window, keep, sink, cap):
    """Rows q [T, H, d] at positions pos over keys [H, S, d], in 64 bits; also the sum of weight x size, for the bound."""
    s = torch.einsum("thd,hsd->ths", q, k) * q.shape[-1] ** -0.5
    if cap:
        s = cap * torch.tanh(s / cap)
    j = torch.arange(k.shape[1], device=q.device)[None, :]
    seen = j <= pos[:, None]
    if window:
        seen &= (pos[:, None] - j < window) | (j < keep)
    w = s.masked_fill(~seen[:, None], float("-inf"))
    if sink:
        w = torch.cat([w, torch.zeros_like(w[:, :, :1])], -1)
    w = torch.softmax(w, -1)[:, :, :k.shape[1]]
    return torch.einsum("ths,hsd->thd", w, v), torch.einsum("ths,hsd->thd", w, v.abs())


@pytest.mark.parametrize("nh,nkv,d", [(8, 4, 256), (4, 1, 128), (6, 2, 64), (2, 2, 256)])
@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("window,keep,sink,cap", [(None, 0, False, 30.0), (None, 0, False, 0.0), (2000, 70, True, 0.0)])
def test_tiles_cut_by_their_own_keys(nh, nkv, d, few, window, keep, sink, cap):
    from kungfu_b200 import ops
    from test_gpu_kernels import _Ctx, _View, _paged_setup
    n_tiles = 2 if few else 6
    max_keys = min(PLANNED, window + 128 + -(-keep // 64) * 64) if window else PLANNED
    parts = ops.library().kf_attention_prefill_tc_plan(n_tiles, nh, max_keys, ctypes.byref(ctypes.c_int(0)))
    assert parts > 1
    # one tile of 70 to 128 rows for each of: the longest that stays whole and one key tile more; short ones, a long one
    line = max(n for n in range(1, 30) if _whole(n, parts, n_tiles, nh, d, cap > 0))
    ends = [64 * n - 6 for n in ([line, line + 1] if few else [line, line + 1, 2, 3, line + 3, 40])]
    spans = [(max(0, z - 70 - 10 * i), z) for i, z in enumerate(ends)]
    pages, table, ks, vs = _paged_setup(torch.bfloat16, nh, nkv, d, 64, ends, seed=9)
    rows = [(r, p) for r, (a, z) in enumerate(spans) for p in range(a, z)]
    g = torch.Generator().manual_seed(4)
    q = torch.randn(len(rows), nh * d, generator=g).to(torch.bfloat16).to(DEV)
    ctx = _Ctx(torch.tensor([p for _, p in rows], dtype=torch.int32, device=DEV), torch.tensor([r for r, _ in rows], dtype=torch.int32, device=DEV),
               table.to(DEV), dec_rows=[], pre_rows=list(range(len(rows))))
    ctx.max_kv_len = PLANNED
    assert ctx.n_wide == n_tiles
    view = _View(pages.to(DEV), 64)

    def attend(plan=None):
        out = torch.full((len(rows), nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.prefill_plan_override = plan
        try:
            before = ops.launch_count()
            ops.paged_attention(q, out, ctx, view, nh, nkv, d, d ** -0.5, cap, window, keep_first=keep, sink=sink)
            return out, ops.launch_count() - before
        finally:
            ops.prefill_plan_override = None

    (got, launches), (uncut, alone), (cut, _) = attend(), attend((1, 0)), attend((parts, 0))
    ops.raise_on_device_error()
    assert launches == 2 and alone == 1
    kinds, at = [], 0
    for r, (a, z) in enumerate(spans):
        mine = slice(at, at + z - a)
        at += z - a
        kinds.append(_whole(_key_tiles(a, z - a, window, keep), parts, n_tiles, nh, d, cap > 0))
        assert torch.equal(got[mine], (uncut if kinds[-1] else cut)[mine]), (r, z - a, kinds)
        if not kinds[-1]:
            assert not torch.equal(uncut[mine], cut[mine])           # the two kinds can be told apart
        k, v = (x[r].to(DEV).double().transpose(0, 1).repeat_interleave(nh // nkv, 0) for x in (ks, vs))
        y, size = _exact(q[mine].double().view(-1, nh, d), k, v, torch.arange(a, z, device=DEV), window, keep, sink, cap)
        # weights and the result are rounded to bfloat16 (2^-9 of each); scores of 32-bit sums move a weight by less than 2^-10
        err = (got[mine].double().view_as(y) - y).abs()
        assert bool((err <= 2.0 ** -8 * size + 2.0 ** -9 * y.abs() + 1e-6).all()), (r, float((err / size).max()))
    assert set(kinds) == {True, False}
