"""Short convolutions across requests, blocks of rows and tap counts; the gated group norm in whole vectors and beside them."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# requests that start and end inside a block of rows, shorter than the taps, of one row, none; padding rows; channels of whole
# vectors and not; every count of rows per block (below 64 rows, below 1,024, above)
@pytest.mark.parametrize("C", [8, 10, 1028])
@pytest.mark.parametrize("taps", [1, 2, 4, 8])
@pytest.mark.parametrize("rows", [(1, 1, 1), (5, 0, 2, 9), (70, 3, 1, 17), (1030, 6)])
@pytest.mark.parametrize("bias", [False, True])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
def test_short_conv(C, taps, rows, bias, wdtype):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(C + taps + len(rows))
    T, ld, col0 = sum(rows) + 2, C + 8, 4
    x, w = torch.randn(T, ld, generator=g), torch.randn(C, taps, generator=g)
    ib, ob = (torch.randn(C, generator=g), torch.randn(C, generator=g)) if bias else (None, None)
    w, ib, ob = (None if t is None else t.to(wdtype) for t in (w, ib, ob))
    state = torch.randn(6, max(taps - 1, 1), C, generator=g)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    starts, slots, req = [sum(rows[:i]) for i in range(len(rows))], [4, 0, 2, 5][:len(rows)], []
    for r, n in enumerate(rows):
        req += [r] * n
    st = types.SimpleNamespace(row_req=ints(req + [-1, -1]), req_row_start=ints(starts), req_state_slot=ints(slots), req_n_rows=ints(rows), n_reqs=len(rows))
    out = torch.full((T, C), 5.0, device=DEV)
    dev = state.to(DEV)
    up = lambda t: None if t is None else t.to(DEV)
    single = max(rows) == 1
    done = ops.short_conv(x.to(DEV), col0, up(ib), w.to(DEV), up(ob), "silu", dev, out, st, commit_inline=single)
    assert done == (single and taps > 1)
    for r, n in enumerate(rows):
        past = state[slots[r]][:taps - 1].double()
        u = torch.cat([past, x[starts[r]:starts[r] + n, col0:col0 + C].double() + (ib.double() if bias else 0.0)])
        for i in range(n):
            y = (u[i:i + taps] * w.double().T).sum(0) + (ob.double() if bias else 0.0)
            size = (u[i:i + taps] * w.double().T).abs().sum(0) + (ob.abs().double() if bias else 0.0)
            # taps + 2 roundings of what is added; the slope of x sigmoid(x) is at most 1.1; a few roundings of the result
            assert bool(((out[starts[r] + i].cpu().double() - y * torch.sigmoid(y)).abs() <= 1.1 * (taps + 2) * 2.0 ** -24 * size + 8 * 2.0 ** -24 * y.abs() + 1e-30).all())
        if done:
            assert torch.equal(dev[slots[r]][:taps - 2].cpu(), state[slots[r]][1:taps - 1])
            assert bool(((dev[slots[r]][taps - 2].cpu().double() - u[-1]).abs() <= 2.0 ** -24 * u[-1].abs()).all())
    assert float(out[-2:].min()) == 5.0 and torch.equal(dev[[1, 3]].cpu(), state[[1, 3]])


@pytest.mark.parametrize("T,inner,parts,z0", [(3, 4096, 1, 4), (300, 4096, 2, 0), (2, 12, 1, 4), (5, 24, 3, 8), (3, 60, 4, 2), (2, 16384, 1, 0), (256, 200, 1, 0)])
@pytest.mark.parametrize("wd,od", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_gated_group_norm(T, inner, parts, z0, wd, od):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(inner + T)
    y, z = torch.randn(T, inner, generator=g), 2.0 * torch.randn(T, inner + 12, generator=g)
    w = torch.randn(inner, generator=g).to(wd)
    st = types.SimpleNamespace(row_req=torch.tensor([0] * (T - 1) + [-1], dtype=torch.int32, device=DEV))
    out = torch.full((T, inner), 5.0, dtype=od, device=DEV)
    ops.gated_group_norm(y.to(DEV), z.to(DEV), z0, w.to(DEV), 1e-5, parts, out, st)
    zz = z[:, z0:z0 + inner].double()
    v = (y.double() * zz * torch.sigmoid(zz)).view(T, parts, -1)
    want = ((v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + 1e-5)).view(T, inner) * w.double())[:-1]
    unit = 2.0 ** -8 if od == torch.bfloat16 else 2.0 ** -24
    # exponential, quotient, products, the mean square's tree of at most 30 levels and its root: under 60 roundings
    assert bool(((out[:-1].cpu().double() - want).abs() <= (unit + 60 * 2.0 ** -24) * want.abs() + 1e-30).all())
    assert float(out[-1].float().abs().max()) == 0.0
