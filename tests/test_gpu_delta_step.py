"""The delta rule's kernel for steps of single rows gives the bits of the walk."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# key sizes of every instance and beside its edge, value columns around a block's 32, shared key heads
@pytest.mark.parametrize("H,KH,d,dv", [(2, 1, 16, 24), (3, 3, 33, 31), (4, 2, 64, 33), (2, 2, 65, 64), (4, 2, 128, 128), (2, 1, 129, 20), (1, 1, 256, 70)])
@pytest.mark.parametrize("per_channel", [False, True])
@pytest.mark.parametrize("wdtype", [torch.float32, torch.bfloat16])
def test_single_rows_as_the_walk(H, KH, d, dv, per_channel, wdtype):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(H * 1000 + d)
    C, na = 2 * KH * d + H * dv, H * d if per_channel else H
    x, beta, dec = torch.randn(4, C + 5, generator=g), torch.randn(4, H + 2, generator=g), torch.randn(4, na + 1, generator=g)
    a_log, dt_bias = (-2.0 + torch.rand(H, generator=g)).to(wdtype), (0.5 * torch.randn(na, generator=g)).to(wdtype)
    state0 = torch.randn(5, H, d, dv, generator=g)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    res = []
    for single in (False, True):
        st = types.SimpleNamespace(n_reqs=4, req_row_start=ints([0, 1, 2, 2]), req_n_rows=ints([1, 1, 0, 1]), req_state_slot=ints([3, 0, 1, 4]),
                                   decode_only=single, buf=lambda tag, shape, dt: torch.empty(shape, dtype=dt, device=DEV))
        for writes in (True, False):
            state, out = state0.to(DEV), torch.full((4, H * dv), 5.0, device=DEV)
            ops.delta_rule(x.to(DEV), 3, 3 + KH * d, 3 + 2 * KH * d, beta.to(DEV), 2, dec.to(DEV), 1, per_channel, dt_bias.to(DEV),
                           a_log.to(DEV), state, out, H, KH, d, dv, st, writes)
            res.append((out, state))
    for (o1, s1), (o2, s2) in zip(res[:2], res[2:]):
        assert torch.equal(o1, o2) and torch.equal(s1, s2)
    assert float(o1[3].min()) == 5.0 and torch.equal(res[2][1][[1, 2]].cpu(), state0[[1, 2]]) and torch.equal(res[3][1].cpu(), state0)
