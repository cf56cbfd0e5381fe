"""Kernels for a few rows: the short products of 32-bit rows and bfloat16 weights, the heads' norm and gate in whole vectors."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# k of one vector, at and beside the instances' edges; features off a block's 32; up to 64 rows the kernel of few rows, at 65 the tiles
@pytest.mark.parametrize("N,K", [(1, 8), (33, 64), (100, 72), (2048, 64), (31, 128)])
@pytest.mark.parametrize("od", [torch.float32, torch.bfloat16])
def test_few_rows_give_the_bits_of_many(N, K, od):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(N + K)
    base = torch.randn(65, K + 12, generator=g).to(DEV)
    w = torch.randn(N, K, generator=g).to(torch.bfloat16).to(DEV)
    whole = torch.empty(65, N, dtype=od, device=DEV)
    ops.linear_cols(base, 4, w, whole)
    want = base[:, 4:4 + K].double() @ w.double().T
    bound = (K + 2) * 2.0 ** -24 * (base[:, 4:4 + K].double().abs() @ w.double().abs().T) + (2.0 ** -8 if od == torch.bfloat16 else 0.0) * want.abs()
    assert bool(((whole.double() - want).abs() <= bound).all())
    for T in (1, 2, 7, 8, 9, 64):
        out = torch.full((T + 1, N), 5.0, dtype=od, device=DEV)
        ops.linear_cols(base[:T].contiguous(), 4, w, out[:T])
        assert torch.equal(out[:T], whole[:T]) and float(out[T].float().min()) == 5.0, T


@pytest.mark.parametrize("H,dv", [(3, 4), (16, 128), (2, 132), (5, 256), (1, 260)])
@pytest.mark.parametrize("wd,od", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (None, torch.bfloat16)])
@pytest.mark.parametrize("act", ["silu", "sigmoid"])
def test_heads_in_whole_vectors(H, dv, wd, od, act):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(H + dv)
    T = 7
    o, gate = 3.0 * torch.randn(T, H * dv, generator=g), 2.0 * torch.randn(T, H * dv + 8, generator=g)
    w = None if wd is None else torch.randn(H * dv, generator=g).to(wd)
    out = torch.full((T, H * dv + 4), 5.0, dtype=od, device=DEV)
    ops.head_norm_gate(o.to(DEV), None if w is None else w.to(DEV), 1e-5, gate.to(DEV), 4, act, out, H, dv, out_col0=4, scale=0.5)
    x, z = o.double().view(T, H, dv), gate[:, 4:4 + H * dv].double()
    y = (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5)).view(T, H * dv) * (1.0 if w is None else w.double())
    want = y * torch.sigmoid(z) * (z if act == "silu" else 1.0) * 0.5
    unit = 2.0 ** -8 if od == torch.bfloat16 else 2.0 ** -24
    # the mean square (a chain of 8 and a tree of 5), root, quotient, exponential and four products: under 40 roundings
    assert bool(((out[:, 4:].cpu().double() - want).abs() <= (unit + 40 * 2.0 ** -24) * want.abs() + 1e-30).all())
    assert float(out[:, :4].float().min()) == 5.0
