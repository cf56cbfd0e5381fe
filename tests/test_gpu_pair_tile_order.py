"""Products on CTA pairs at the line between the two orders of their tiles: as many token rows as weight rows, one less, one more."""
import ctypes
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# rows of the weights, K; the last tiles are ragged in both directions
@pytest.mark.parametrize("rows,K", [(2306, 136), (2560, 64)])
@pytest.mark.parametrize("step", [-1, 0, 1, 700])
@pytest.mark.parametrize("gated", [False, True])
def test_both_orders_of_tiles(rows, K, step, gated):
    from kungfu_b200 import ops
    T, N = rows + step, rows // 2 if gated else rows
    bn, splits = ctypes.c_int(0), ctypes.c_int(0)
    ops.library().kf_linear_tc_plan(T, N, K, int(gated), ctypes.byref(bn), ctypes.byref(splits))
    assert (bn.value, splits.value) == (256, 1)
    g = torch.Generator().manual_seed(T + K)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(rows, K, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    ref = x.double() @ w.double().T
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T)                  # 32-bit sums of exact products
    if gated:
        out = torch.full((T, N), float("nan"), dtype=torch.bfloat16, device=DEV)
        ops.linear_gated(x, w, out, "silu", None)
        a, b = ref[:, :N], ref[:, N:]
        y = a * torch.sigmoid(a) * b
        # slopes of silu are below 1.1; its hardware exponential and reciprocal are within 2^-19; one bfloat16 rounding
        bound = 1.1 * b.abs() * bound[:, :N] + a.abs() * bound[:, N:] + (2.0 ** -8 + 2.0 ** -19) * y.abs() + 1e-7
    else:
        out = torch.full((T, N), float("nan"), device=DEV)
        ops.linear(x, w, out)
        y = ref
        bound = bound + 2.0 ** -22 * y.abs() + 1e-7
    ops.raise_on_device_error()
    assert bool(((out.double() - y).abs() <= bound).all())
