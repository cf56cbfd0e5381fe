"""The error word names the wait that ran out first, not the ones that followed it."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T,N,K", [(8, 2304, 2304), (40, 256, 520)])
def test_a_product_whose_operands_never_arrive(T, N, K):
    """A test hook makes the producer leave out its loads from the second stage on, with a limit of 2 ms: the issuer gives up, and the
    epilogue, which waits for it, must not write its own code over that."""
    from kungfu_b200 import ops
    lib = ops.library()
    x, w = torch.randn(T, K, device=DEV).to(torch.bfloat16), torch.randn(N, K, device=DEV).to(torch.bfloat16)
    out = torch.zeros(T, N, device=DEV)
    ops.linear(x, w, out)
    torch.cuda.synchronize()
    assert lib.kf_test_gemm_give_up(ctypes.c_ulonglong(2_000_000), 1) == 0
    try:
        ops.linear(x, w, out)
        torch.cuda.synchronize()
        assert ops.device_error() == 1
        with pytest.raises(ops.KernelError, match="a product, operands never arrived"):
            ops.raise_on_device_error()
    finally:
        assert lib.kf_test_gemm_give_up(ctypes.c_ulonglong(0), -1) == 0
        ops.clear_device_error()


# one stage and none before the loads stop; K of two stages, of the ring (four stages gated, three not) and of more
@pytest.mark.parametrize("drop,K", [(0, 72), (1, 128), (3, 256), (2, 1024)])
@pytest.mark.parametrize("gated", [False, True])
def test_experts_whose_operands_never_arrive(drop, K, gated, monkeypatch):
    """The same for the experts' kernel: it comes back by itself with its code, stores nothing, and the product is right again after."""
    from kungfu_b200 import ops
    from test_gpu_grouped_tc import _Ctx
    monkeypatch.setattr(ops, "grouped_on_tcgen05", "always")
    lib, E, N, P = ops.library(), 2, 256, 260
    plan = ops.moe_plan((torch.arange(P, device=DEV, dtype=torch.int32) % E)[:, None].contiguous(), E, _Ctx())
    x = torch.randn(P, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(E, 2 * N if gated else N, K, device=DEV).to(torch.bfloat16)
    right, out = (torch.full((P, N), 7.0, device=DEV) for _ in range(2))
    ops.moe_linear(x, plan, w, right, gather=True, gated=gated, limit=1.0)
    torch.cuda.synchronize()
    assert ops.device_error() == 0
    assert lib.kf_test_grouped_give_up(ctypes.c_ulonglong(2_000_000), drop) == 0
    try:
        ops.moe_linear(x, plan, w, out, gather=True, gated=gated, limit=1.0)
        torch.cuda.synchronize()
        assert ops.device_error() == 49
        with pytest.raises(ops.KernelError, match="a mixture's experts, operands never arrived"):
            ops.raise_on_device_error()
    finally:
        assert lib.kf_test_grouped_give_up(ctypes.c_ulonglong(0), -1) == 0
        ops.clear_device_error()
    assert bool((out == 7.0).all())
    ops.moe_linear(x, plan, w, out, gather=True, gated=gated, limit=1.0)
    ops.raise_on_device_error()
    assert torch.equal(out, right)
