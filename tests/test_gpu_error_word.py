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
