"""The kernel that brings a branch into the residual stream and norms it, at the edges of its vectors and thread counts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# rows around the line between a vector and four per thread; widths of one vector, off and at whole warps, above 1,024 vectors,
# the widest, one beyond it and one of no whole vectors (the scalar kernels)
@pytest.mark.parametrize("T,H", [(1, 4), (3, 132), (255, 2304), (256, 2304), (257, 100), (5, 4096), (5, 4100), (300, 3584), (2, 16384), (2, 16388), (4, 130)])
@pytest.mark.parametrize("wd,od", [(torch.float32, torch.float32), (torch.bfloat16, torch.bfloat16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("mode", ["normed", "scaled", "plain", "plain2"])
def test_branch_and_next_norm(T, H, wd, od, mode):
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(T + H)
    a, b, x = (torch.randn(T, H, generator=g) for _ in range(3))
    w1, w2 = torch.randn(H, generator=g).to(wd), torch.randn(H, generator=g).to(wd)
    dx, out = x.to(DEV), torch.full((T + 1, H), 3.0, dtype=od, device=DEV)
    copy = torch.empty(T, H, dtype=od, device=DEV)
    da, db, dw1, dw2 = a.to(DEV), b.to(DEV), w1.to(DEV), w2.to(DEV)
    A, B, X, W1, W2 = a.double(), b.double(), x.double(), w1.double(), w2.double()
    if mode == "normed":
        ops.add_rmsnorm(da, dw1, 1e-6, True, dx, next_weight=dw2, next_eps=1e-5, next_plus_one=True, next_out=out[:T])
        branch = A * torch.rsqrt(A.pow(2).mean(-1, keepdim=True) + 1e-6) * (1 + W1)
    elif mode == "scaled":
        ops.scale_add_rmsnorm(da, dw1, dx, next_weight=dw2, next_eps=1e-5, next_plus_one=True, next_out=out[:T], copy_out=copy)
        branch = A * W1
    else:
        ops.add2_rmsnorm(da, db if mode == "plain2" else None, dx, next_weight=dw2, next_eps=1e-5, next_plus_one=True, next_out=out[:T])
        branch = A + B if mode == "plain2" else A
    want = X + branch
    size = X.abs() + branch.abs()
    # a handful of roundings of what is added, and the mean square's (a tree of at most 64 levels and terms) on the branch
    assert bool(((dx.cpu().double() - want).abs() <= 40 * 2.0 ** -24 * size + 1e-30).all())
    normed = want * torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * (1 + W2)
    unit = 2.0 ** -8 if od == torch.bfloat16 else 2.0 ** -24
    root = torch.rsqrt(want.pow(2).mean(-1, keepdim=True) + 1e-5) * (1 + W2).abs()
    assert bool(((out[:T].cpu().double() - normed).abs() <= unit * normed.abs() + 100 * 2.0 ** -24 * size * root + 1e-30).all())
    assert float(out[T].float().min()) == 3.0
    if mode == "scaled":
        assert torch.equal(copy.cpu(), dx.cpu().to(od))


# one warp of vectors, ragged and whole warps, 1,024 vectors, more than those, and no whole vectors
@pytest.mark.parametrize("H", [4, 132, 2048, 2304, 4096, 4100, 130])
@pytest.mark.parametrize("mode", ["normed", "scaled", "plain2", "gated"])
def test_a_row_has_the_same_bits_in_steps_of_255_and_256_rows(H, mode):
    import types
    from kungfu_b200 import ops
    g = torch.Generator().manual_seed(H)
    a, b, x = (torch.randn(256, H, generator=g).to(DEV) for _ in range(3))
    w1, w2 = torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)
    got = []
    for T in (255, 256):
        dx, out = x[:T].clone(), torch.empty(T, H, device=DEV)
        nxt = dict(next_weight=w2, next_eps=1e-5, next_plus_one=True, next_out=out)
        if mode == "normed":
            ops.add_rmsnorm(a[:T], w1, 1e-6, True, dx, **nxt)
        elif mode == "scaled":
            ops.scale_add_rmsnorm(a[:T], w1, dx, **nxt)
        elif mode == "plain2":
            ops.add2_rmsnorm(a[:T], b[:T], dx, **nxt)
        else:
            ops.gated_group_norm(a[:T], b[:T], 0, w1, 1e-5, 1, out, types.SimpleNamespace(row_req=torch.zeros(T, dtype=torch.int32, device=DEV)))
        got.append((dx[:255], out[:255]))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
