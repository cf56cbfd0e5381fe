"""Grouped products whose groups have few rows: every count of row tiles, ragged sizes, groups larger than expected."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from kungfu_b200 import ops as o
    return o


class _Ctx:
    def buf(self, name, shape, dtype):
        return torch.empty(shape, dtype=dtype, device=DEV)


# tokens 1..33 cross the counts of row tiles (8, 16, 32) and the rule's line; with T = 60 and 100 over more experts the mean is
# small and one expert has every token (60 rows: eight row tiles; 100: two tiles of the plan); N and K off the tiles of 32
# features, 64 features and 64 k
@pytest.mark.parametrize("T,E,top,N,K,out", [(1, 4, 1, 33, 72, "bfloat16"), (8, 32, 3, 256, 2048, "bfloat16"), (9, 8, 2, 100, 64, "float32"),
                                             (16, 3, 2, 64, 136, "float32"), (17, 5, 2, 31, 200, "bfloat16"), (32, 2, 1, 96, 8, "float32"),
                                             (33, 64, 2, 40, 328, "bfloat16"), (60, 40, 2, 70, 264, "float32"), (100, 64, 2, 70, 264, "bfloat16"),
                                             (33, 2, 2, 70, 264, "float32")])
@pytest.mark.parametrize("gated", [False, True])
def test_few_rows_per_expert(ops, T, E, top, N, K, out, gated):
    g = torch.Generator().manual_seed(T + N)
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32)
    if top > 1 and E > 2:
        ids[:, 0] = 1                                             # every token's first choice
        ids[:, 1:] = torch.stack([torch.randperm(E - 2, generator=g)[:top - 1] + 2 for _ in range(T)])
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    scale = torch.rand(T, top, generator=g) if gated else None
    plan = ops.moe_plan(ids.to(DEV), E, _Ctx())
    dt = getattr(torch, out)
    got = torch.full((T * top + 1, N), float("nan"), dtype=dt, device=DEV)
    ops.moe_linear(x.to(DEV), plan, w.to(DEV), got[:-1], gather=True, gated=gated, limit=0.9,
                   row_scale=scale.to(DEV) if gated else None)
    assert bool(got[-1].isnan().all())
    pair = plan["sorted_pair"].cpu().long()
    xs, ws = x.double()[pair // top], w.double()[ids.view(-1).long()[pair]]
    y = torch.einsum("rk,rnk->rn", xs, ws)
    err = K * 2.0 ** -23 * torch.einsum("rk,rnk->rn", xs.abs(), ws.abs())        # 32-bit sums of exact products
    if gated:
        r = scale.view(-1)[pair][:, None].double()
        gate, up = (y[:, :N] * r).clamp(max=0.9), (y[:, N:] * r).clamp(-0.9, 0.9)
        y = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        err = 4 * (err[:, :N] + err[:, N:]) + 1e-6                                # slopes of the activation are below 2
    err = err + (2.0 ** -8 if out == "bfloat16" else 2.0 ** -22) * y.abs() + 1e-7
    assert bool(((got[:-1].cpu().double() - y).abs() <= err).all())
    # rows that were gathered before give the same product
    again = torch.empty_like(got[:-1])
    if not gated:
        ops.moe_linear(x[pair // top].to(DEV), plan, w.to(DEV), again, gather=False)
        assert torch.equal(again, got[:-1])


@pytest.mark.parametrize("T", [1, 9, 20, 30])
@pytest.mark.parametrize("gated", [False, True])
def test_a_row_has_the_same_bits_in_a_step_of_few_rows_and_of_many(ops, T, gated):
    """The first T of 70 tokens over two experts, alone (streamed weights) and in the whole step (tiles of 64 rows)."""
    g = torch.Generator().manual_seed(T)
    E, N, K = 2, 70, 264
    ids = torch.randint(0, E, (70, 1), generator=g).to(torch.int32)
    x = torch.randn(70, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    got = {}
    for n in (T, 70):
        plan = ops.moe_plan(ids[:n].to(DEV), E, _Ctx())
        out = torch.empty(n, N, device=DEV)
        ops.moe_linear(x[:n], plan, w, out, gather=True, gated=gated, limit=0.9)
        got[n] = torch.empty_like(out)
        got[n][plan["sorted_pair"].long()[:n]] = out
    assert torch.equal(got[T], got[70][:T])


@pytest.mark.parametrize("T", [1, 8, 9, 17, 32, 33])
def test_head_maps_of_few_rows(ops, T):
    g = torch.Generator().manual_seed(T)
    H, O, I = 3, 50, 72
    x = torch.randn(T, 8 + H * I + 16, generator=g).to(torch.bfloat16)
    w = (torch.randn(H, O, I, generator=g) * 0.1).to(torch.bfloat16)
    got = torch.empty(T, H * O, device=DEV)
    ops.head_linear(x.to(DEV), 8, w.to(DEV), got)
    xs = x[:, 8:8 + H * I].double().view(T, H, I)
    want = torch.einsum("thi,hoi->tho", xs, w.double()).reshape(T, H * O)
    bound = I * 2.0 ** -23 * torch.einsum("thi,hoi->tho", xs.abs(), w.double().abs()).reshape(T, H * O)
    assert bool(((got.cpu().double() - want).abs() <= bound).all())
