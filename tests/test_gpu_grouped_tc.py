"""Experts of many rows on tcgen05: ragged sizes, one and two tiles of the plan a block, experts without rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(autouse=True)
def every_size(monkeypatch):
    """The kernel's edges lie at sizes at which the other one is faster."""
    from kungfu_b200 import ops
    monkeypatch.setattr(ops, "grouped_on_tcgen05", "always")


class _Ctx:
    def buf(self, name, shape, dtype):
        return torch.empty(shape, dtype=dtype, device=DEV)


# rows an expert: 130 (two tiles and one of 2 rows), 64 exactly, 1 to 300 with one empty expert; features and k around tiles of
# 128 and 64, k shorter than the ring
@pytest.mark.parametrize("counts,top,N,K", [((130, 130), 1, 128, 72), ((64, 64, 64), 1, 300, 264), ((1, 300, 0, 65, 128, 129, 63, 200), 1, 200, 520),
                                            ((128, 129, 200), 2, 1000, 64)])
@pytest.mark.parametrize("act", ["", "clamped_swish", "silu"])
@pytest.mark.parametrize("out", ["bfloat16", "float32"])
def test_many_rows_per_expert(counts, top, N, K, act, out):
    from kungfu_b200 import ops
    E = len(counts)
    g = torch.Generator().manual_seed(N + K)
    first = torch.cat([torch.full((n,), e) for e, n in enumerate(counts)])
    first = first[torch.randperm(len(first), generator=g)]
    ids = torch.stack([(first + j) % E for j in range(top)], 1).to(torch.int32)
    T, gated = len(first), bool(act)
    x = torch.randn(T, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g) * K ** -0.5).to(torch.bfloat16)
    scale = torch.rand(T, top, generator=g) if act == "silu" else None
    assert ops.library().kf_grouped_tc_supported(0, 0, T * top, E, N, K)
    plan = ops.moe_plan(ids.to(DEV), E, _Ctx())
    got = torch.full((T * top + 1, N), float("nan"), dtype=getattr(torch, out), device=DEV)
    ops.moe_linear(x.to(DEV), plan, w.to(DEV), got[:-1], gather=True, gated=gated, limit=0.9, activation=act or "clamped_swish",
                   row_scale=scale.to(DEV) if scale is not None else None)
    assert bool(got[-1].isnan().all())
    pair = plan["sorted_pair"].cpu().long()
    e_of = ids.view(-1).long()[pair]
    xs = x.double()[pair // top]
    y, err = torch.empty(T * top, w.shape[1], dtype=torch.float64), torch.empty(T * top, w.shape[1], dtype=torch.float64)
    for e in range(E):
        rows = e_of == e
        y[rows] = xs[rows] @ w[e].double().T
        err[rows] = K * 2.0 ** -23 * (xs[rows].abs() @ w[e].double().abs().T)       # 32-bit sums of exact products
    if gated:
        r = scale.view(-1)[pair][:, None].double() if scale is not None else 1.0
        gate, up = y[:, :N] * r, y[:, N:] * r
        if act == "silu":
            size = 1 + up.abs().clamp(min=gate.abs())
            y = gate * torch.sigmoid(gate) * up
        else:
            size = 4.0
            gate, up = gate.clamp(max=0.9), up.clamp(-0.9, 0.9)
            y = gate * torch.sigmoid(1.702 * gate) * (up + 1)
        err = 2 * size * (err[:, :N] + err[:, N:]) + 1e-6                          # slopes of the activations
    err = err + (2.0 ** -8 if out == "bfloat16" else 2.0 ** -22) * y.abs() + 1e-7
    assert bool(((got[:-1].cpu().double() - y).abs() <= err).all())
    if not gated:
        again = torch.empty_like(got[:-1])
        ops.moe_linear(x[pair // top].to(DEV), plan, w.to(DEV), again, gather=False)
        assert torch.equal(again, got[:-1])
    ops.raise_on_device_error()


def test_the_sorted_rows_belong_to_the_plan():
    """A gathered product writes its result and a buffer of the plan's context; the scratch that every launch of the device shares stays
    as it is."""
    from kungfu_b200 import ops
    P, E, N, K = 256, 2, 128, 64
    taken = {}

    class Ctx(_Ctx):
        def buf(self, name, shape, dtype):
            taken[name] = super().buf(name, shape, dtype)
            return taken[name]

    plan = ops.moe_plan((torch.arange(P, device=DEV, dtype=torch.int32) % E)[:, None].contiguous(), E, Ctx())
    x = torch.randn(P, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(E, N, K, device=DEV).to(torch.bfloat16)
    out = torch.empty(P, N, device=DEV)
    shared = ops._partial(torch.device(DEV), P * K)
    shared.fill_(-3.0)
    assert ops.library().kf_grouped_tc_supported(0, 0, P, E, N, K)
    ops.moe_linear(x, plan, w, out, gather=True)
    assert bool((shared == -3.0).all()) and ops._partial(torch.device(DEV), 1) is shared
    assert torch.equal(taken["moe_sorted_rows"], x[plan["sorted_pair"].long()])


@pytest.mark.parametrize("gather,gated,N,K,takes", [(True, True, 384, 768, True), (True, True, 383, 768, False), (True, True, 384, 760, False), (True, True, 128, 1536, True),
                                                    (False, True, 128, 1528, False), (True, False, 512, 512, False), (False, False, 128, 256, True), (False, False, 128, 248, False)])
def test_the_line_between_the_two_kernels(gather, gated, N, K, takes, monkeypatch):
    """Which kernel a product of 64 rows an expert takes; one row fewer an expert never takes the tcgen05 one."""
    from kungfu_b200 import ops
    monkeypatch.setattr(ops, "grouped_on_tcgen05", True)
    lib, seen = ops.library(), []

    class Spy:
        def __getattr__(self, name):
            if name in ("kf_grouped_tc", "kf_grouped_linear"):
                seen.append(name)
            return getattr(lib, name)

    monkeypatch.setattr(ops, "library", Spy)
    x = torch.randn(128, K, device=DEV).to(torch.bfloat16)
    w = torch.randn(2, 2 * N if gated else N, K, device=DEV).to(torch.bfloat16)
    for rows in (128, 126):
        plan = ops.moe_plan((torch.arange(rows, device=DEV, dtype=torch.int32) % 2)[:, None].contiguous(), 2, _Ctx())
        ops.moe_linear(x[:rows], plan, w, torch.empty(rows, N, device=DEV), gather=gather, gated=gated, limit=1.0)
    assert seen == ["kf_grouped_tc" if takes else "kf_grouped_linear", "kf_grouped_linear"]


# 63 and 64 rows an expert on average; the second step holds the first one's tokens.  K with a last slice of 8 and of 64, one stage and many.
@pytest.mark.parametrize("E,N,K", [(2, 128, 8), (3, 200, 520), (2, 1000, 264), (8, 512, 768), (4, 300, 2048)])
@pytest.mark.parametrize("act", ["", "clamped_swish", "silu"])
@pytest.mark.parametrize("out", ["bfloat16", "float32"])
def test_a_row_has_the_same_bits_on_either_side_of_the_line(E, N, K, act, out):
    """A token's result does not depend on what else is in the step, although from 64 rows an expert on average another kernel takes the
    product: both sum a row's products in 32 bits over k in ascending slices of 16."""
    from kungfu_b200 import ops
    gated, many, few = bool(act), 64 * E, 64 * E - 1
    g = torch.Generator().manual_seed(E + K)
    ids = torch.randint(0, E, (many, 1), generator=g).to(torch.int32)
    x = torch.randn(many, K, generator=g).to(torch.bfloat16).to(DEV)
    x[::7] *= 1e4                                              # rows whose sums cancel differently in another order
    w = (torch.randn(E, 2 * N if gated else N, K, generator=g) * K ** -0.5).to(torch.bfloat16).to(DEV)
    scale = torch.rand(many, 1, generator=g).to(DEV) if act == "silu" else None
    got = {}
    for n in (few, many):
        plan = ops.moe_plan(ids[:n].to(DEV), E, _Ctx())
        assert bool(ops.library().kf_grouped_tc_supported(0, 0, n, E, N, K)) == (n == many)
        y = torch.empty(n, N, dtype=getattr(torch, out), device=DEV)
        ops.moe_linear(x[:n], plan, w, y, gather=True, gated=gated, limit=0.9, activation=act or "clamped_swish",
                       row_scale=scale[:n] if scale is not None else None)
        got[n] = torch.empty_like(y)
        got[n][plan["sorted_pair"].long()] = y
    assert torch.equal(got[few], got[many][:few])
    ops.raise_on_device_error()
