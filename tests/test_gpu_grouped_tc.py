"""The grouped product on pairs of CTAs (rows sorted by expert), plain and with the gated unit in its epilogue, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tiny_transformer_inference_engine_b200.ops import get_ops
    return get_ops(DEV)


def plan_of(ops, counts, identity, top, g):
    """A plan whose experts have the given numbers of rows (the last `identity` of them own no matrix)."""
    ids = torch.cat([torch.full((n,), e, dtype=torch.int32) for e, n in enumerate(counts)])
    ids = ids[torch.randperm(len(ids), generator=g)]
    return ops.moe_plan(ids.view(-1, top).to(DEV), len(counts), identity=identity)


CASES = [([256, 256], 0, 1, 128, 64), ([257, 255, 1, 0, 127], 0, 2, 136, 72), ([0, 0, 300, 0], 0, 1, 8, 8), ([40, 600, 3, 5], 1, 2, 264, 200), ([129] * 7 + [3], 2, 2, 392, 1032)]


@pytest.mark.parametrize("counts,identity,top,F,K", CASES)
@pytest.mark.parametrize("consts", [(1.702, 7.0, 1.0), (1.0, 0.0, 0.0), (1.0, 0.5, 0.0)])
def test_gated(ops, counts, identity, top, F, K, consts):
    """Experts without rows, rows at the edges of the 256-row tiles, widths and depths that do not fill a tile."""
    g = torch.Generator().manual_seed(len(counts) + F)
    plan = plan_of(ops, counts, identity, top, g)
    E, P = len(counts) - identity, sum(counts)
    x = torch.randn(P // top, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn(E, 2 * F, K, generator=g) * 2 * K ** -0.5).bfloat16().to(DEV)
    got = ops._grouped_tc(x, w, plan, top, F, *consts)
    pos, off = plan["pair_of_pos"].long().cpu(), plan["offsets"].cpu()
    alpha, limit, shift = consts
    for e in range(E):
        rows = x.double().cpu()[pos[off[e]:off[e + 1]] // top]
        gate, up = (rows @ w[e].double().cpu().T).split(F, dim=1)
        if limit:
            gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
        exp = gate * torch.sigmoid(alpha * gate) * (up + shift)
        # one rounding to bfloat16 of 32-bit sums of K products of unit size
        assert torch.allclose(got[off[e]:off[e + 1]].double().cpu(), exp, rtol=2.0 ** -8, atol=2e-5 * K ** 0.5)
    assert ops.tc_error() == 0


@pytest.mark.parametrize("counts,identity,top,N,K", CASES)
def test_plain(ops, counts, identity, top, N, K):
    g = torch.Generator().manual_seed(len(counts) + N + 1)
    plan = plan_of(ops, counts, identity, top, g)
    E, P = len(counts) - identity, sum(counts)
    rows = torch.randn(P, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().to(DEV)
    got = ops._grouped_tc(rows, w, plan, 0)
    off = plan["offsets"].cpu()
    for e in range(E):
        exp = rows[off[e]:off[e + 1]].double().cpu() @ w[e].double().cpu().T
        assert torch.allclose(got[off[e]:off[e + 1]].double().cpu(), exp, rtol=2.0 ** -8, atol=1e-5 * K ** 0.5)
    assert ops.tc_error() == 0


@pytest.mark.parametrize("rows", [3, 300])
@pytest.mark.parametrize("consts", [(1.702, 7.0, 1.0), (1.0, 0.0, 0.0)])
def test_gated_on_what_is_not_finite(ops, rows, consts):
    """Gates and up values that are not finite, through the public call in every form it has: NaN without clamps stays NaN, with clamps it is what
    the clamp makes of it; infinities likewise.  The gates' columns (+inf, -inf, NaN, 1) against the up columns of the same."""
    odd = torch.tensor([float("inf"), float("-inf"), float("nan"), 1.0])
    x, w = torch.zeros(rows, 64), torch.zeros(2, 2 * 16, 64)
    x[:, 0], x[:, 1] = 1.0, 0.0
    w[:, :16, 0], w[:, 16:, 0] = odd.repeat_interleave(4), odd.repeat(4)
    w[:, :, 1:] = 0.0
    ids = torch.arange(rows, dtype=torch.int32) % 2
    plan = ops.moe_plan(ids.view(-1, 1).to(DEV), 2)
    alpha, limit, shift = consts
    g, u = odd.repeat_interleave(4), odd.repeat(4)
    if limit:                                                         # (fminf and fmaxf return the number of a number and NaN)
        g, u = torch.fmin(g, torch.tensor(limit)), torch.fmin(torch.fmax(u, torch.tensor(-limit)), torch.tensor(limit))
    exp = (g / (1 + torch.exp(-alpha * g)) * (u + shift)).bfloat16()
    xs, ws = x.bfloat16().to(DEV), w.bfloat16().to(DEV)
    forms = {"own": ops._grouped_tc(xs, ws, plan, 1, 16, *consts), "call": ops.grouped_glu(xs, ws, plan, 1, 16, *consts),
             "kernel": ops.glu(torch.cat([odd.repeat_interleave(4), odd.repeat(4)])[None].bfloat16().to(DEV), 16, *consts)}
    for name, got in forms.items():
        assert torch.allclose(got.float().cpu(), exp.float().expand(len(got), 16), rtol=2.0 ** -7, equal_nan=True), name
    assert ops.tc_error() == 0


@pytest.mark.parametrize("alpha", [1.0, 1.702])
def test_gated_gate_far_below_zero(ops, alpha):
    """A gate whose 1 + e^(-alpha g) lies above 2^126 still divides: small, not zero (one rounding to bfloat16; the rest is 2^-21 and below)."""
    z = torch.tensor([-87.4, -88.0, -88.5, -60.0, -3.0, 2.0, -0.125, -30.0], dtype=torch.float64)
    parts, rest = [], z / alpha
    for _ in range(3):                                                # a gate in three bfloat16 pieces
        parts.append(rest.bfloat16()); rest = rest - parts[-1].double()
    x, w = torch.zeros(300, 64), torch.zeros(2, 16, 64)
    x[:, :3] = 1.0
    for i, p in enumerate(parts):
        w[:, :8, i] = p.float()
    w[:, 8:, 0] = 2.0 ** 100
    plan = ops.moe_plan((torch.arange(300, dtype=torch.int32) % 2).view(-1, 1).to(DEV), 2)
    got = ops._grouped_tc(x.bfloat16().to(DEV), w.bfloat16().to(DEV), plan, 1, 8, alpha, 0.0, 0.0).double().cpu()
    g = sum(p.double() for p in parts)
    assert torch.allclose(got, (g / (1 + torch.exp(-alpha * g)) * 2.0 ** 100).expand(300, 8), rtol=2.0 ** -8, atol=0.0)
    assert ops.tc_error() == 0


def test_gated_unit_in_32_bits(ops):
    """The unit on gates and up values that are known exactly (one product each): all but a few results are the correctly rounded ones.  Errors of
    some four units of 2^-24 turn a rounding to 2^-9 one time in four thousand; the fast exponential's twenty would one time in seven hundred."""
    F = 8192
    g = torch.Generator().manual_seed(3)
    x, w = torch.zeros(260, 64), torch.zeros(1, 2 * F, 64)
    x[:, 0] = 1.0
    w[0, :F, 0] = (torch.rand(F, generator=g) * 50 - 40)
    w[0, F:, 0] = torch.randn(F, generator=g)
    w = w.bfloat16()
    plan = ops.moe_plan(torch.zeros(260, 1, dtype=torch.int32, device=DEV), 1)
    got = ops._grouped_tc(x.bfloat16().to(DEV), w.to(DEV), plan, 1, F, 1.702, 0.0, 1.0).cpu()
    gate, up = w[0, :F, 0].double(), w[0, F:, 0].double()
    exp = (gate / (1 + torch.exp(-float(torch.tensor(1.702)) * gate)) * (up + 1)).bfloat16()
    assert torch.equal(got, got[:1].expand_as(got))
    assert (got[0] != exp).sum().item() <= 6


@pytest.mark.parametrize("side", ["own", "library"])
@pytest.mark.parametrize("counts,identity,top,N,K", CASES[1:])
def test_both_sides_of_the_rule_through_the_public_calls(ops, monkeypatch, side, counts, identity, top, N, K):
    """``grouped_linear`` and ``grouped_act`` on the product that the rows-per-expert rule names, over the same plan: experts without rows,
    and experts without a matrix, whose pairs stand behind all others."""
    g = torch.Generator().manual_seed(len(counts) + K)
    plan = plan_of(ops, counts, identity, top, g)
    E, P = len(counts) - identity, sum(counts)
    monkeypatch.setattr(ops, "_grouped_few", lambda x, plan: 0)
    monkeypatch.setattr(ops, "grouped_tc_plain_rows", 1 << 20 if side == "own" else 0)
    ran, call = [], ops._library_grouped
    monkeypatch.setattr(ops, "_library_grouped", lambda *a: ran.append(call(*a)) or ran[-1])
    x = torch.randn(P // top, K, generator=g).bfloat16().to(DEV)
    w = (torch.randn(E, N, K, generator=g) * K ** -0.5).bfloat16().to(DEV)
    scale = torch.rand(P // top, top, generator=g)
    rows, up = ops.grouped_linear(x, w, plan, top), ops.grouped_act(x, w, plan, top, "relu2", row_scale=scale.to(DEV))
    assert len(ran) == (0 if side == "own" else 2) and all(r is not None for r in ran)
    pos, off = plan["pair_of_pos"].long().cpu(), plan["offsets"].cpu()
    for e in range(E):
        at = pos[off[e]:off[e + 1]]
        exp = x.double().cpu()[at // top] @ w[e].double().cpu().T
        assert torch.allclose(rows[off[e]:off[e + 1]].double().cpu(), exp, rtol=2.0 ** -8, atol=1e-5 * K ** 0.5)
        # (the square doubles the rounding of the product, which stands in bfloat16 ahead of it)
        exp = torch.relu(exp * scale.reshape(-1)[at][:, None].double()) ** 2
        assert torch.allclose(up[off[e]:off[e + 1]].double().cpu(), exp, rtol=2.0 ** -6, atol=1e-4 * K ** 0.5)
