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
