"""Routing and plan of few tokens in one launch, against the two launches that it takes the place of."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# one token to the most and one more, all experts of a lane's worth and one more, every choice taken, an expert that nobody or everybody chose
@pytest.mark.parametrize("T,E,top,identity", [(1, 1, 1, 0), (1, 32, 32, 0), (8, 18, 4, 2), (31, 8, 2, 0), (32, 16, 3, 16), (32, 1, 1, 0), (32, 32, 32, 3),
                                              (32, 4, 4, 0), (33, 8, 2, 0), (8, 33, 2, 1)])
def test_route_and_plan(T, E, top, identity):
    from tiny_transformer_inference_engine_b200.ops import get_ops
    ops = get_ops(DEV)
    g = torch.Generator(device=DEV)
    g.manual_seed(T * E + top)
    wide = torch.randn(T, E + 3, generator=g, device=DEV)
    for score, corrected, renorm, bad in (("sigmoid", False, False, False), ("softmax", True, True, False), ("sigmoid", True, True, True)):
        logits = wide[:, 1:1 + E].clone() if bad else wide[:, 1:1 + E]          # (rows further apart than E)
        if bad:
            logits[T // 2] = float("nan")                              # nothing compares: the first experts, and some of them twice
            logits[T - 1, : (E + 1) // 2] = float("nan")
        corr = torch.randn(E, generator=g, device=DEV) if corrected else None
        idx, wts = ops.moe_route(logits, 1, 1, 1, top, 1.5, renorm, score=score, correction=corr)
        ref = ops.moe_plan(idx, E, identity=identity)
        before = ops.launches
        idx2, wts2, plan = ops.moe_route_plan(logits, 1, 1, 1, top, 1.5, renorm, score=score, correction=corr, identity=identity)
        assert ops.launches - before == (1 if T <= 32 and E <= 32 else 2)
        assert torch.equal(idx, idx2) and torch.equal(wts.view(torch.int32), wts2.view(torch.int32))      # (NaN too)
        assert torch.equal(plan["offsets"], ref["offsets"]) and plan["meta"][0] == ref["meta"][0]
        n = 4 * int(ref["meta"][0])
        assert torch.equal(plan["tiles"][:n], ref["tiles"][:n])
        pos, pair, P = plan["pos_of_pair"].long(), plan["pair_of_pos"].long(), T * top
        assert torch.equal(pair[pos], torch.arange(P, device=DEV))
        of = plan["offsets"].long()[idx2.flatten().long()]
        assert ((pos >= of) & (pos < plan["offsets"].long()[idx2.flatten().long() + 1])).all()
        assert plan["pairs"] == P and plan["real_experts"] == E - identity and plan["max_tiles"] == ref["max_tiles"]
    assert torch.equal(ops.moe_route_plan(wide[:0, :E], 1, 1, 1, top, 1.0)[0], torch.empty(0, top, dtype=torch.int32, device=DEV))


def test_route_and_plan_of_groups():
    """More groups than one: the two launches, and what they refuse."""
    from tiny_transformer_inference_engine_b200.ops import KernelError, get_ops
    ops = get_ops(DEV)
    logits = torch.randn(8, 16, device=DEV)
    idx, wts = ops.moe_route(logits, 4, 2, 2, 3, 1.0)
    idx2, wts2, plan = ops.moe_route_plan(logits, 4, 2, 2, 3, 1.0)
    assert torch.equal(idx, idx2) and torch.equal(wts, wts2) and plan["offsets"][-1] == 24
    for groups, keep, group_top, top in ((1, 1, 1, 17), (1, 2, 1, 2), (1, 1, 3, 2), (1, 1, 1, 0)):
        with pytest.raises(KernelError):
            ops.moe_route_plan(logits, groups, keep, group_top, top, 1.0)
