"""One attention launch for decoded tokens and prompt portions at head size 256 (`lead`), against a launch for each."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tiny_transformer_inference_engine_b200.ops import get_ops
    return get_ops(DEV)


@pytest.mark.parametrize("heads,kv_heads,page,decoding,portions,pieces,extra", [
    (8, 1, 64, [(700, 1)], [(0, 17)], 1, {}), (8, 1, 64, [(129, 1), (0, 1), (64, 1)], [(0, 300), (777, 33)], 3, {}),
    (8, 1, 16, [(1000, 1), (90, 1)], [(200, 130)], 4, {}), (8, 1, 128, [(63, 1)] * 9, [(1, 512)], 2, {"softcap": 20.0}),
    (4, 2, 64, [(500, 1), (31, 1)], [(100, 200)], 3, {"window": 150}), (8, 1, 64, [(500, 1), (31, 1)], [(100, 200)], 2, {"window": 128, "keep_first": 5}),
    (8, 2, 256, [(300, 1), (30, 1)], [(90, 70)], 2, {"chunk": 96}), (8, 1, 64, [(900, 1), (10, 1)], [(50, 65), (0, 129)], 5, {"weights": "sigmoid"}),
    (16, 1, 64, [(400, 8), (3, 2)], [(0, 40)], 1, {})])
def test_one_launch_for_both_classes(ops, heads, kv_heads, page, decoding, portions, pieces, extra):
    """Outputs are convex combinations of values (sigmoid weights: sums) with weights rounded to bfloat16 (2^-9) and rounded once more, in either
    launch: at most 2^-7 of the largest value apart, 2^-8 in the 2-norm."""
    D, g = 256, torch.Generator(device=DEV)
    g.manual_seed(7)
    seqs = decoding + portions
    n, nd, T = len(seqs), len(decoding), sum(t for _, t in seqs)
    pages = [-(-(s + t) // page) for s, t in seqs]
    kp, vp = (torch.randn(sum(pages) + 1, kv_heads, page, D, generator=g, device=DEV).bfloat16() for _ in range(2))
    order = (torch.randperm(sum(pages), generator=g, device=DEV) + 1).int()
    table, at = torch.zeros(n, max(pages), dtype=torch.int32, device=DEV), 0
    for i, k in enumerate(pages):
        table[i, :k] = order[at:at + k]
        at += k
    q = torch.randn(T, (heads + 2 * kv_heads) * D, generator=g, device=DEV).bfloat16()
    start = [sum(t for _, t in seqs[:i]) for i in range(n + 1)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    lens = ints([s + t for s, t in seqs])
    kw = dict(extra)
    window = kw.pop("window", 0)
    if kw.get("weights") == "sigmoid":
        kw["head_bias"] = torch.randn(heads, generator=g, device=DEV) - 4
    want, got = (torch.zeros(T, heads * D, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    for lo, hi in ((0, nd), (nd, n)):
        a, b = start[lo], start[hi]
        ops.paged_attention(q[a:b], heads, kv_heads, D, kp, vp, table[lo:hi], page, ints([x - a for x in start[lo:hi + 1]]), lens[lo:hi], hi - lo,
                            max(t for _, t in seqs[lo:hi]), max(s + t for s, t in seqs[lo:hi]), D ** -0.5, window, want[a:b], **kw)
    longest = max(s + t for s, t in seqs)
    piece = -(-longest // (128 * pieces)) * 128
    ops.paged_attention(q, heads, kv_heads, D, kp, vp, table, page, ints(start), lens, n, max(t for _, t in portions), longest, D ** -0.5, window, got,
                        plan=("tcpp", pieces, piece if pieces > 1 else 0), lead=nd, **kw)
    torch.cuda.synchronize()
    assert not ops.tc_error()
    most = vp.float().abs().max() * (longest if kw.get("weights") == "sigmoid" else 1)
    assert (got.float() - want.float()).abs().max() <= 2.0 ** -7 * most
    assert (got.double() - want.double()).norm() <= 2.0 ** -8 * want.double().norm()
