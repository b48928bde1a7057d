"""One attention launch for decoded tokens and prompt portions at head size 256 (`lead`), against a launch for each."""
import pytest
import torch

from tiny_transformer_inference_engine_b200.ops import KernelError

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tiny_transformer_inference_engine_b200.ops import get_ops
    return get_ops(DEV)


def paged(heads, kv_heads, page, decoding, portions):
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
    return q, kp, vp, table, start, ints, lens, seqs, n, nd, T, D, g


@pytest.mark.parametrize("heads,kv_heads,page,decoding,portions,pieces,extra", [
    (8, 1, 64, [(700, 1)], [(0, 17)], 1, {}), (8, 1, 64, [(129, 1), (0, 1), (64, 1)], [(0, 300), (777, 33)], 3, {}),
    (8, 1, 16, [(1000, 1), (90, 1)], [(200, 130)], 4, {}), (8, 1, 128, [(63, 1)] * 9, [(1, 512)], 2, {"softcap": 20.0}),
    (4, 2, 64, [(500, 1), (31, 1)], [(100, 200)], 3, {"window": 150}), (8, 1, 64, [(500, 1), (31, 1)], [(100, 200)], 2, {"window": 128, "keep_first": 5}),
    (8, 2, 256, [(300, 1), (30, 1)], [(90, 70)], 2, {"chunk": 96}), (8, 1, 64, [(900, 1), (10, 1)], [(50, 65), (0, 129)], 5, {"weights": "sigmoid"}),
    (16, 1, 64, [(400, 8), (3, 2)], [(0, 40)], 1, {})])
def test_one_launch_for_both_classes(ops, heads, kv_heads, page, decoding, portions, pieces, extra):
    """Outputs are convex combinations of values (sigmoid weights: sums) with weights rounded to bfloat16 (2^-9) and rounded once more, in either
    launch: at most 2^-7 of the largest value apart, 2^-8 in the 2-norm."""
    q, kp, vp, table, start, ints, lens, seqs, n, nd, T, D, g = paged(heads, kv_heads, page, decoding, portions)
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


@pytest.mark.parametrize("heads,kv_heads,page,decoding,portions,pieces,extra", [
    (8, 1, 64, [(700, 1), (0, 1), (128, 1)], [(0, 17), (300, 40)], 1, {}), (8, 1, 16, [(1000, 1), (90, 1)], [(200, 130)], 4, {}), (8, 2, 128, [(63, 1)] * 5, [(1, 300)], 2, {"softcap": 20.0}),
    (4, 2, 64, [(500, 1), (31, 1)], [(100, 200)], 3, {"window": 150}), (8, 1, 64, [(900, 1), (10, 1)], [(50, 65)], 5, {"weights": "sigmoid"}), (16, 1, 64, [(400, 8)], [(0, 40)], 1, {})])
def test_one_launch_against_64_bits(ops, heads, kv_heads, page, decoding, portions, pieces, extra):
    """Weights of a row are rounded to bfloat16 (2^-9 of each) and the result once more: 2^-8 in the 2-norm, of the sum of the weighted values' sizes at most."""
    q, kp, vp, table, start, ints, lens, seqs, n, nd, T, D, g = paged(heads, kv_heads, page, decoding, portions)
    kw, scale, G = dict(extra), D ** -0.5, heads // kv_heads
    window = kw.pop("window", 0)
    bias = torch.zeros(heads, device=DEV)
    if kw.get("weights") == "sigmoid":
        bias = kw["head_bias"] = torch.randn(heads, generator=g, device=DEV) - 4
    longest = max(s + t for s, t in seqs)
    piece = -(-longest // (128 * pieces)) * 128
    got = torch.full((T, heads * D), 7.0, dtype=torch.bfloat16, device=DEV)
    ops.paged_attention(q, heads, kv_heads, D, kp, vp, table, page, ints(start), lens, n, max(t for _, t in portions), longest, scale, window, got,
                        plan=("tcpp", pieces, piece if pieces > 1 else 0), lead=nd, lead_q_len=max(t for _, t in decoding), **kw)
    assert not ops.tc_error()
    for i, (before, new) in enumerate(seqs):
        keys = torch.arange(before + new, device=DEV)
        flat = lambda pool: pool.double()[table[i, keys // page].long(), :, keys % page].transpose(0, 1).repeat_interleave(G, 0)      # [heads, keys, D]
        rows = q[start[i]:start[i + 1], :heads * D].double().view(new, heads, D).transpose(0, 1)
        score = rows @ flat(kp).transpose(1, 2) * scale
        if "softcap" in kw:
            score = kw["softcap"] * torch.tanh(score / kw["softcap"])
        pos = before + torch.arange(new, device=DEV)[:, None]
        seen = (keys <= pos) & ((keys > pos - window) if window else True)
        if kw.get("weights") == "sigmoid":
            p = torch.sigmoid(score + bias.double()[:, None, None]) * seen
        else:
            p = torch.softmax(score.masked_fill(~seen, -float("inf")), -1)
        want = (p @ flat(vp)).transpose(0, 1).flatten(1)
        assert (got[start[i]:start[i + 1]].double() - want).norm() <= 2.0 ** -8 * max(want.norm(), (p @ flat(vp).abs()).norm() * 2.0 ** -3)


def test_leading_requests_of_more_rows_than_a_tile_are_refused(ops):
    """Said beforehand: refused.  Not said: the step's error word has it."""
    q, kp, vp, table, start, ints, lens, seqs, n, nd, T, D, g = paged(8, 1, 64, [(30, 20)], [(0, 40)])
    out = torch.zeros(T, 8 * D, dtype=torch.bfloat16, device=DEV)
    run = lambda plan=("tcpp", 1, 0), head_dim=D, **kw: ops.paged_attention(q, 8, 1, head_dim, kp, vp, table, 64, ints(start), lens, n, 40, 50, 0.1, 0, out,
                                                                           plan=plan, **kw)
    with pytest.raises(KernelError, match="row tile"):
        run(lead=1, lead_q_len=17)
    with pytest.raises(KernelError):
        run(plan=("mma", 1, 0), lead=1, lead_q_len=1)
    run(lead=1, lead_q_len=16)
    torch.cuda.synchronize()
    with pytest.raises(KernelError, match="113"):
        ops.check_tc()
    run()
    assert not ops.tc_error()
