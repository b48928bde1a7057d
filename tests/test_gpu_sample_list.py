"""The short list of the sampler at the edges of its ways: how many groups of warps give the bound, how many tokens a CTA hands in at once, and what lies
at the bound."""
import pytest
import torch
from test_gpu_kernels import DEV, PLAIN, ops, sampler_state, uniform_from_state  # noqa: F401

pytestmark = pytest.mark.gpu


# slices just long enough for every warp to have tokens and just not (3,969 and 3,968 of them), of one load a thread and of many; 64, 128 and all groups
@pytest.mark.parametrize("V,ctas", [(31748, 8), (31744, 8), (4096, 4), (32000, 4), (8192, 2), (700, 1), (128256, 8)])
def test_bound_and_list(ops, V, ctas):  # noqa: F811
    """Against the plain sampler (probabilities are sums of 64-bit fixed point: 2^-40 of the maximum's mass a token, 1e-4 for expf and its argument),
    and the same tokens with another number of CTAs."""
    g = torch.Generator().manual_seed(V + ctas)
    quarter, hand_in = 32 * ctas // 4, 512 // ctas
    rows, logits = [], []

    def row(x, top_k, top_p, temp=0.9):
        logits.append(x)
        rows.append((41 + len(rows), len(rows), min(top_k, V - 1), temp, top_p, 0))

    for k in (1, 32, 33, min(64, quarter), quarter):
        row(torch.randn(V, generator=g), k, 0.9)
    slice_ = (V + ctas - 1) // ctas
    for n in (hand_in, hand_in + 1):                                   # so many tokens of the list in the second CTA, or in the only one
        x = torch.randn(V, generator=g).clamp(max=2.0)
        at = slice_ + 8 if ctas > 1 else 8
        x[at:at + min(n, slice_ - 16)] = 3.0 + torch.rand(min(n, slice_ - 16), generator=g)
        row(x, 5, 0.8)
    x = -torch.rand(V, generator=g) - 1.0                              # minus zeros are the largest values: they stay, and nothing else
    x[5::97] = -0.0
    row(x, 2, 1.0)
    x = torch.full((V,), float("-inf"))                                # fewer tokens than top_k have a probability
    x[11::max(1, V // 7)] = torch.randn(x[11::max(1, V // 7)].shape, generator=g)
    row(x, quarter, 0.95)
    logits = torch.stack(logits)
    n = len(rows)
    out, again, probs = torch.empty(n, dtype=torch.int32, device=DEV), torch.empty(n, dtype=torch.int32, device=DEV), torch.zeros(n, V, device=DEV)
    slots = torch.arange(n, dtype=torch.int32, device=DEV)
    ops.sample(logits.to(DEV), slots, sampler_state(rows).to(DEV), out, probs_out=probs, ctas_per_row=ctas)
    for other in (1, 2, 8):
        ops.sample(logits.to(DEV), slots, sampler_state(rows).to(DEV), again, ctas_per_row=other)
        assert torch.equal(again, out)
    out, probs = out.cpu(), probs.cpu()
    for r, (seed, draws, top_k, temp, top_p, _) in enumerate(rows):
        exp = PLAIN.filtered_probs(logits[r], temp, top_k, top_p).float()
        assert torch.equal(probs[r] > 0, exp > 0), f"row {r}: kept sets differ"
        assert torch.allclose(probs[r], exp, atol=2e-6, rtol=1e-4)
        u = uniform_from_state(seed & 0x7fffffff, seed >> 31, draws)
        cdf, tok = torch.cumsum(probs[r].double(), 0), int(out[r])
        assert (cdf[tok - 1].item() if tok else 0.0) - 1e-5 <= u <= cdf[tok].item() + 1e-5


def test_rows_that_are_not_finite(ops):  # noqa: F811
    """Infinite maxima have no probabilities: a token of the row all the same, from the list or (greedy) without."""
    logits = torch.randn(3, 32000, device=DEV)
    logits[0, 77] = logits[0, 20000] = float("inf")
    logits[1] = float("-inf")
    logits[2, 500] = float("inf")
    out = torch.full((3,), -7, dtype=torch.int32, device=DEV)
    ops.sample(logits, torch.arange(3, dtype=torch.int32, device=DEV), sampler_state([(1, 0, 8, 0.8, 0.9, 0), (2, 0, 8, 1.0, 1.0, 1), (3, 0, 8, 0.8, 0.9, 0)]).to(DEV), out)
    assert ((out >= 0) & (out < 32000)).all()
