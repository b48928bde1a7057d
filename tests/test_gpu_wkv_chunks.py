"""Chunks of the wkv recurrence at the edges of their forms: three or four CTAs per SM, decays off 16 bytes, keys that outlast their decays."""
import pytest
import torch
from test_gpu_chunks import DEV, Scan, ops, rel  # noqa: F401

pytestmark = pytest.mark.gpu


# (slots = tokens / 64 + requests, times heads: up to and above 444, three CTAs on each of 148 SMs); partial chunks, heads below 64 channels, and of 128
@pytest.mark.parametrize("lens,H,D", [([700], 40, 64), ([700], 41, 64), ([63, 64, 65, 1, 300], 60, 64), ([130, 500], 64, 40), ([200], 150, 8), ([70, 129], 3, 128), ([65], 2, 104)])
def test_wkv_chunks_by_grid_and_head(ops, lens, H, D):  # noqa: F811
    """Some hundred products whose factors carry a few roundings each of 2^-24: 1e-6, as for the other forms."""
    sc = Scan("wkv", lens, H, D, D, seed=3)
    out, states = sc.forced(ops, True)
    exp, exp_states = sc.exact()
    assert rel(out, exp) < 1e-6 and rel(states[0], exp_states[0]) < 1e-6


@pytest.mark.parametrize("D", [64, 128])
def test_wkv_decays_off_16_bytes(ops, D):  # noqa: F811
    sc = Scan("wkv", [100, 30], 2, D, D, seed=6)
    out, states = sc.forced(ops, True)
    room = torch.empty(sc.w.numel() + 1, device=DEV)
    room[1:] = sc.w.flatten()
    sc.w = room[1:].view_as(sc.w)
    out2, states2 = sc.forced(ops, True)
    assert torch.equal(out, out2) and torch.equal(states[0], states2[0])


def test_wkv_keys_that_outlast_their_decays(ops):  # noqa: F811
    """Products of decays below 2^-126 beside keys of 2^100: the state is what the walk has, whose every step stays in range."""
    sc = Scan("wkv", [40], 2, 64, 64, seed=2)
    sc.k.zero_()
    sc.k[0], sc.k[3] = 2.0 ** 100, -(2.0 ** 100)
    sc.w.fill_(2.0 ** -4)
    sc.S0.zero_()
    out, (S, _) = sc.forced(ops, True)
    walk, (W, _) = sc.forced(ops, False)
    assert W.abs().max() > 0 and torch.allclose(S, W, rtol=1e-6) and torch.allclose(out, walk, rtol=1e-5, atol=1e-5 * float(walk.abs().max()))


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("key", [2.0 ** 9, -(2.0 ** 11), 2.0 ** 39])
@pytest.mark.parametrize("tokens", [30, 34, 37, 40, 64])
def test_wkv_large_keys_behind_small_decays(ops, tokens, key, D):  # noqa: F811
    """Products of decays from 2^-99 to 2^-300 beside a key: the state to 32 bits (2e-6), or to 2^-131 of the values where the planes of a key end at 2^-133."""
    sc = Scan("wkv", [tokens], 2, D, D, seed=2)
    sc.k.zero_()
    sc.k[0] = key
    sc.w.uniform_(0.03, 0.1, generator=torch.Generator(device=DEV).manual_seed(5))
    sc.S0.zero_()
    out, (S, _) = sc.forced(ops, True)
    exp, (E,) = sc.exact()
    assert ((S.double() - E).abs() <= 2e-6 * E.abs() + 2.0 ** -131 * float(sc.v.float().abs().max())).all()
    assert rel(out, exp) < 1e-6


@pytest.mark.parametrize("D", [64, 128])
def test_wkv_large_states_behind_small_decays(ops, D):  # noqa: F811
    """The state's factor over a chunk, 2^-114 beside states of 2^60."""
    sc = Scan("wkv", [30], 2, D, D, seed=2)
    sc.k.zero_()
    sc.w.uniform_(0.06, 0.08, generator=torch.Generator(device=DEV).manual_seed(5))
    sc.S0 *= 2.0 ** 60
    _, (S, _) = sc.forced(ops, True)
    _, (E,) = sc.exact()
    assert float(E.abs().max()) > 2.0 ** -70 and rel(S, E) < 2e-7
