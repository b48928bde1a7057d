"""The chunked recurrences that norm and gate their read-outs themselves, against the pass over the read-outs that they take the place of."""
import functools

import pytest
import torch

from test_gpu_chunks import DEV, KINDS, Scan, ops  # noqa: F401  (ops: a fixture)

pytestmark = pytest.mark.gpu


class Gating:
    """The ops with ``gated`` on every scan."""

    def __init__(self, ops, gated):
        self.ops, self.gated = ops, gated

    def __getattr__(self, name):
        f = getattr(self.ops, name)
        return functools.partial(f, gated=self.gated) if name in ("retention_scan", "mlstm_scan", "mlstm_chunks", "wkv_scan") else f


def same(y, ref):
    """The sums of squares may be added in another order: a bfloat16 off by one step at most; what is not finite in the same places."""
    y, ref = y.float(), ref.float()
    assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf())
    assert ((y - ref).abs() <= 2.0 ** -7 * ref.abs())[ref.isfinite()].all()


# one request and several, whole and partial chunks, heads that fill a tile, a part of one and more than one
SIZES = [([64], 2, 64, 64), ([128, 129], 2, 64, 128), ([65, 1], 3, 128, 128), ([63, 1, 130], 2, 48, 72), ([300], 4, 8, 8), ([1, 200, 2, 17], 1, 128, 136),
         ([129, 127], 2, 24, 16), ([30] * 9, 40, 64, 48), ([1000], 4, 64, 128)]


@pytest.mark.parametrize("lens,H,D,Dv", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_gated_read_outs(ops, kind, lens, H, D, Dv):  # noqa: F811
    if kind == "wkv":
        Dv = D
    T, mode = sum(lens), KINDS.index(kind)
    g = torch.Generator(device=DEV)
    g.manual_seed(T + Dv)
    wide = (torch.randn(T, H * Dv + 48, generator=g, device=DEV) * 3).bfloat16()
    weight = torch.randn(H * Dv, generator=g, device=DEV)
    for bad in (None, float("inf"), float("nan")):                    # (what is not finite is walked)
        sc = Scan(kind, lens, H, D, Dv, seed=Dv)
        if bad is not None:
            sc.v[T // 2, Dv // 2] = bad
        ref, states = sc.forced(ops, True)
        plain = sc.launched
        tokens = ops._chunk_tokens(mode, torch.bfloat16, T, len(lens), sc.S0.shape[-1], Dv, H, ops.num_sms)
        for w, act, at in ((weight, "silu", 8), (None, "sigmoid", 0), (weight[:], "silu", 3)):
            gate = wide[:, at:at + H * Dv]                            # (from column 3: no row of it takes 16-byte loads)
            before = ops.launches
            y, states2 = sc.run(Gating(ops, (gate, w, 1e-5, act)))
            fused = (tokens == 128 or (kind == "wkv" and D <= 64)) and at % 8 == 0
            assert ops.launches - before == plain + (not fused)
            assert y.dtype == torch.bfloat16
            same(y, ops.head_norm_gate(ref, gate, w, H, Dv, 1e-5, act))
            assert all(torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)) for a, b in zip(states, states2))


@pytest.mark.parametrize("act", ["silu", "sigmoid"])
@pytest.mark.parametrize("kind", KINDS)
def test_gates_far_from_zero(ops, kind, act):  # noqa: F811
    """Gates at which e^-x takes the largest exponents.  The results are correctly rounded but where the exact value lies within their 32-bit error of a
    tie: 2^-21.2 of the gate at most, about a quarter of it on average, some 2^-23 of the norm, beside ties 2^-8 to 2^-7 apart, so 2^-14 of them differ
    and 2^-13 are the limit (with the exponent's rounding left in, 2^-19.5 on average at these gates, 2^-12).  Beyond -87 a gate is 0 to 2^-126."""
    H, D = (16, 64) if kind == "wkv" else (8, 64)
    Dv, T = (64, 1000) if kind == "wkv" else (128, 1000)
    sc = Scan(kind, [T], H, D, Dv, seed=8)
    o, _ = sc.forced(ops, True)
    g = torch.Generator(device=DEV)
    g.manual_seed(9)
    gate = (torch.rand(T, H * Dv, generator=g, device=DEV) * -16 - 64).bfloat16()
    y, _ = sc.run(Gating(ops, (gate, None, 0.0, act)))
    x = o.double().view(T, H, Dv)
    x = (x / (x * x).mean(-1, keepdim=True).sqrt()).flatten(1)
    of = lambda gate: torch.sigmoid(gate.double()) * (gate.double() if act == "silu" else 1.0)
    assert (y != (x * of(gate)).bfloat16()).double().mean() <= 2.0 ** -13
    special = [float("inf"), -float("inf"), float("nan"), -87.0, -88.0, -89.0, -104.0, -3e38, 3e38, 88.0, 200.0, -0.0]
    gate[:] = torch.tensor((special * (H * Dv))[:H * Dv], device=DEV).bfloat16()
    y, _ = sc.run(Gating(ops, (gate, None, 0.0, act)))
    ref = ops.head_norm_gate(o, gate, None, H, Dv, 0.0, act)
    assert torch.equal(y.isnan(), ref.isnan()) and torch.equal(y.isinf(), ref.isinf()) and y.isinf().any() == (act == "silu")
    assert ((y.float() - ref.float()).abs() <= 2.0 ** -7 * ref.float().abs() + 1e-33)[ref.isfinite()].all()


@pytest.mark.parametrize("kind", KINDS)
def test_gated_in_passes_and_walked(ops, kind):  # noqa: F811
    """A step in passes: the same bits.  A walk: the pass over the read-outs, also for gates of 32 bits."""
    sc = Scan(kind, [500, 3, 260], 2, 64, 64, seed=4)
    gate = torch.randn(763, 128, device=DEV).bfloat16()
    gated = (gate, torch.rand(128, device=DEV), 1e-6, "silu")
    ops.scan_chunk_tokens = 1
    y, _ = sc.run(Gating(ops, gated))
    ops.scan_chunk_bytes = 3 * 2 * 64 * 64 * 4
    y2, _ = sc.run(Gating(ops, gated))
    assert torch.equal(y, y2)
    f32 = (gate.float(),) + gated[1:]
    o, _ = sc.run(ops)
    assert torch.equal(sc.run(Gating(ops, f32))[0], ops.head_norm_gate(o, f32[0], gated[1], 2, 64, 1e-6, "silu"))
    ops.scan_chunk_tokens = 1 << 30
    o, _ = sc.run(ops)
    assert torch.equal(sc.run(Gating(ops, gated))[0], ops.head_norm_gate(o, gate, gated[1], 2, 64, 1e-6, "silu"))
