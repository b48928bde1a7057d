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
