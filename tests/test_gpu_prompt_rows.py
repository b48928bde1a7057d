"""The row kernels of prompt portions (wide loads, several values per thread) against 64 bits, at sizes they take and sizes they leave to
the general forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ops():
    from tiny_transformer_inference_engine_b200.ops import get_ops
    return get_ops(DEV)


def randn(seed, *shape):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV)


# one rounding to bfloat16 (2^-9 of the value) over a few 32-bit roundings
BF16 = dict(rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("T,H,Dv,weight,act", [(1, 1, 16, True, "silu"), (3, 3, 32, False, "sigmoid"), (67, 5, 64, True, "sigmoid"), (130, 2, 128, False, "silu"),
                                               (9, 3, 20, True, "silu"), (5, 2, 256, True, "silu")])
def test_head_norm_gate(ops, T, H, Dv, weight, act):
    o, wide = randn(1, T, H * Dv) * 3, randn(2, T, H * Dv + 8).bfloat16()
    gate = wide[:, 4:4 + H * Dv]
    w = randn(3, H * Dv) if weight else None
    got = ops.head_norm_gate(o, gate, w, H, Dv, 1e-6, act)
    x = o.double().view(T, H, Dv)
    x = (x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-6)).flatten(1)
    g = torch.sigmoid(gate.double()) * (gate.double() if act == "silu" else 1.0)
    assert torch.allclose(got.double(), x * (w.double() if weight else 1.0) * g, **BF16)


@pytest.mark.parametrize("style", [0, 1])
@pytest.mark.parametrize("T,heads,D,rot", [(65, 1, 8, 8), (70, 3, 128, 128), (67, 4, 64, 32), (66, 2, 48, 8), (90, 3, 24, 0), (9, 2, 20, 12), (6, 2, 40, 20), (64, 2, 64, 64)])
def test_rotate_heads(ops, T, heads, D, rot, style):
    src = randn(4, T, heads * D + 8).bfloat16()
    pos = torch.arange(T, dtype=torch.int32, device=DEV) * 37
    inv = (1.0 / 10000.0 ** (torch.arange(0, max(rot, 2), 2, device=DEV).float() / max(rot, 2)))
    cs = ops.rope_table(pos, inv) if rot else None
    got = ops.rotate_heads(src, heads, D, cs, rot, style, scale_from=1, scale=0.125)
    x = src[:, :heads * D].double().view(T, heads, D).clone()
    if rot:
        c, s = cs[..., 0].double()[:, None], cs[..., 1].double()[:, None]
        a, b = (x[..., 0:rot:2], x[..., 1:rot:2]) if style == 0 else (x[..., :rot // 2], x[..., rot // 2:rot])
        ra, rb = a * c - b * s, b * c + a * s
        if style == 0:
            x[..., 0:rot:2], x[..., 1:rot:2] = ra, rb
        else:
            x[..., :rot // 2], x[..., rot // 2:rot] = ra, rb
    x[:, 1:] *= 0.125
    assert torch.allclose(got.double().view(T, heads, D), x, rtol=1e-6, atol=1e-6)     # two products and a sum in 32 bits


@pytest.mark.parametrize("T,HD", [(1, 4), (67, 64), (5, 130), (3, 7)])
def test_wkv_decay(ops, T, HD):
    wide, w0 = randn(5, T, HD + 4) * 2, randn(6, HD)
    got = ops.wkv_decay(wide[:, :HD], w0)
    assert torch.allclose(got.double(), torch.exp(-torch.exp(wide[:, :HD].double() + w0.double())), rtol=1e-5, atol=1e-7)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("lens,I,N", [([1], 8, 16), ([7, 1, 9], 130, 16), ([64], 128, 4), ([65, 200], 129, 5), ([300], 40, 8), ([8, 16, 2], 7, 1), ([700, 3], 264, 13),
                                      ([2100], 16, 16)])
def test_selective_scan_forms(ops, lens, I, N, wide):
    """A thread per channel and a thread per four states, in one piece and in parts, against the recurrence in 64 bits.  Operands are
    bfloat16; decays come from the hardware's exponential (2^-22 each, whose errors add up over a state's memory)."""
    T, R, pad = sum(lens), len(lens), ops.selective_state_pad(N)
    u, z, low = randn(11, T, I).bfloat16(), randn(12, T, I + 8).bfloat16()[:, 8:], randn(13, T, 2 * N + 8).bfloat16()
    dt, bias, D, xin = randn(14, T, I), randn(15, I) - 4, randn(16, I), randn(17, T, I).bfloat16()
    A = torch.zeros(I, pad, device=DEV)
    A[:, :N] = -torch.exp(randn(18, I, N))
    S0 = torch.zeros(R + 1, I, pad, device=DEV)
    S0[..., :N] = randn(19, R + 1, I, N)
    tail0 = randn(20, R + 1, 3, I)
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    keep = ops.selective_wide_work
    ops.selective_wide_work = 0 if wide else 1 << 60
    S, tail = S0.clone(), tail0.clone()
    try:
        got = ops.selective_scan(u, dt, bias, A, D, low, 8, 8 + N, z, S, xin, tail, 4, t(qsl), t(list(range(R))[::-1]), R, N)
    finally:
        ops.selective_wide_work = keep
    d = torch.nn.functional.softplus(dt.double() + bias.double())
    for r in range(R):
        slot = R - 1 - r
        s = S0[slot, :, :N].double()
        for k in range(qsl[r], qsl[r + 1]):
            s = torch.exp(d[k][:, None] * A[:, :N].double()) * s + (d[k] * u[k].double())[:, None] * low[k, 8:8 + N].double()
            y = s @ low[k, 8 + N:8 + 2 * N].double() + D.double() * u[k].double()
            e = y * z[k].double() * torch.sigmoid(z[k].double())
            assert torch.allclose(got[k].double(), e, rtol=2.0 ** -7, atol=2e-2 * float(e.abs().max()) / 10), (r, k)
        assert ((S[slot, :, :N].double() - s).norm() / s.norm()).item() < 2e-5
        want = torch.cat([tail0[slot].double(), xin[qsl[r]:qsl[r + 1]].double()])[-3:]
        assert torch.equal(tail[slot].double(), want)
    assert torch.equal(S[R], S0[R])


@pytest.mark.parametrize("lens,I,N", [([1] * 23 + [700], 264, 16), ([1, 64, 65, 1, 500], 130, 8), ([3] * 40 + [130], 40, 4), ([128] * 5, 72, 13)])
def test_selective_scan_of_a_mixed_step_in_parts(ops, monkeypatch, lens, I, N):
    """Decoding requests beside a portion that is walked in parts, with a thread per channel, when the longest request is known: the form with
    a thread per four states gives the same (one rounding to bfloat16 apart; states to 2e-5, whose decays come from the hardware's exponential)."""
    T, R, pad = sum(lens), len(lens), ops.selective_state_pad(N)
    u, z, low = randn(21, T, I).bfloat16(), randn(22, T, I).bfloat16(), randn(23, T, 2 * N).bfloat16()
    dt, bias, D, xin = randn(24, T, I), randn(25, I) - 4, randn(26, I), randn(27, T, I).bfloat16()
    A = torch.zeros(I, pad, device=DEV)
    A[:, :N] = -torch.exp(randn(28, I, N))
    S0, tail0 = torch.zeros(R + 1, I, pad, device=DEV), randn(30, R + 1, 3, I)
    S0[..., :N] = randn(29, R + 1, I, N)
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    monkeypatch.setattr(ops, "selective_wide_full", 0.0)
    got = []
    for work in (0, 1 << 60):
        monkeypatch.setattr(ops, "selective_wide_work", work)
        wide = ops.selective_wide(torch.bfloat16, T, R, I, N, max(lens))
        assert wide is (work == 0)
        if wide:
            monkeypatch.setattr(ops, "selective_wide_full", 1e9)      # (parts, however few warps there are)
            assert ops.selective_parts(T, R, I, N, True, max(lens)) > 1
        S, tail = S0.clone(), tail0.clone()
        monkeypatch.setattr(ops, "selective_wide", lambda *a: wide)
        got.append((ops.selective_scan(u, dt, bias, A, D, low, 0, N, z, S, xin, tail, 4, t(qsl), t(list(range(R))[::-1]), R, N, max_q_len=max(lens)), S, tail))
        monkeypatch.delattr(ops, "selective_wide")
    (y, S, tail), (y2, S2, tail2) = got
    assert torch.allclose(y.double(), y2.double(), rtol=2.0 ** -7, atol=2e-3 * float(y2.abs().max()))
    assert ((S - S2).norm() / S2.norm()).item() < 2e-5 and torch.equal(tail, tail2)


@pytest.mark.parametrize("lens,I,N,parts", [([2048], 1024, 16, 7), ([1] * 23 + [520], 136, 16, 4), ([259, 64, 65], 132, 16, 4), ([200, 8, 300], 130, 7, 3),
                                            ([71, 1, 136], 127, 4, 2), ([64 * 5 + 1], 260, 16, 5)])
def test_selective_scan_with_a_thread_per_channel_at_its_edges(ops, monkeypatch, lens, I, N, parts):
    """Rows on 16, 8, 4 and 2 bytes, runs of fewer than eight tokens, channels past the last whole CTA, parts whose last one is short, and the
    last request placed first, against the form with a thread per four states (bfloat16 outputs one rounding apart; states to 2e-5, whose decays come
    from the hardware's exponential)."""
    T, R, pad = sum(lens), len(lens), ops.selective_state_pad(N)
    u, z, low = randn(41, T, I).bfloat16(), randn(42, T, 2 * I).bfloat16()[:, I:], randn(43, T, 2 * N).bfloat16()
    dt, bias, D, xin = randn(44, T, I), randn(45, I) - 4, randn(46, I), randn(47, T, I).bfloat16()
    A = torch.zeros(I, pad, device=DEV)
    A[:, :N] = -torch.exp(randn(48, I, N))
    S0, tail0 = torch.zeros(R + 1, I, pad, device=DEV), randn(50, R + 1, 3, I)
    S0[..., :N] = randn(49, R + 1, I, N)
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    import tiny_transformer_inference_engine_b200.ops as module
    got = []
    for wide in (True, False):
        with monkeypatch.context() as m:
            m.setattr(ops, "selective_wide", lambda *a: wide)
            if wide:
                m.setattr(ops, "selective_parts", lambda *a: parts)
                m.setattr(module, "_even_parts", lambda *a: parts)
            S, tail = S0.clone(), tail0.clone()
            got.append((ops.selective_scan(u, dt, bias, A, D, low, 0, N, z, S, xin, tail, 4, t(qsl), t(list(range(R))[::-1]), R, N, max_q_len=max(lens)), S, tail))
    (y, S, tail), (y2, S2, tail2) = got
    assert torch.allclose(y.double(), y2.double(), rtol=2.0 ** -7, atol=2e-3 * float(y2.abs().max()))
    assert ((S - S2).norm() / S2.norm()).item() < 2e-5 and torch.equal(tail, tail2) and torch.equal(S[R], S0[R])


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("lens,width,wdtype", [([1027], 1024, torch.float32), ([1, 2, 3, 1, 700, 2, 400], 1032, torch.float32), ([5] * 60, 4096, torch.bfloat16), ([130], 8200, torch.bfloat16)])
def test_causal_conv_in_runs_of_tokens(ops, lens, width, wdtype, taps):
    """Runs that start inside a request, cross requests and end short, behind state rows, with and without silu and bias; 32-bit sums of five terms
    (2^-23 each of the largest) and one rounding to bfloat16."""
    T, R = sum(lens), len(lens)
    assert T * width >= 1 << 20
    x = randn(51, T, width + 8).bfloat16()
    w, b = randn(52, taps, width).to(wdtype), randn(53, width).to(wdtype)
    state = randn(54, R + 1, max(1, taps - 1), width)
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    seq = t([r for r, n in enumerate(lens) for _ in range(n)])
    rows = torch.cat([torch.cat([state[R - 1 - r, :taps - 1].double(), x[qsl[r]:qsl[r + 1], 8:].double()]).unfold(0, taps, 1) for r in range(R)])
    terms = rows * w.double().t()
    for bias, act in ((b, "silu"), (None, None), (None, "silu")):
        u32, u = ops.causal_conv(x, 8, width, taps, w, bias, state, seq, t(qsl), t(list(range(R))[::-1]), True, first_row=0, act=act, want_f32=act is None)
        e = terms.sum(-1) + (bias.double() if bias is not None else 0.0)
        slack = 5 * 2.0 ** -23 * (terms.abs().sum(-1) + (bias.double().abs() if bias is not None else 0.0))
        if u32 is not None:
            assert ((u32.double() - e).abs() <= slack).all()
        y = e * torch.sigmoid(e) if act else e
        assert ((u.double() - y).abs() <= 2.0 ** -8 * y.abs() + 2 * slack + 1e-6).all()


def test_causal_conv_silu_of_large_sums(ops):
    """One tap: the sum is one rounded product, and silu of it is rounded correctly but where the exact value lies within the function's 32-bit
    error of a tie (2^-21.2 at most, about a quarter of it on average, beside ties 2^-8 to 2^-7 apart: 2^-15 of them, 2^-13 are the limit; with
    the exponent's rounding left in, 2^-19.5 on average at -80 to -64, 2^-12).  Beyond -87 it is 0 to 2^-119; what is not finite as in the general form."""
    T, W = 1024, 1024
    x = randn(61, T, W)
    x[:, ::2] = x[:, ::2].abs().clamp(max=1.0) * -16 - 64
    special = torch.tensor([float("inf"), -float("inf"), float("nan"), -88.5, -104.0, -3e38, 3e38, 88.5, -0.0], device=DEV)
    x[5, :9], x[1023, :9] = special, special
    x, w = x.bfloat16(), 1 + 0.1 * randn(62, 1, W)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    conv = lambda x, T: ops.causal_conv(x, 0, W, 1, w, None, torch.zeros(1, 1, W, device=DEV), t([0] * T), t([0, T]), t([0]), True,
                                        first_row=0, act="silu", want_f32=False)[1]
    got, x32 = conv(x, T), x.float() * w
    exact = x32.double() * torch.sigmoid(x32.double())
    assert (got != exact.bfloat16())[(x32 > -87) & (x32 <= -64)].double().mean() <= 2.0 ** -13
    assert (got.double() - exact)[x.isfinite()].abs().le(2.0 ** -8 * exact.abs()[x.isfinite()] + 2.0 ** -119).all()
    general = conv(x[1020:].contiguous(), 4)
    assert torch.equal(got[1020:].isnan(), general.isnan()) and torch.equal(got[1020:].isinf(), general.isinf())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,d,off", [(1, 8, 0), (3, 12, 0), (5, 1032, 0), (2, 4104, 8), (4, 100, 0), (3, 64, 1), (70, 516, 4)])
def test_embed_forms(ops, T, d, off, dtype):
    """Rows that fill their last piece and not, tables on 16 bytes and off them, ids past either end: one 32-bit multiplication, exactly."""
    V = 50
    table = randn(61, V * d + off).to(dtype)[off:].view(V, d)
    ids = torch.randint(0, V, (T,), dtype=torch.int32, device=DEV)
    ids[0], ids[-1] = -3, V + 7
    out = torch.empty(T, d, device=DEV)
    ops.embed(ids, table, out, scale=1.7)
    assert torch.equal(out, table[ids.clamp(0, V - 1).long()].float() * 1.7)
