"""The matrix-state recurrences over prompts in chunks of 64 tokens on tensor cores, against the token-by-token recurrence in 64 bits, and
against the walk that decoded tokens run."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture()
def ops():
    from tiny_transformer_inference_engine_b200.ops import get_ops
    o = get_ops(DEV)
    keep = o.scan_chunk_tokens, o.scan_chunk_more, o.scan_chunk_bytes
    o.scan_chunk_more = 0
    yield o
    o.scan_chunk_tokens, o.scan_chunk_more, o.scan_chunk_bytes = keep


def step_tensors(lens):
    qsl = [0]
    for n in lens:
        qsl.append(qsl[-1] + n)
    slots = [(2 * i + 1) % (len(lens) + 1) for i in range(len(lens))] if len(lens) % 2 == 0 else list(range(len(lens)))[::-1]
    return torch.tensor(qsl, dtype=torch.int32, device=DEV), torch.tensor(slots, dtype=torch.int32, device=DEV), qsl, slots


class Scan:
    """One kind of recurrence on random inputs: run(ops) -> (out, state tensors), exact() the same in 64 bits."""

    def __init__(self, kind, lens, H, D, Dv, seed=0, strong=False, values=torch.bfloat16):
        self.kind, self.lens, self.H, self.D, self.Dv = kind, lens, H, D, Dv
        g = torch.Generator(device=DEV)
        g.manual_seed(seed)
        T, R = sum(lens), len(lens) + 2
        rn = lambda *s: torch.randn(s, generator=g, device=DEV)
        self.qsl, self.slots, self.q_at, self.s_at = step_tensors(lens)
        P = 4
        while P < D:
            P *= 2
        self.S0 = torch.zeros(R, H, Dv, P, device=DEV)
        self.S0[..., :D] = rn(R, H, Dv, D) * 0.5
        if kind == "retention":
            self.qk = rn(T, 2 * H * D) * torch.cat([torch.ones(H * D), torch.full((H * D,), D ** -0.5)]).to(DEV)
            self.q, self.k = self.qk[:, :H * D], self.qk[:, H * D:]
            self.v = rn(T, H * Dv).to(values)
            base = [1.0, 0.0, 0.5, -0.7] if strong else [1 - 2.0 ** (-5 - i % 4) for i in range(H)]
            self.decay = torch.tensor([base[i % len(base)] for i in range(H)], device=DEV)
        elif kind == "mlstm":
            proj = rn(T, 2 * H * D + H * Dv).bfloat16()
            self.q, self.k, self.v = proj[:, :H * D], proj[:, H * D:2 * H * D], proj[:, 2 * H * D:]
            self.pre = rn(T, 2 * H) * (15.0 if strong else 1.5) + torch.cat([torch.zeros(H), torch.linspace(1, 6, H)]).to(DEV)
            self.n0, self.m0 = torch.zeros(R, H, P, device=DEV), rn(R, H)
            self.n0[..., :D] = rn(R, H, D)
        else:
            proj = rn(3, T, H * D).bfloat16()
            self.q, self.k, self.v = proj
            self.w = torch.exp(-torch.exp(torch.rand(T, H * D, generator=g, device=DEV) * (13.0 if strong else 6.5) - (8.0 if strong else 6.0)))
            self.u, self.x, self.prev0 = rn(H * D) * 0.5, rn(T, 40).bfloat16(), rn(R, 40)

    def forced(self, ops, chunks):
        """run() in chunks or token by token, and sure of it."""
        ops.scan_chunk_tokens = 1 if chunks else 1 << 30
        mode = ["retention", "mlstm", "wkv"].index(self.kind)
        assert ops._in_chunks(mode, sum(self.lens), len(self.lens), None, self.H, self.D, self.Dv, self.q, self.k, self.v) is chunks
        before = ops.launches
        result = self.run(ops)
        self.launched = ops.launches - before
        assert self.launched >= 3 if chunks else self.launched <= 2
        return result

    def run(self, ops):
        H, D, Dv, N = self.H, self.D, self.Dv, len(self.lens)
        S = self.S0.clone()
        if self.kind == "retention":
            return ops.retention_scan(self.q, self.k, self.v, self.decay, S, self.qsl, self.slots, N, H, D, Dv), [S]
        if self.kind == "mlstm":
            n, m = self.n0.clone(), self.m0.clone()
            if ops.mlstm_in_chunks(self.q, self.k, self.v, N, D, Dv):
                return ops.mlstm_chunks(self.q, self.k, self.v, self.pre, S, n, m, self.qsl, self.slots, N, H, D, Dv, 15.0, D ** -0.5), [S, n, m]
            w, before = ops.mlstm_gates(self.pre, m, n, self.qsl, self.slots, N, H, 15.0)
            return ops.mlstm_scan(self.q, self.k, self.v, w, S, n, before, self.qsl, self.slots, N, H, D, Dv, D ** -0.5), [S, n, m]
        prev = self.prev0.clone()
        return ops.wkv_scan(self.q, self.k, self.v, self.w, self.u, S, self.x, prev, self.qsl, self.slots, N, H, D), [S, prev]

    def exact(self):
        H, D, Dv = self.H, self.D, self.Dv
        heads = lambda x, d: x.double().reshape(x.shape[0], H, d)
        q, k, v = heads(self.q, D), heads(self.k, D), heads(self.v, Dv)
        out, S_all = torch.empty(q.shape[0], H, Dv, dtype=torch.float64, device=DEV), self.S0.double()
        n_all = m_all = None
        self.near = torch.zeros(q.shape[0], H, dtype=torch.bool, device=DEV)   # rows that divide by a sum that nearly cancels
        if self.kind == "mlstm":
            n_all, m_all = self.n0.double(), self.m0.double()
            ig = 15.0 * torch.tanh(self.pre[:, :H].double() / 15.0)
            fg = torch.nn.functional.logsigmoid(15.0 * torch.tanh(self.pre[:, H:].double() / 15.0))
        for r, slot in enumerate(self.s_at):
            S = S_all[slot, :, :, :D]
            for t in range(self.q_at[r], self.q_at[r + 1]):
                kv = v[t][:, :, None] * k[t][:, None, :]
                if self.kind == "retention":
                    S = S * self.decay.double()[:, None, None] + kv
                    out[t] = (S @ q[t][:, :, None])[..., 0]
                elif self.kind == "wkv":
                    out[t] = ((S + heads(self.u[None], D)[0][:, None, :] * kv) @ q[t][:, :, None])[..., 0]
                    S = S * heads(self.w[t:t + 1], D)[0][:, None, :] + kv
                else:
                    n, m = n_all[slot, :, :D], m_all[slot]
                    m1 = torch.maximum(fg[t] + m, ig[t])
                    a, b = torch.exp(fg[t] + m - m1)[:, None], torch.exp(ig[t] - m1)[:, None]
                    S, n = a[..., None] * S + b[..., None] * kv, a * n + b * k[t]
                    qs = q[t] * D ** -0.5
                    den = torch.maximum((n * qs).sum(-1).abs(), torch.exp(-m1)) + 1e-6
                    self.near[t] = den < 0.02 * n.norm(dim=-1) * qs.norm(dim=-1)
                    out[t] = (S @ qs[:, :, None])[..., 0] / den[:, None]
                    n_all[slot, :, :D], m_all[slot] = n, m1
            S_all[slot, :, :, :D] = S
        return out.flatten(1), [S_all] + ([n_all, m_all] if self.kind == "mlstm" else [])


def rel(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


KINDS = ["retention", "mlstm", "wkv"]
SIZES = [([64], 2, 64, 64), ([65, 1], 3, 128, 128), ([63, 1, 130], 2, 48, 72), ([300], 4, 8, 8), ([1, 200, 2, 17], 1, 128, 136), ([129, 127], 2, 24, 16),
         ([1000], 4, 64, 128)]


@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("lens,H,D,Dv", SIZES)
@pytest.mark.parametrize("kind", KINDS)
def test_chunks_against_64_bits(ops, kind, lens, H, D, Dv, strong):
    """Whole and partial chunks, one and several requests, heads that do not fill a tile, decays from none to ones that leave nothing
    (negative and zero ones too).  The bound: a read-out adds up some hundreds of products whose factors carry a few
    roundings each, 2^-24 apart.  The matrix memory divides by a sum that can nearly cancel, which multiplies the error of that row:
    rows whose divisor is below 2 % of what it could be are left out, the others' error may be fifty times as large."""
    if kind == "wkv":
        Dv = D
    sc = Scan(kind, lens, H, D, Dv, seed=len(lens) + D, strong=strong)
    out, states = sc.forced(ops, True)
    exp, exp_states = sc.exact()
    bound = 2e-5 if kind == "mlstm" else 1e-6
    rows = lambda x: x.double().view(-1, H, Dv)[~sc.near]
    assert sc.near.float().mean() < 0.25
    assert rel(rows(out), rows(exp)) < bound
    for s, e in zip(states, exp_states):
        assert rel(s, e) < 1e-6
    walk, walk_states = sc.forced(ops, False)
    assert rel(rows(walk), rows(exp)) < bound
    for s, e in zip(walk_states, exp_states):                         # (mlstm's walk has its weights from 32-bit sums of 32 log gates of up to 15, off by 480 * 2^-25 = 1.4e-5)
        assert rel(s, e) < (bound if kind == "mlstm" else 1e-6)
    if kind == "wkv":
        assert torch.equal(states[1], walk_states[1])                 # the request's last input
    print(kind, lens, D, Dv, strong, "out %.3g %.3g" % (rel(rows(out), rows(exp)), rel(rows(walk), rows(exp))),
          "states", ["%.3g" % rel(s, e) for s, e in zip(states, exp_states)], ["%.3g" % rel(s, e) for s, e in zip(walk_states, exp_states)])


def test_retention_chunks_with_32_bit_values(ops):
    sc = Scan("retention", [200, 70], 2, 128, 128, seed=9, values=torch.float32)
    out, (S,) = sc.forced(ops, True)
    exp, (e,) = sc.exact()
    assert rel(out, exp) < 1e-6 and rel(S, e) < 1e-6


@pytest.mark.parametrize("kind", KINDS)
def test_chunks_in_passes(ops, kind):
    """A step whose states between chunks do not fit the workspace runs in passes that carry the state rows on: the same bits."""
    sc = Scan(kind, [500, 3, 260], 2, 64, 64, seed=4)
    out, states = sc.forced(ops, True)
    ops.scan_chunk_bytes = 3 * 2 * 64 * 64 * 4
    out2, states2 = sc.forced(ops, True)
    assert sc.launched > 3                                            # more than one pass
    assert torch.equal(out, out2) and all(torch.equal(a, b) for a, b in zip(states, states2))


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("what", ["v", "k"])
def test_what_is_not_finite_stays_behind(ops, kind, what):
    """A value or key that is not finite reaches its own and later tokens of its request; earlier tokens and other requests are as if
    it were not there."""
    lens, at = [150, 40], 75
    for bad in (float("inf"), float("nan")):
        sc, clean = Scan(kind, lens, 2, 64, 64, seed=5), Scan(kind, lens, 2, 64, 64, seed=5)
        getattr(sc, what)[at, 70] = bad
        out, states = sc.forced(ops, True)
        ref, _ = clean.run(ops)
        # (the read-outs of a chunk in which something is not finite are computed token by token: other roundings)
        assert torch.allclose(out[:at], ref[:at], rtol=1e-5, atol=1e-5) and torch.equal(out[150:], ref[150:])
        assert not torch.isfinite(out[at + 1:150, 64:]).all()
        walk, walk_states = sc.forced(ops, False)
        assert torch.equal(torch.isfinite(out), torch.isfinite(walk))
        assert torch.equal(torch.isfinite(states[0]), torch.isfinite(walk_states[0]))


def class_of(x):
    return torch.where(x.isnan(), 3, torch.where(x == float("inf"), 1, torch.where(x == float("-inf"), 2, 0)))


@pytest.mark.parametrize("D,Dv", [(64, 64), (48, 136), (128, 128)])
@pytest.mark.parametrize("what", ["v", "k", "q", "S0"])
@pytest.mark.parametrize("kind", KINDS)
def test_what_is_not_finite_comes_out_as_the_walk_has_it(ops, kind, what, D, Dv):
    """Infinities of either sign and NaN, brought by a token or found in the state row: the same infinities and NaN in every read-out and
    state element as token by token, and the same values elsewhere."""
    if kind == "wkv":
        Dv = D
    for bad in (float("inf"), float("-inf"), float("nan")):
        sc = Scan(kind, [150, 40, 9], 2, D, Dv, seed=6)
        if what == "S0":
            sc.S0[sc.s_at[0], 1, 3, 5] = bad
        else:
            getattr(sc, what)[75, (Dv if what == "v" else D) + 6] = bad
        out, states = sc.forced(ops, True)
        walk, walk_states = sc.forced(ops, False)
        for got, want in zip([out] + states, [walk] + walk_states):
            assert torch.equal(class_of(got), class_of(want)), (bad, got.shape)
            fine = want.isfinite()
            assert torch.allclose(got[fine], want[fine], rtol=1e-2, atol=1e-3)
        assert not out.isfinite().all()


def test_retention_chunks_near_the_largest_number(ops):
    """Keys that round to an infinite bfloat16 and are finite themselves: no plane form, the same sums."""
    sc = Scan("retention", [150], 2, 64, 64, seed=8, values=torch.float32)
    sc.k[75, 64 + 6], sc.k[140, 9] = 3.395e38, -3.39e38
    sc.v[75], sc.v[140] = 2.0 ** -3, 2.0 ** -4
    sc.q.mul_(2.0 ** -6)
    out, (S,) = sc.forced(ops, True)
    exp, (e,) = sc.exact()
    assert out.isfinite().all() and S.isfinite().all()
    assert rel(out * 2.0 ** -100, exp * 2.0 ** -100) < 1e-6 and rel(S * 2.0 ** -100, e * 2.0 ** -100) < 1e-6


@pytest.mark.parametrize("lens", [[1000], [40], [129, 5, 127]])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lo,hi", [(0.0, 3.0), (-8.0, 5.0), (-6.0, 0.5), (-8.0, -6.0)])
def test_wkv_state_is_no_further_off_than_the_walks(ops, lens, D, lo, hi):
    """Decays exp(-exp(x)), x between lo and hi: from ones that leave the last token alone to ones that forget little.  The walk rounds once a
    token and ends with a rounding that nothing can spare; the chunks' state may not be further from 64 bits (a tenth for chance)."""
    sc = Scan("wkv", lens, 4, D, D, seed=7)
    g = torch.Generator(device=DEV)
    g.manual_seed(8)
    sc.w = torch.exp(-torch.exp(torch.rand(sc.w.shape, generator=g, device=DEV) * (hi - lo) + lo))
    out, states = sc.forced(ops, True)
    exp, exp_states = sc.exact()
    walk, walk_states = sc.forced(ops, False)
    assert rel(states[0], exp_states[0]) < 1.1 * rel(walk_states[0], exp_states[0])
    assert rel(out, exp) < 1.1 * rel(walk, exp)


# whole and partial chunks of 128, requests of one token, heads of one piece of 8 channels up to a full tile, padded keys
@pytest.mark.parametrize("strong", [False, True])
@pytest.mark.parametrize("lens,H,D,Dv", [([128], 2, 128, 128), ([129, 127], 3, 64, 128), ([1, 255, 2], 2, 40, 104), ([300], 2, 8, 8), ([64, 1, 130], 1, 96, 64), ([1000], 2, 128, 120)])
@pytest.mark.parametrize("kind", ["retention", "mlstm"])
def test_chunks_of_128_tokens_against_64_bits(ops, monkeypatch, kind, lens, H, D, Dv, strong):
    """The tcgen05 form against 64 bits and against the chunks of 64 tokens; bounds as above, and no further from 64 bits than the
    walk (the matrix memory under strong gates, where single rows that nearly cancel decide, apart)."""
    sc = Scan(kind, lens, H, D, Dv, seed=len(lens) + D, strong=strong)
    exp, exp_states = sc.exact()
    rows = lambda x: x.double().view(-1, H, Dv)[~sc.near]
    results = {}
    for tokens in (64, 128):
        monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a: tokens))
        results[tokens] = sc.forced(ops, True)
    walk, walk_states = sc.forced(ops, False)
    bound = 2e-5 if kind == "mlstm" else 1e-6
    for out, states in results.values():
        assert rel(rows(out), rows(exp)) < bound
        for s, e in zip(states, exp_states):
            assert rel(s, e) < 1e-6
    out, states = results[128]
    if kind == "retention":
        assert rel(out, exp) < 1.2 * max(rel(walk, exp), rel(results[64][0], exp))
    # (the matrix state: the normaliser's and the maximum's few numbers are a rounding off or not)
    assert rel(states[0], exp_states[0]) < 1.2 * max(rel(walk_states[0], exp_states[0]), rel(results[64][1][0], exp_states[0]))
    assert ops.lib.ttie_tc_error() == 0


@pytest.mark.parametrize("tokens", [64, 128])
@pytest.mark.parametrize("kind", ["retention", "mlstm"])
def test_chunks_in_passes_carry_on(ops, monkeypatch, kind, tokens):
    """Room for two chunks' states: a step of 700 tokens runs in passes, with the state between them."""
    monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a: tokens))
    sc = Scan(kind, [500, 200], 2, 64, 128, seed=4)
    once, states = sc.forced(ops, True)
    ops.scan_chunk_bytes = 2 * 2 * 64 * 128 * 4
    passes, pass_states = sc.forced(ops, True)
    assert sc.launched > 3
    assert rel(passes, once.double()) < 1e-5 and all(rel(a, b.double()) < 1e-6 for a, b in zip(pass_states, states))


@pytest.mark.parametrize("lens", [[1], [130], [300, 5]])
@pytest.mark.parametrize("D,Dv", [(8, 128), (64, 128), (128, 128), (128, 72)])
@pytest.mark.parametrize("tokens", [64, 128])
def test_sums_that_32_bits_hold_come_out_exactly(ops, monkeypatch, tokens, D, Dv, lens):
    """Retention that forgets nothing, of small whole numbers: every partial sum is one below 2^24, so the read-outs and the state are exact."""
    monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a: tokens))
    sc = Scan("retention", lens, 2, D, Dv, seed=D + len(lens))
    for t in (sc.qk, sc.v, sc.S0):
        t.copy_((t * 2).round().clamp(-3, 3))
    sc.qk[:, 2 * D:].copy_((torch.randn(sum(lens), 2 * D, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1)) * 2).round().clamp(-3, 3))
    sc.decay.fill_(1.0)
    exp, exp_states = sc.exact()
    assert exp.abs().max() < 2 ** 24
    out, states = sc.forced(ops, True)
    assert torch.equal(out.double(), exp) and torch.equal(states[0].double(), exp_states[0])


@pytest.mark.parametrize("kind,D,Dv", [("retention", 128, 128), ("retention", 64, 128), ("retention", 16, 128), ("mlstm", 64, 128), ("mlstm", 128, 128)])
def test_chunks_of_128_tokens_are_no_further_off_than_chunks_of_64(ops, monkeypatch, kind, D, Dv):
    """Error against 64 bits of read-outs and state, mean of six inputs (one input's mean is good to some percent: 4 % allowed)."""
    err = {64: [0.0, 0.0], 128: [0.0, 0.0]}
    for seed in range(6):
        sc = Scan(kind, [700, 130], 2, D, Dv, seed=seed)
        exp, exp_states = sc.exact()
        rows = lambda x: x.double().view(-1, 2, Dv)[~sc.near]
        for tokens in err:
            monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a, n=tokens: n))
            out, states = sc.forced(ops, True)
            err[tokens][0] += rel(rows(out), rows(exp))
            err[tokens][1] += rel(states[0], exp_states[0])
    assert err[128][0] < 1.04 * err[64][0] and err[128][1] < 1.04 * err[64][1], err


@pytest.mark.parametrize("odd", [False, True])
def test_gate_bias_added_in_the_chunks(ops, monkeypatch, odd):
    """The matrix memory with the gates' bias read in its kernels against the same bias added to the pre-activations before: the same 32-bit sums, so
    the same to the last bit; also where a chunk and the states behind it are not finite and are walked.  And against 64 bits."""
    monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a: 128))
    H, D, Dv = 3, 64, 128
    sc = Scan("mlstm", [300, 7, 130], H, D, Dv, seed=9)
    bias = torch.cat([torch.linspace(-1.3, 2.1, H), torch.linspace(3.0, -0.7, H)]).bfloat16().to(DEV)      # input gates, forget gates
    if odd:
        sc.v[150, 5], sc.v[310, 200] = float("inf"), float("nan")
    ops.scan_chunk_tokens = 1
    added = sc.pre + bias.float()
    results = []
    for pre, b in ((sc.pre, bias), (added, None)):
        S, n, m = sc.S0.clone(), sc.n0.clone(), sc.m0.clone()
        out = ops.mlstm_chunks(sc.q, sc.k, sc.v, pre, S, n, m, sc.qsl, sc.slots, 3, H, D, Dv, 15.0, D ** -0.5, pre_bias=b)
        results.append((out, S, n, m))
    for a, b in zip(*results):
        assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    assert torch.isfinite(results[0][0]).all() != odd
    if not odd:
        sc.pre = added
        exp, exp_states = sc.exact()
        rows = lambda x: x.double().view(-1, H, Dv)[~sc.near]
        assert rel(rows(results[0][0]), rows(exp)) < 2e-6
        for s, e in zip(results[0][1:], exp_states):
            assert rel(s, e) < 1e-6


def test_gate_bias_is_refused_by_chunks_of_64(ops, monkeypatch):
    from tiny_transformer_inference_engine_b200.ops import KernelError
    monkeypatch.setattr(type(ops), "_chunk_tokens", staticmethod(lambda *a: 64))
    ops.scan_chunk_tokens = 1
    sc = Scan("mlstm", [200], 2, 64, 128)
    with pytest.raises(KernelError, match="gate bias"):
        ops.mlstm_chunks(sc.q, sc.k, sc.v, sc.pre, sc.S0, sc.n0, sc.m0, sc.qsl, sc.slots, 1, 2, 64, 128, 15.0, 0.125, pre_bias=torch.zeros(4, dtype=torch.bfloat16, device=DEV))


@pytest.mark.parametrize("lens", [[256], [1, 300, 200]])
def test_mlstm_layer_hands_its_gate_bias_to_the_chunks(ops, monkeypatch, lens):
    """The layer over a prompt in chunks of 128 tokens: it leaves the bias to the chunks, and gives what it gives with the bias in the product."""
    from test_gpu_mizupel import part_with_weights, ctx_for, rel_norm, pm
    from tiny_transformer_inference_engine_b200.parts.base import FixedStateView, PartSpec
    heads, dim, vdim, d = 2, 64, 128, 64
    spec = PartSpec("mlstm", "", {"d_model": d, "num_heads": heads, "dim": dim, "vdim": vdim, "gate_cap": 15.0, "eps": 1e-5})
    part, w = part_with_weights("mixer", spec, "bfloat16", ops, 5, scale=0.2, scales={"i": 0.5, "f": 0.5, "i.b": 1.0, "f.b": 2.0})
    assert len(set(part.b_gates.tolist())) == 2 * heads
    x = torch.randn(sum(lens), d, generator=torch.Generator().manual_seed(3)).bfloat16()
    ops.scan_chunk_tokens = 1
    took, results = [], []
    adds = type(ops).mlstm_adds_bias
    for answer in (adds, lambda *a: False):
        monkeypatch.setattr(type(ops), "mlstm_adds_bias", lambda *a, f=answer: took.append(f(*a)) or took[-1])
        states = [torch.zeros(len(lens) + 1, *need.shape, device=DEV) for need in part.cache_needs()]
        y = part.forward(x.to(DEV), ctx_for(ops, torch.bfloat16, [(0, n) for n in lens], None, slots=list(range(len(lens)))), [FixedStateView(s) for s in states])
        results.append([y.sum(0) if y.dim() == 3 else y] + states)
    assert took == [True, False]
    assert all(torch.equal(a, b) for a, b in zip(*results))
    at = 0
    for n in lens:
        exp = pm.mlstm(x[at:at + n].double(), w, "", {"heads": heads, "dim": dim, "vdim": vdim, "gate_cap": 15.0}, 1e-5)
        assert rel_norm(results[0][0][at:at + n], exp) < 3e-2
        at += n
