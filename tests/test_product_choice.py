"""Which form a product or a scan takes: by the sizes of the step alone."""
import random

import pytest
import torch

from tiny_transformer_inference_engine_b200.ops import CudaOps, _even_parts, _floor_sum, _ring_form


@pytest.mark.parametrize("rows,hidden,K,fused", [
    (2048, 11008, 4096, True), (1024, 11008, 4096, True), (4096, 18176, 4544, True), (2048, 16384, 2048, True), (2048, 8192, 2048, True),
    (2000, 11008, 4096, False), (2047, 16384, 2048, False), (1300, 18176, 4544, False), (5000, 18176, 4544, True),      # ragged last tiles
    (768, 16384, 2048, False), (1023, 16384, 2048, False),                                                            # fewer than 1,024 rows
    (1280, 4096, 4096, False), (1024, 8192, 2048, False), (2048, 8192, 1024, False), (8192, 4096, 1024, False),      # few waves, small K
])
def test_gate_up_form_by_sizes(rows, hidden, K, fused):
    assert CudaOps._fused_swiglu_wins(148, rows, hidden, K) is fused


RETENTION, MLSTM, WKV = 0, 1, 2


def in_chunks(mode, lens, width, known=True, dtype=torch.bfloat16, dim=None, stride=0, at=0):
    """The decision for a step of requests that bring these many tokens, at the layer sizes of a width."""
    heads, k, v = {RETENTION: (width // 128, 128, 128), MLSTM: (width // 128, 64, 128), WKV: (width // 64, 64, 64)}[mode]
    k = dim or k
    T = sum(lens)
    qk_type = torch.float32 if mode == RETENTION else dtype
    rows = lambda n, t: torch.empty_strided((T, n), (n + stride, 1), dtype=t)
    q, vals = rows(heads * k + at, qk_type)[:, at:], rows(heads * v, dtype)
    ops = CudaOps.__new__(CudaOps)
    return ops._in_chunks(mode, T, len(lens), max(lens) if known else None, heads, k, v, q, q, vals)


# (what a step brings, kind, width) and whether chunks were measured ahead by enough to pay for their call
@pytest.mark.parametrize("mode,lens,width,chunks", [
    (RETENTION, [128], 2048, False), (RETENTION, [512], 2048, True), (RETENTION, [192], 512, False), (RETENTION, [2048], 1024, True),
    (MLSTM, [128], 2048, False), (MLSTM, [256], 2048, False), (MLSTM, [400], 2048, True), (WKV, [160], 2048, False), (WKV, [512], 2048, True), (WKV, [300], 1024, False), (WKV, [500], 1024, True), (RETENTION, [300], 1024, True),
    (RETENTION, [16] * 8, 2048, False), (RETENTION, [32] * 8, 512, False), (MLSTM, [32] * 8, 2048, False), (WKV, [64] * 8, 1024, False),      # short prompts
    (RETENTION, [64] * 8, 2048, True), (MLSTM, [128] * 8, 2048, True), (RETENTION, [128] * 24, 1024, True),                # many: work, not length
    (RETENTION, [1] * 23 + [192], 2048, False), (WKV, [1] * 23 + [256], 2048, False), (MLSTM, [1] * 7 + [512], 2048, True), (RETENTION, [1] * 23 + [256], 4096, False),
    (RETENTION, [1] * 256, 2048, False), (WKV, [1] * 64, 4096, False), (MLSTM, [1], 512, False),                          # decoded tokens
])
def test_scans_in_chunks_by_cost(mode, lens, width, chunks):
    assert in_chunks(mode, lens, width) is chunks


def test_scans_in_chunks_without_the_longest_request():
    """A caller that does not say what the longest request brings: the step's tokens less one for every other request."""
    assert in_chunks(WKV, [512], 2048, known=False) and in_chunks(WKV, [1] * 7 + [512], 2048, known=False)
    assert in_chunks(WKV, [120] * 8, 1024, known=False) and not in_chunks(WKV, [120] * 8, 1024)


@pytest.mark.parametrize("mode", [RETENTION, MLSTM, WKV])
def test_scans_in_chunks_only_for_rows_and_heads_that_fit(mode):
    assert in_chunks(mode, [1024], 2048)
    assert not in_chunks(mode, [1024], 2048, dim=136) and not in_chunks(mode, [1024], 2048, dim=20) and not in_chunks(mode, [1024], 2048, dim=4)
    assert not in_chunks(mode, [1024], 2048, stride=2) and not in_chunks(mode, [1024], 2048, at=2)


def selective(lens, channels, states, known=True, dtype=torch.bfloat16):
    """(a thread per channel?, parts) of a selective scan on 148 SMs."""
    ops = CudaOps.__new__(CudaOps)
    ops.num_sms = 148
    step = (sum(lens), len(lens), channels, states)
    wide = ops.selective_wide(dtype, *step, max(lens) if known else None)
    return wide, ops.selective_parts(*step, wide, max(lens) if known else None)


# (as measured: the form ahead, with the parts that were)
@pytest.mark.parametrize("lens,channels,states,form", [
    ([2048], 4096, 16, (True, 32)), ([1024], 4096, 16, (True, 16)), ([512], 8192, 16, (True, 8)), ([512] * 4, 4096, 16, (True, 8)),
    ([512], 4096, 16, (False, 8)), ([100], 8192, 16, (False, 1)),
    ([1] * 23 + [2000], 8192, 16, (True, 5)), ([1] * 7 + [1000], 8192, 16, (True, 15)), ([1] * 23 + [2000], 4096, 8, (True, 18)),
    ([1] * 200 + [2000], 8192, 16, (False, 1)),                       # the parts' sums of so many requests would not fit
    ([128] * 16, 4096, 16, (True, 1)), ([256] * 8, 4096, 16, (True, 1)), ([128] * 16, 8192, 8, (True, 1)),
    ([8] * 150, 8192, 4, (False, 1)), ([64] * 32, 4096, 4, (True, 1)), ([2048], 4096, 32, (False, 8)),
])
def test_selective_scan_forms(lens, channels, states, form):
    assert selective(lens, channels, states) == form
    assert not selective(lens, channels, states, dtype=torch.float32)[0]


# (what a step brings, channels) and the parts of the wide form: as measured, us of the choice | of other counts
@pytest.mark.parametrize("lens,channels,parts", [
    ([2048], 4096, 19), ([2048], 2048, 26), ([4096], 2048, 27), ([1024], 4096, 13), ([512], 8192, 7),                      # one long request: even waves
    ([512] * 4, 4096, 8), ([512] * 2, 8192, 8), ([512] * 8, 2048, 8), ([512] * 16, 1024, 8), ([1024] * 4, 4096, 8),        # 97 | 114 in one part, 179 | 225
    ([500] * 3, 5120, 7), ([512] * 2, 4096, 8), ([700, 300], 8192, 10), ([512, 1, 1, 512, 512, 1, 512], 4096, 8),          # 87 | 112, 59 | 68 in seven, 95 | 106 in six
    ([512] * 3, 4096, 6), ([2048] * 3, 2048, 12), ([2048] * 2, 2048, 19), ([400] * 6, 4096, 1), ([128] * 16, 4096, 1), ([256] * 8, 4096, 1), ([200] * 12, 4096, 1),      # 75 | 81, 145 | 164, 99 | 110, 101 | 110; 60 | 80 in two
])
def test_parts_of_a_selective_scan_with_a_thread_per_channel(lens, channels, parts):
    wide, most = selective(lens, channels, 16)
    T, longest = sum(lens), max(lens)
    assert wide and _even_parts(-(-channels // 128) * T / longest, longest, most, 148, T > 1.2 * longest) == parts


def test_selective_scan_form_without_the_longest_request():
    assert selective([2048], 4096, 16, known=False) == (True, 32) and selective([1] * 7 + [2000], 8192, 16, known=False) == (True, 2)


def test_float32_products_on_tensor_cores_by_shape_and_alignment():
    """The rule that sends a float32 product to the three-plane kernel: sizes, strides and addresses that its copies can take."""
    ok = CudaOps._f32_planes_ok
    w = torch.zeros(1024, 2048)
    x = torch.zeros(64, 2048)
    assert ok(x, w) and ok(x[:33], w) and ok(x[:17], w) and not ok(x[:16], w)
    assert not ok(x[:, 1:], w[:, 1:]) and not ok(x[:, :2046], w[:, :2046])              # rows off 16 bytes; K % 4
    assert ok(x[:, 4:], w[:, 4:]) and not ok(torch.zeros(64, 2049)[:, :2048], w)        # a stride that is not a multiple of 4
    assert not ok(x, w[:511]) and not ok(x[:, :512], w[:, :512]) and ok(torch.zeros(33, 128), torch.zeros(12288, 128))
    assert not ok(x[:32, :1020], torch.zeros(4096, 1020)) and ok(x[:32, :1024], w[:, :1024])


@pytest.mark.parametrize("mode,lens,key,value,dtype,tokens", [
    (RETENTION, [2048], 128, 128, torch.bfloat16, 128), (MLSTM, [128], 64, 128, torch.bfloat16, 128), (RETENTION, [100] * 4, 128, 128, torch.bfloat16, 128),
    (RETENTION, [2048], 64, 64, torch.bfloat16, 64), (RETENTION, [2048], 128, 136, torch.bfloat16, 64), (RETENTION, [2048], 128, 128, torch.float32, 64),
    (WKV, [2048], 128, 128, torch.bfloat16, 64), (RETENTION, [1] * 23 + [256], 128, 128, torch.bfloat16, 64), (MLSTM, [1] * 31 + [2000], 64, 128, torch.bfloat16, 128)])
def test_tokens_of_a_chunk(mode, lens, key, value, dtype, tokens):
    assert CudaOps._chunk_tokens(mode, dtype, sum(lens), len(lens), key, value) == tokens


@pytest.mark.parametrize("heads,rows,group,dim,new,keys", [(1, 64, 16, 128, 4, 4), (1, 4800, 16, 128, 300, 300), (8, 300, 1, 64, 300, 300), (1, 2048, 16, 128, 128, 4096),
                                                           (4, 80, 16, 128, 5, 1000), (16, 64, 16, 128, 4, 4096), (1, 32768, 16, 128, 2048, 2048),
                                                           (6, 64, 1, 36, 64, 100000)])
def test_float32_pieces_cover_the_keys(heads, rows, group, dim, new, keys):
    """Pieces of whole tiles that cover every key, the last one not empty; many row tiles are left uncut."""
    ops = CudaOps.__new__(CudaOps)
    ops.num_sms = 148
    kernel, n, length = ops._f32_tile_pieces(heads, rows, group, dim, new, keys)
    assert kernel == "simt" and n >= 1
    if n > 1:
        assert length % 64 == 0 and (n - 1) * length < keys <= n * length
    if keys <= 64 or rows >= 32768:
        assert n == 1
    if keys >= 32 * new:                                                             # few rows behind many keys
        assert n >= 8


@pytest.mark.parametrize("N,K", [(4352, 4096), (4096, 4096), (4096, 11008), (32000, 4096), (1024, 4096), (256000, 2048), (5120, 1024), (2304, 64 * 31), (8192, 28672)])
def test_form_of_a_decode_product_comes_from_its_sizes(N, K):
    """K ranges and row sets of the weight-streaming product: ranges that cover K, the last one not empty, 512 or more; whole where the caller
    wants whole sums; the same answer every time."""
    for few in (True, False):
        kslice, code = _ring_form(N, K, 148, True, few)
        S = -(-K // kslice)
        assert kslice % 128 == 0 and code in (0, 16) and (S == 1 or K >= 512 * S) and S <= 8 and (S - 1) * kslice < K
        whole, code = _ring_form(N, K, 148, False, few)
        assert whole == -(-K // 128) * 128 and code in (0, 16)
        _ring_form.cache_clear()
        assert _ring_form(N, K, 148, True, few)[0] == kslice
    if N <= 4352 and K >= 4096:
        assert S >= 2


@pytest.mark.parametrize("mode,lens,heads,tokens", [
    (RETENTION, [2048], 16, 128), (MLSTM, [2048] * 4, 64, 128), (RETENTION, [128] * 16, 16, 128),            # full chunks, however many
    (RETENTION, [1] * 31 + [2000], 16, 64), (MLSTM, [1] * 15 + [512], 32, 64), (MLSTM, [64] * 32, 16, 64),   # short chunks, more of them and heads than run at once
    (RETENTION, [1] * 7 + [512], 16, 128), (MLSTM, [1] * 15 + [512], 8, 128), (RETENTION, [64] * 8, 16, 128)])   # ... and fewer
def test_tokens_of_a_chunk_by_what_runs_at_once(mode, lens, heads, tokens):
    assert CudaOps._chunk_tokens(mode, torch.bfloat16, sum(lens), len(lens), 128, 128, heads, 148) == tokens


def _pieces_tile_by_tile(num_sms, heads, rows, group, head_dim, max_q_len, max_kv_len):
    """The cost model of the float32 pieces, every candidate and every tile."""
    step, tiles, ctx = 3.4 + 0.061 * (64 if head_dim <= 64 else 128), -(-rows // 64), max(0, max_kv_len - max_q_len)
    ends = [ctx + -(-min(rows, (t + 1) * 64) // group) for t in range(tiles)]
    work = sum(-(-e // 64) for e in ends) * heads / num_sms * 0.92 * step
    best, best_cost, last = ("simt", 1, 0), None, 0
    for want in range(1, min(64, -(-max_kv_len // 64)) + 1):
        length = -(-(-(-max_kv_len // want)) // 64) * 64
        n = -(-max_kv_len // length)
        if n == last:
            continue
        last = n
        ctas, alone = heads * sum(-(-e // length) for e in ends), length / 64 * step
        cost = alone if ctas <= num_sms else max(1.84 * alone, work) if ctas <= 2.2 * num_sms or n == 1 else work + 0.5 * alone
        if n > 1:
            cost += 3.0 + heads * rows * (n * (4 * head_dim + 8) + 4 * head_dim) / 2e6
        if best_cost is None or cost < 0.97 * best_cost:
            best, best_cost = (("simt", n, length) if n > 1 else ("simt", 1, 0)), cost
    return best


def test_float32_pieces_in_closed_form():
    """The plan is the one of the model tile by tile, for all kinds of portions, and is not paid for tile by tile."""
    rng = random.Random(5)
    ops = CudaOps.__new__(CudaOps)
    for _ in range(600):
        group, kv_heads, seqs = rng.choice([1, 2, 3, 7, 8, 16, 32, 71]), rng.choice([1, 1, 2, 4, 8]), rng.choice([1, 1, 2, 5, 16])
        new = int(2 ** rng.uniform(0, 11))
        keys = new + rng.choice([0, 0, int(2 ** rng.uniform(0, 13))])
        if new * group < 64:
            continue
        case = (seqs * kv_heads, new * group, group, rng.choice([36, 64, 128]), new, keys)
        assert ops._f32_tile_pieces(*case) == _pieces_tile_by_tile(148, *case), case


def test_float32_pieces_stop_where_no_candidate_can_be_better(monkeypatch):
    from tiny_transformer_inference_engine_b200 import ops as module
    calls = []
    monkeypatch.setattr(module, "_floor_sum", lambda *a: calls.append(a) or _floor_sum(*a))
    ops = CudaOps.__new__(CudaOps)
    for heads, group, new in ((1, 71, 2048), (1, 32, 2048), (8, 4, 2048), (32, 1, 2048)):
        calls.clear()
        assert ops._f32_tile_pieces(heads, new * group, group, 128, new, new) == ("simt", 1, 0)
        assert len(calls) == 2


@pytest.mark.parametrize("n,m,a,b", [(0, 5, 3, 2), (1, 1, 0, 0), (7, 3, 5, 4), (500, 64 * 71, 64, 4543), (33, 10, 10, 0), (12, 7, 0, 20), (1000, 997, 996, 5)])
def test_floor_sum(n, m, a, b):
    assert _floor_sum(n, m, a, b) == sum((a * i + b) // m for i in range(n))


@pytest.mark.parametrize("M,N,K,planes", [
    (320, 1024, 1024, True), (200, 1024, 1024, True), (33, 512, 2048, True), (1200, 1024, 256, True), (600, 4096, 128, True), (33, 1536, 1024, True),
    (48, 1024, 1024, False), (320, 512, 512, False), (96, 2048, 256, False), (200, 2048, 128, False), (64, 1024, 1024, False), (1200, 256, 1024, False)])
def test_float32_products_on_tensor_cores_by_their_work(M, N, K, planes):
    """Both sides of each line of the rule: the weights, the three sizes' product, a long K."""
    assert CudaOps._f32_planes_ok(torch.zeros(M, K), torch.zeros(N, K)) is planes
