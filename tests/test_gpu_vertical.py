"""GPU parity tests: vertical-line scores, exact top-k, cache reorganisation."""

import numpy as np
import pytest
import torch

import hyquant_b200 as hq
from hyquant_b200 import _lib
from hyquant_b200.synth import gen_numpy
from oracle import hq_oracle as orc
from tests.helpers import load, max_abs, sha
from tests.test_topk_form import form          # noqa: F401

pytestmark = pytest.mark.gpu
DEV = "cuda"


def t_bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DEV).to(torch.bfloat16)


@pytest.mark.parametrize("B,H_Q,H_KV,N,W,nq", [(2, 8, 2, 640, 64, 640), (1, 32, 8, 1024, 128, 1024), (1, 4, 4, 200, 64, 7),
                                                (1, 16, 1, 333, 32, 100), (1, 8, 8, 129, 128, 1)])
def test_vertical_scores_and_topk(B, H_Q, H_KV, N, W, nq):
    case = gen_numpy(B, H_Q, H_KV, N, 128, W, 0.05, 21, n_qry=nq)
    q, k = orc.bf16_round(case.q), orc.bf16_round(case.k)
    R = H_Q // H_KV
    s_gpu = hq.vertical_scores(t_bf16(q), t_bf16(k), W, R)
    s_ref = orc.vertical_scores(q, k, W, R)
    assert s_gpu.shape == s_ref.shape
    sg = s_gpu.cpu().numpy()
    assert max_abs(sg, s_ref) <= 1e-3 * max(1.0, np.abs(s_ref).max())
    # top-k: bit-exact given identical fp32 scores (descending, ties to the lower index)
    kk = orc.vertical_topk_count(sg.shape[-1], 0.05)
    idx, asc = hq.topk_indices(s_gpu, kk, want_ascending=True)
    assert idx.dtype == torch.int64 and asc.dtype == torch.int32
    assert np.array_equal(idx.cpu().numpy(), orc.topk_desc(sg, kk))
    assert np.array_equal(asc.cpu().numpy(), np.sort(orc.topk_desc(sg, kk), axis=-1))
    # the public entry point
    out = hq.compute_vertical_indices(t_bf16(q), t_bf16(k), W, 0.05, kv_repeat=R)
    assert np.array_equal(out.cpu().numpy(), orc.topk_desc(sg, kk))
    # K already expanded to H_Q heads gives the same scores
    if R > 1:
        s_exp = hq.vertical_scores(t_bf16(q), t_bf16(np.repeat(k, R, axis=1)), W, 1)
        assert max_abs(s_exp.cpu().numpy(), sg) <= 1e-4 * max(1.0, np.abs(sg).max())


@pytest.mark.parametrize("B,H_KV,R,N,W,nq", [(1, 8, 4, 1024, 128, 128), (2, 2, 16, 600, 64, 64), (1, 4, 7, 300, 32, 5)])
def test_vertical_scores_with_group_mean_inside(B, H_KV, R, N, W, nq):
    """The freeze-side selection: the mean over a kv-head's query heads taken inside the scoring call equals the
    eager mean in the input dtype followed by the plain call."""
    case = gen_numpy(B, H_KV * R, H_KV, N, 128, W, 0.05, 33, n_qry=nq)
    q, k = t_bf16(case.q), t_bf16(case.k)
    fused = hq.vertical_scores(q, k, W, 1, group_mean=R)
    eager = hq.vertical_scores(q.reshape(B, H_KV, R, nq, 128).mean(dim=2), k, W, 1)
    assert fused.shape == eager.shape == (B, H_KV, N - W)
    # the same numbers up to a rare last-bit difference of a 16-bit mean (fp32 summation order over the heads)
    assert max_abs(fused.cpu().numpy(), eager.cpu().numpy()) <= 2e-3 * float(eager.abs().max())
    kk = orc.vertical_topk_count(N - W, 0.05)
    a, b = hq.topk_indices(fused, kk), hq.topk_indices(eager, kk)
    same = np.mean([len(set(x.tolist()) & set(y.tolist())) / kk for x, y in zip(a.reshape(-1, kk).cpu().numpy(), b.reshape(-1, kk).cpu().numpy())])
    assert same >= 0.95


def test_vertical_reference_rounding_mode_and_empty_prefix():
    case = gen_numpy(1, 8, 2, 512, 128, 64, 0.05, 5)
    q, k = orc.bf16_round(case.q), orc.bf16_round(case.k)
    s = hq.vertical_scores(t_bf16(q), t_bf16(k), 64, 4, round_like_reference=True).cpu().numpy()
    assert np.array_equal(orc.bf16_round(s), s)            # scores are bf16-exact in this mode
    pooled = orc.bf16_round(q[:, :, -64:].mean(axis=2))
    ref = np.einsum("bhrd,bhpd->bhrp", pooled.reshape(1, 2, 4, 128), k[:, :, :448]).reshape(1, 8, 448)
    assert max_abs(s, ref) <= 2e-2 * max(1.0, np.abs(ref).max())
    out = hq.compute_vertical_indices(t_bf16(q[:, :, :5]), t_bf16(k[:, :, :60]), 64, 0.05, kv_repeat=4)
    assert out.shape == (1, 8, 0) and out.dtype == torch.int64


@pytest.mark.parametrize("n,k", [(1, 1), (7, 7), (100, 1), (1000, 50), (4097, 205), (131072 - 256, 6541), (20000, 16384)])
def test_topk_exact_with_ties(n, k):
    rng = np.random.Generator(np.random.PCG64(n + k))
    rows = 3
    s = rng.standard_normal((rows, n), dtype=np.float32)
    s[1] = np.round(s[1] * 4) / 4            # heavy ties
    s[2, : n // 2] = 1.5                      # a plateau that straddles the threshold
    s[0, 0] = -0.0
    idx, asc = hq.topk_indices(torch.from_numpy(s).to(DEV), k, want_ascending=True)
    ref = orc.topk_desc(s, k)
    assert np.array_equal(idx.cpu().numpy(), ref)
    assert np.array_equal(asc.cpu().numpy(), np.sort(ref, axis=-1))


@pytest.mark.parametrize("n,k", [(31, 5), (64, 64), (65, 64), (1025, 129), (53000, 2650), (56000, 100), (56300, 100), (60000, 16384)])
def test_topk_edges_of_the_kept_row_and_the_warp_ranges(n, k):
    """Ranges of warps that are empty, lists around the 64 entries a warp sorts by itself (a block a row up to 12K candidates,
    then a cluster); infinities and a row of one value."""
    rng = np.random.Generator(np.random.PCG64(7 * n + k))
    s = rng.standard_normal((4, n), dtype=np.float32)
    s[1] = 0.25
    s[2, rng.integers(0, n, size=max(1, n // 3))] = -np.inf
    s[3, rng.integers(0, n, size=3)] = np.inf
    idx, asc = hq.topk_indices(torch.from_numpy(s).to(DEV), k, want_ascending=True)
    ref = orc.topk_desc(s, k)
    assert np.array_equal(idx.cpu().numpy(), ref)
    assert np.array_equal(asc.cpu().numpy(), np.sort(ref, axis=-1))


@pytest.mark.parametrize("tail,R,offset", [(1, 1, 0), (127, 4, 0), (128, 7, 0), (129, 4, 8), (300, 2, 4), (256, 1, 4)])
def test_pooled_query_is_the_sum_in_token_order(tail, R, offset):
    """The pooled query decides ties of the selection: the fp32 sum over the tokens in their order, bit for bit, from
    aligned and from unaligned rows.  A key row that is a unit vector reads one channel back."""
    g = torch.Generator(device=DEV); g.manual_seed(tail + R)
    q = torch.randn(1, 2 * R, tail, 128 + offset, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)[..., offset:]
    k = torch.eye(128, device=DEV, dtype=torch.bfloat16).expand(1, 2, 128, 128).contiguous()
    keys = torch.cat([k, torch.zeros(1, 2, tail, 128, device=DEV, dtype=torch.bfloat16)], dim=2)
    got = hq.vertical_scores(q, keys, tail, 1, group_mean=R)
    # the pooled query itself, from the buffer that the scoring call fills
    lib, st = hq._lib.lib(), torch.cuda.current_stream().cuda_stream
    pooled, scores = torch.empty(1, 2, 128, device=DEV), torch.empty(1, 2, 128, device=DEV)
    rows = (q.data_ptr(), hq._lib.HQ_BF16, *q.stride()[:3], 1)
    keys_of = (keys.data_ptr(), *keys.stride()[:3])
    if R > 1:
        rc = lib.hq_vertical_scores_grouped(*rows, 2, R, tail, tail, *keys_of, 128, 0, 0, pooled.data_ptr(), scores.data_ptr(), st)
    else:
        rc = lib.hq_vertical_scores(*rows, 2, tail, tail, *keys_of, 2, 128, 0, 0, pooled.data_ptr(), scores.data_ptr(), st)
    assert rc == 0 and torch.equal(scores, got)
    m = q.float().reshape(1, 2, R, tail, 128).cpu().numpy()
    s = np.zeros((1, 2, tail, 128), np.float32)
    for r in range(R):
        s += m[:, :, r]
    if R > 1:
        s = orc.bf16_round(s / np.float32(R))
    acc = np.zeros((1, 2, 128), np.float32)
    for i in range(tail):
        acc += s[:, :, i]
    want = acc / np.float32(tail)
    assert np.array_equal(pooled.cpu().numpy(), want)
    # the scores split the mean into two bf16 parts: 2^-16 of the value at most
    assert np.all(np.abs(got.cpu().numpy() - want) <= 2.0 ** -16 * np.abs(want))


def test_topk_limits():
    s = torch.zeros(1, 40000, device=DEV)
    with pytest.raises(hq.HyQuantError):
        hq.topk_indices(s, 16385)
    with pytest.raises(hq.HyQuantError):
        hq.topk_indices(s[:, :10], 11)


def test_vertical_indices_fixture_sets():
    """The reference's fp32 selection (golden) against the device selection on bf16-rounded
    inputs: sets agree except for near-ties moved by the bf16 rounding of the inputs."""
    g = load("vertical_indices")
    B, H_Q, H_KV, N, W, seed = [int(x) for x in g["meta"]]
    case = gen_numpy(B, H_Q, H_KV, N, 128, W, 0.05, seed)
    out = hq.compute_vertical_indices(t_bf16(case.q), t_bf16(case.k), W, 0.05, kv_repeat=H_Q // H_KV).cpu().numpy()
    ref = g["idx_gqa"]
    assert out.shape == ref.shape
    for a, b in zip(out.reshape(-1, out.shape[-1]), ref.reshape(-1, ref.shape[-1])):
        assert len(set(a.tolist()) & set(b.tolist())) >= 0.9 * len(a)


@pytest.mark.parametrize("BH,N,W,T", [(2, 1024, 128, 45), (3, 300, 64, 0), (1, 130, 128, 1), (2, 64, 64, 0), (8, 4096, 128, 199)])
def test_cache_reorganize_bit_exact(BH, N, W, T):
    rng = np.random.Generator(np.random.PCG64(N + T))
    k = orc.bf16_round(rng.standard_normal((1, BH, N, 128), dtype=np.float32) * 1.7)
    v = orc.bf16_round(rng.standard_normal((1, BH, N, 128), dtype=np.float32))
    P = N - W
    vidx = np.stack([rng.permutation(P)[:T] for _ in range(BH)]).reshape(1, BH, T).astype(np.int64) if T else None
    layer = hq.DStageLayerCache(0, window_size=W, top_ratio=0.05, use_vert=False)
    layer.update_prefill(t_bf16(k), t_bf16(v))
    layer.freeze(kv_repeat=1, vertical_indices=None if vidx is None else torch.from_numpy(vidx))
    qt = np.zeros((1, BH, 1, 128), np.float32)
    oc = orc.freeze(k, v, qt if T else None, 1, W, 0.05, vidx_override=vidx, use_vert=T > 0)
    assert np.array_equal(layer.k_quant_packed.cpu().numpy(), oc.k_quant_packed)
    assert np.array_equal(layer.v_quant_packed.cpu().numpy(), oc.v_quant_packed)
    assert np.array_equal(layer.k_scale.cpu().numpy().view(np.uint16), oc.k_scale.view(np.uint16))
    assert np.array_equal(layer.v_scale.cpu().numpy().view(np.uint16), oc.v_scale.view(np.uint16))
    assert np.array_equal(layer.k_topk.float().cpu().numpy(), oc.k_topk)
    assert np.array_equal(layer.v_topk.float().cpu().numpy(), oc.v_topk)
    assert np.array_equal(layer.k_window.float().cpu().numpy(), oc.k_window)
    assert np.array_equal(layer.v_window.float().cpu().numpy(), oc.v_window)
    assert layer._staging_buf_k.shape == (BH, 128, 128) and float(layer._staging_buf_k.abs().sum()) == 0.0


@pytest.mark.parametrize("rows,n,k,kind", [(3, 12288, 614, "normal"), (2, 12289, 1, "normal"), (1, 16384, 16384, "ties"), (5, 20011, 1000, "ties"),
                                           (2, 32512, 1625, "one slice"), (70, 12301, 77, "normal"), (1, 131071, 6553, "normal"),
                                           (2, 40000, 9000, "infinities"), (1, 400001, 300, "normal")])
def test_topk_of_long_rows(rows, n, k, kind):
    """Long rows, few enough to be shared by clusters of blocks (but for 70 rows): odd slices, ties across slices, everything in
    one slice, lists too long to be brought together; the same list as the oracle's, bit for bit."""
    rng = np.random.default_rng(n + k)
    s = rng.standard_normal((rows, n)).astype(np.float32)
    if kind == "ties":
        s = np.round(2 * s).astype(np.float32)
    elif kind == "one slice":
        s[:, 9000:9000 + k] += 100.0
    elif kind == "infinities":
        s[:, ::7] = -np.inf
        s[:, 5::1000] = np.inf
    idx, asc = hq.topk_indices(torch.from_numpy(s).to(DEV)[None], k, want_ascending=True)
    want = orc.topk_desc(s[None], k)
    assert np.array_equal(idx.cpu().numpy(), want)
    assert np.array_equal(asc.cpu().numpy(), np.sort(want, axis=-1))


@pytest.mark.parametrize("rows,n,k,blocks,kept", [
    (1, 440001, 300, 8, False),          # slices read again, lists brought together in the counters' place
    (1, 200000, 10000, 8, False),        # slices read again, entries searched in the other blocks' lists
    (20, 170000, 8500, 4, False), (20, 50000, 6300, 4, True), (37, 25000, 1250, 8, True), (64, 16400, 820, 4, True),
    ("sms", 12500, 625, 1, True), ("sms", 46900, 2345, 1, True), ("sms", 57000, 2850, 1, False), (40, 60000, 16384, 1, False),
    (75, 30000, 1500, 1, True)])
def test_topk_in_every_form(form, rows, n, k, blocks, kept):      # noqa: F811
    """Each kernel that the rule can pick, with ties across slices in every other row; "sms": a row more than the chip has SMs."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = sms + 1 if rows == "sms" else rows
    assert form(rows, n, k, sms)[0] == blocks and bool(form(rows, n, k, sms)[3]) == kept
    rng = np.random.default_rng(rows + n)
    s = rng.standard_normal((rows, n), dtype=np.float32)
    s[1::2] = np.round(2 * s[1::2])
    s[0, 100:] = np.where(s[0, 100:] > 0.5, np.float32(0.5), s[0, 100:])      # a plateau at the threshold
    idx, asc = hq.topk_indices(torch.from_numpy(s).to(DEV), k, want_ascending=True)
    want = orc.topk_desc(s, k)
    assert np.array_equal(idx.cpu().numpy(), want)
    assert np.array_equal(asc.cpu().numpy(), np.sort(want, axis=-1))


@pytest.mark.parametrize("N,W,T,dense", [(700, 64, 32, False), (700, 64, 33, False), (5000, 128, 1025, False), (1000, 100, 200, True),
                                         (129, 1, 127, True), (260, 4, 0, False)])
def test_reorganisation_places_every_row(N, W, T, dense):
    """The list search (32 probes a round) and the rank bits at the edges of tiles: vertical rows anywhere, or filling
    whole tiles; the rest in order, as the quantiser packs it."""
    g = torch.Generator(device="cpu").manual_seed(N + T)
    kv = torch.randn(2, 1, 2, N, 128, generator=g).to(torch.bfloat16).to(DEV)
    P = N - W
    picks = [torch.arange(3, 3 + T) % P if dense else torch.randperm(P, generator=g)[:T] for _ in range(2)]
    idx = torch.stack(picks)[None].to(DEV)
    layer = hq.DStageLayerCache(0, k_bits=4, v_bits=8, window_size=W, use_vert=False)
    layer.update_prefill(kv[0], kv[1])
    layer.freeze(1, vertical_indices=idx)
    for h in range(2):
        rest = torch.ones(P, dtype=torch.bool)
        rest[picks[h]] = False
        for x, bits, packed, scale, topk in ((kv[0], 4, layer.k_quant_packed, layer.k_scale, layer.k_topk), (kv[1], 8, layer.v_quant_packed, layer.v_scale, layer.v_topk)):
            row = x[0, h]
            codes, sc = hq.quantize_per_token(row[:P][rest.to(DEV)][None], bits)
            assert torch.equal(topk[h], row[picks[h].to(DEV)])
            assert packed.shape[1] == P - T
            assert torch.equal(packed[h].view(torch.int8), codes[0]) and torch.equal(scale[h].reshape(-1), sc[0])


@pytest.mark.parametrize("N,positions", [(700, [5] * 3 + [40, 41, 41, 127, 127, 128, 128, 128, 300]), (700, [130] * 200 + list(range(140, 200))), (300, [0, 0, 255, 255])])
def test_reorganisation_with_positions_given_more_than_once(N, positions):
    """A list that repeats positions (within a tile, across a tile's edge, more entries than a tile has rows): every entry counts
    for the rows behind it, so that row p stands at p minus the entries below it; where two rows meet, either may stand."""
    g = torch.Generator(device="cpu").manual_seed(N)
    W, T = 44, len(positions)
    kv = torch.randn(2, 1, 1, N, 128, generator=g).to(torch.bfloat16).to(DEV)
    layer = hq.DStageLayerCache(0, k_bits=4, v_bits=2, window_size=W, use_vert=False)
    layer.update_prefill(kv[0], kv[1])
    layer.freeze(1, vertical_indices=torch.tensor(positions)[None, None].to(DEV))
    sources = {}
    for p in range(N - W):
        at = p - sum(x < p for x in positions)
        if p not in positions and 0 <= at < N - W - T:
            sources.setdefault(at, []).append(p)
    alone = {at: ps[0] for at, ps in sources.items() if len(ps) == 1}
    assert len(alone) >= (N - W - T) // 4
    at, ps = torch.tensor(list(alone)).to(DEV), torch.tensor(list(alone.values())).to(DEV)
    for x, bits, packed, scale, topk in ((kv[0], 4, layer.k_quant_packed, layer.k_scale, layer.k_topk), (kv[1], 2, layer.v_quant_packed, layer.v_scale, layer.v_topk)):
        codes, sc = hq.quantize_per_token(x[0, :, ps], bits)
        assert torch.equal(packed[0, at].view(torch.int8), codes[0]) and torch.equal(scale[0, at], sc[0])
        assert torch.equal(topk[0], x[0, 0, torch.tensor(positions).to(DEV)])


@pytest.mark.parametrize("bits", [2, 4, 8])
def test_quantiser_words_that_leave_the_common_path(bits):
    """Rows of subnormal scale (where a quotient can round past q_max), rows full of half-integers, and a NaN or an infinity in
    one word of a row: the codes of the oracle; a NaN is the lowest code and does not count for the scale.  An infinite scale
    (an infinity in the row, or a maximum past fp16) makes every finite value 0 and infinities the lowest code."""
    rng = np.random.default_rng(bits)
    qmax = 2 ** (bits - 1) - 1
    x = rng.standard_normal((1, 200, 128)).astype(np.float32)
    x[0, :60] *= np.geomspace(1e-9, 1e-2, 60)[:, None].astype(np.float32)
    x[0, 60:140] = (rng.integers(-2 * qmax, 2 * qmax + 1, (80, 128)) * 0.5).astype(np.float32)
    x[0, 60:140, 5] = qmax                                    # scale 1: every odd half is a tie
    x = orc.bf16_round(x)
    for mode in (0, 1):
        pk = torch.empty(1, 200, 16 * bits, dtype=torch.int8, device=DEV)
        sc = torch.empty(1, 200, dtype=torch.float16, device=DEV)
        hq.quantize_per_token_into(t_bf16(x), pk, sc, 0, nbits=bits, scale_mode=mode)
        po, so = orc.quantize_per_token(x, bits, reciprocal_scale=mode == 1)
        assert np.array_equal(pk.cpu().numpy(), po) and np.array_equal(sc.cpu().numpy().view(np.uint16), so.view(np.uint16))
    odd = x[:, 150:152].copy()
    clean, _ = hq.quantize_per_token(t_bf16(np.where(np.arange(128) == 40, 0, odd)), bits)
    odd[0, :, 40] = np.nan
    got, _ = hq.quantize_per_token(t_bf16(odd), bits)
    per = 8 // bits
    low = np.uint8(((1 << (bits - 1)) & ((1 << bits) - 1)) << (bits * (40 % per)))
    want = clean.cpu().numpy().view(np.uint8).copy()
    want[0, :, 40 // per] |= low
    assert np.array_equal(got.cpu().numpy().view(np.uint8), want)
    odd[0, 0, 40], odd[0, 1, 40] = np.inf, -np.inf
    got, scale = hq.quantize_per_token(t_bf16(odd), bits)
    want = np.zeros_like(want)
    want[0, :, 40 // per] = low
    assert bool(torch.isinf(scale).all()) and np.array_equal(got.cpu().numpy().view(np.uint8), want)
    big = torch.randn(1, 3, 128, device=DEV) * torch.tensor([1e7, 1e20, 3e37], device=DEV)[None, :, None]
    got, scale = hq.quantize_per_token(big, bits)
    assert bool(torch.isinf(scale).all()) and not bool(got.any())
