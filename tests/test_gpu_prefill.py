"""GPU parity tests of the hybrid prefill path (operand preparation + attention kernel).

Tolerances: INT8 codes and scales bit-exact against the oracle's block quantiser (block = 1 row);
attention outputs max-abs <= 2e-2 and rel-MSE <= 1e-4 against float64 dense causal attention
on the same BF16 inputs."""

import numpy as np
import pytest
import torch

import hyquant_b200 as hq
from hyquant_b200 import sage_unified as su
from hyquant_b200.synth import gen_numpy
from oracle import hq_oracle as orc
from tests.helpers import max_abs

pytestmark = pytest.mark.gpu
DEV = "cuda"
MAX_ABS, REL_MSE = 2e-2, 1e-4


def t_bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DEV).to(torch.bfloat16)


def to_np(t):
    return t.detach().float().cpu().numpy()


def make(B, H_Q, H_KV, N, W, seed, rho=0.05):
    case = gen_numpy(B, H_Q, H_KV, N, 128, W, rho, seed)
    rb = orc.bf16_round
    return rb(case.q), rb(case.k), rb(case.v)


@pytest.mark.parametrize("N", [64, 200, 1000])
@pytest.mark.parametrize("smooth", [True, False])
def test_operand_preparation_bit_exact(N, smooth):
    q, k, v = make(1, 4, 2, N, 64, N)
    sm = 128 ** -0.5
    q_i8, q_bf, q_sc, k_i8, k_bf, k_sc, k_mean = su.quantize_operands(t_bf16(q), t_bf16(k), sm, smooth)
    km = to_np(k_mean)[:, :, None, :]
    if smooth:
        assert max_abs(km, k.mean(axis=2, keepdims=True)) <= 2e-2       # bf16 rounding of the mean
    else:
        assert np.abs(km).max() == 0
    ksm = orc.bf16_round(k - km)
    assert np.array_equal(to_np(k_bf), ksm)
    ki, ks = orc.quant_per_block_int8(ksm, 1, 1.0)           # the block quantiser's arithmetic, one row per block
    assert np.array_equal(k_sc.cpu().numpy()[..., :N], ks) and not k_sc.cpu().numpy()[..., N:].any()
    assert np.array_equal(k_i8.cpu().numpy(), ki)
    qi, qs = orc.quant_per_block_int8(q, 1, sm * orc.LOG2E)
    assert np.allclose(q_sc.cpu().numpy()[..., :N], qs, rtol=1e-6)
    assert (np.abs(q_i8.cpu().numpy().astype(int) - qi.astype(int)) <= 1).all()      # fp32 product order of sm * log2e
    assert (q_i8.cpu().numpy() != qi).mean() < 1e-3
    assert np.array_equal(to_np(q_bf), q)


def test_row_codes_on_and_beside_ties():
    """Rows whose quotients are half-integers or one step beside them, all-zero rows, rows of the smallest values: the
    codes of the division, bit for bit (the kernel corrects the product with the reciprocal by its remainder)."""
    rng = np.random.Generator(np.random.PCG64(3))
    N = 333
    k = (rng.integers(-127, 127, size=(1, 2, N, 128)) + 0.5).astype(np.float32)
    k[:, :, :, 0] = 127.0                                    # scale 2^e: every quotient is a half-integer
    k *= (2.0 ** rng.integers(-12, 12, size=(1, 2, N, 1))).astype(np.float32)
    k[:, :, 100:200] = orc.bf16_round(k[:, :, 100:200] * np.float32(1.0078125))       # beside the ties
    k[:, :, 200:220] *= rng.uniform(0.5, 2.0, size=(1, 2, 20, 1)).astype(np.float32)
    k[:, :, 220] = 0.0
    k[:, :, 221] = 1e-38
    k = orc.bf16_round(k)
    q = orc.bf16_round(rng.standard_normal((1, 4, N, 128), dtype=np.float32))
    _, _, _, k_i8, _, k_sc, _ = su.quantize_operands(t_bf16(q), t_bf16(k), 128 ** -0.5, False)
    ki, ks = orc.quant_per_block_int8(k, 1, 1.0)
    live = np.ones(N, bool); live[220:222] = False           # the oracle divides a zero row by zero
    assert np.array_equal(k_i8.cpu().numpy()[:, :, live], ki[:, :, live])
    assert np.array_equal(k_sc.cpu().numpy()[..., :N][..., live], ks[..., live])
    assert not k_i8.cpu().numpy()[:, :, 220:222].any()


def test_row_codes_of_nan_and_infinite_elements():
    """A NaN does not count for its row's maximum and gets the lowest code; its neighbours are quantised as without it.  In a
    row with an infinity the finite elements are 0 and the infinity (inf / inf) is the lowest code."""
    rng = np.random.Generator(np.random.PCG64(11))
    N = 100
    x = orc.bf16_round(rng.standard_normal((1, 2, N, 128), dtype=np.float32))
    x[0, :, 3, 7] = np.nan
    x[0, :, 40, [0, 31, 32, 127]] = np.nan
    x[0, :, 41] = np.nan
    x[0, :, 63, 5] = np.inf
    x[0, :, 64, 90] = -np.inf
    x[0, :, 65, 1], x[0, :, 65, 2] = np.inf, np.nan
    sm = 1.0 / orc.LOG2E                                     # q is scaled by sm * log2 e = 1, up to the fp32 rounding
    q_i8, _, q_sc, k_i8, _, k_sc, _ = su.quantize_operands(t_bf16(x), t_bf16(x), sm, False)
    with np.errstate(invalid="ignore"):
        amax = np.fmax.reduce(np.abs(x), axis=-1, initial=0.0)
        scale = (np.maximum(amax, np.float32(1e-30)) / np.float32(127.0)).astype(np.float32)
        y = (x / scale[..., None]).astype(np.float32)
        y = np.trunc(y + np.where(y >= 0, np.float32(0.5), np.float32(-0.5)))
    codes = np.where(np.isnan(y), -128, np.clip(np.nan_to_num(y), -128, 127)).astype(np.int8)
    assert np.array_equal(k_i8.cpu().numpy(), codes)
    assert np.array_equal(k_sc.cpu().numpy()[..., :N], scale)
    special = [3, 40, 41, 63, 64, 65]
    low = np.isnan(y[:, :, special])
    assert (q_i8.cpu().numpy()[:, :, special][low] == -128).all()
    assert (np.abs(q_i8.cpu().numpy().astype(int) - codes.astype(int)) <= 1).all()


@pytest.mark.parametrize("T,last", [(1, 0), (64, 63), (65, 4000), (1600, 32639), (500, 100), (16384, (1 << 20) - 1)])
def test_vertical_sort_is_the_clamped_ascending_list(T, last):
    """Positions out of range and positions given twice (or T times) among them."""
    g = torch.Generator(device=DEV); g.manual_seed(T)
    idx = torch.randint(-3, last + 5, (3, T), generator=g, device=DEV)
    if T <= 1600:
        idx[1] = last // 2
    asc = torch.empty(3, T, dtype=torch.int32, device=DEV)
    lib = hq._lib.lib()
    assert lib.hq_prefill_vertical_sort(idx.data_ptr(), 3, T, last, asc.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(asc.long(), idx.clamp(0, last).sort(dim=-1).values)


@pytest.mark.parametrize("T,last", [(16384, 99), (16384, (1 << 20) - 1), (5000, 40000)])
def test_vertical_sort_of_lists_that_repeat_positions_is_linear(T, last):
    """Long lists over few positions, every position twice, one position in half of the places: the sorted list, in not
    much more time than a list without repetitions takes (each form is one launch of a few passes; a walk over the
    repeated entries per position took over a hundred times as long)."""
    g = torch.Generator(device=DEV); g.manual_seed(T)
    lib, asc = hq._lib.lib(), torch.empty(1, T, dtype=torch.int32, device=DEV)

    def run(idx, last):
        assert lib.hq_prefill_vertical_sort(idx.data_ptr(), 1, T, last, asc.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0

    def best_us(idx, last):
        times = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(); run(idx, last); b.record(); b.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return min(times)

    plain = torch.randperm(1 << 20, generator=g, device=DEV)[None, :T].contiguous()
    limit = 12 * best_us(plain, (1 << 20) - 1)
    some = torch.randint(0, last + 1, (1, T), generator=g, device=DEV)
    twice = some.clone(); twice[:, 1::2] = some[:, ::2][:, :T // 2]
    half = some.clone(); half[:, ::2] = last // 3
    for idx in (some % 100, twice, half, torch.full_like(some, last)):
        run(idx, last)
        assert torch.equal(asc.long(), idx.clamp(0, last).sort(dim=-1).values)
        assert best_us(idx, last) <= limit


def test_the_one_shot_calls_leave_their_inputs_alone():
    """The one-shot entry points may read q and k in place where a plan copies them: same result, inputs unchanged."""
    q, k, v = make(2, 4, 2, 333, 128, 3)
    for window, smooth in ((128, True), (333, False), (500, False), (0, True)):
        tq, tk, tv = t_bf16(q), t_bf16(k), t_bf16(v)
        a = su.hybrid_prefill(tq, tk, tv, None, window, None, smooth)
        b = su.PrefillPlan(tq, tk, tv, None, window, None, smooth).run()
        assert torch.equal(a, b)
        assert np.array_equal(to_np(tq), q) and np.array_equal(to_np(tk), k) and np.array_equal(to_np(tv), v)


@pytest.mark.parametrize("form", ["tokens_first", "padded_rows", "every_other_head"])
def test_the_one_shot_calls_on_strided_inputs(form):
    """q, k and v as the models hand them over (transposed projections), as slices of wider rows and of more heads: the
    results of contiguous tensors, bit for bit, on the hybrid, the 16-bit and the FP8 route; inputs unchanged."""
    def strided(x):
        t = t_bf16(x)
        if form == "tokens_first":
            return t.transpose(1, 2).contiguous().transpose(1, 2)
        if form == "padded_rows":
            return torch.cat([t, torch.full_like(t[..., :8], 3.0)], dim=-1)[..., :128]
        return torch.stack([t, torch.full_like(t, 5.0)], dim=2).flatten(1, 2)[:, ::2]

    N, W = 333, 64
    q, k, v = make(2, 4, 2, N, W, 12)
    a, b = [t_bf16(x) for x in (q, k, v)], [strided(x) for x in (q, k, v)]
    assert all(torch.equal(x, y) and not y.is_contiguous() for x, y in zip(a, b))
    idx = uneven_lists(2, 4, N, W, 40)
    for call in (lambda t: su.hybrid_prefill(*t, idx, W, None, True), lambda t: su.hybrid_prefill(*t, None, N, None, False),
                 lambda t: su.full_attention_fp16_triton(*t), lambda t: su.sage_fp8_attention(*t),
                 lambda t: su.sage_unified_attention(*t, window_size=W, smooth_k=False)):
        assert torch.equal(call(a), call(b))
    for x, y in zip((q, k, v), b):
        assert np.array_equal(to_np(y), x)


def check(out, ref):
    assert np.isfinite(out).all()
    assert max_abs(out, ref) <= MAX_ABS, max_abs(out, ref)
    assert orc.rel_mse(out, ref) <= REL_MSE, orc.rel_mse(out, ref)


@pytest.mark.parametrize("B,H_Q,H_KV,N,W", [(1, 4, 2, 128, 64), (1, 4, 1, 200, 64), (2, 8, 2, 512, 128), (1, 4, 4, 1000, 256),
                                            (1, 8, 2, 2048, 128), (1, 2, 1, 1500, 0), (1, 2, 2, 77, 128)])
def test_vertical_attention_vs_dense(B, H_Q, H_KV, N, W):
    q, k, v = make(B, H_Q, H_KV, N, W, N + W)
    R = H_Q // H_KV
    vidx = hq.compute_vertical_indices(t_bf16(q), t_bf16(k), W, 0.05, kv_repeat=R)
    out = hq.sage_vertical_attention_v2(t_bf16(q), t_bf16(k), t_bf16(v), vidx, window_size=W)
    assert out.dtype == torch.bfloat16 and out.shape == (B, H_Q, N, 128)
    ref = orc.dense_causal_attention(q, k, v)
    check(to_np(out), ref)
    # the reference restatement (INT8 rest / fp16 vertical + window) lands in the same place
    if N <= 512:
        rr = orc.hybrid_prefill_reference(q, k, v, vidx.cpu().numpy(), window_size=W, round_fn=orc.bf16_round)
        assert max_abs(to_np(out), rr) <= MAX_ABS


@pytest.mark.parametrize("window,smooth", [(64, True), (200, False), (500, False)])
def test_an_unknown_scale_granularity_is_refused(window, smooth):
    q, k, v = [t_bf16(x) for x in make(1, 2, 1, 200, 64, 4)]
    with pytest.raises(ValueError):
        su.hybrid_prefill(q, k, v, None, window, None, smooth, scale_granularity="tile")


def uneven_lists(B, H_Q, N, W, T):
    """[B, H_Q, T] positions: heads in turn with all lines early, all late, spread, in the middle - every block then serves
    two heads with up to T / 64 tiles more for the one than for the other."""
    prefix = N - W
    forms = [np.arange(T), prefix - T + np.arange(T), np.arange(T) * prefix // T, (prefix - T) // 2 + np.arange(T)]
    return torch.from_numpy(np.stack([np.stack([forms[(h + b) % 4][::-1] for h in range(H_Q)]) for b in range(B)]).copy()).to(DEV)


@pytest.mark.parametrize("H_Q,H_KV,N,W,T", [(4, 1, 2600, 128, 700), (3, 1, 1500, 64, 640), (4, 2, 2300, 0, 330), (2, 1, 3000, 256, 1900)])
@pytest.mark.parametrize("pv_fp8", [False, True])
def test_heads_with_unequal_numbers_of_vertical_tiles(H_Q, H_KV, N, W, T, pv_fp8):
    q, k, v = make(1, H_Q, H_KV, N, W, N + T)
    plan = su.PrefillPlan(t_bf16(q), t_bf16(k), t_bf16(v), uneven_lists(1, H_Q, N, W, T), W, None, True, pv_fp8=pv_fp8)
    out = to_np(plan.run())
    plan.check_status()
    ref = orc.dense_causal_attention(q, k, v)
    if pv_fp8:                                # the price of the format, as in test_gpu_fp8_pv.py
        assert np.isfinite(out).all() and orc.rel_mse(out, ref) <= 5e-3
    else:
        check(out, ref)
    # the other order of each pair of heads (a warp's rows past N are the next head's and may make it move its
    # references earlier: whole warps of the head's own rows are compared)
    flip = torch.arange(H_Q - 1, -1, -1, device=DEV)
    if H_KV == 1 and H_Q % 2 == 0:
        other = su.hybrid_prefill(t_bf16(q)[:, flip], t_bf16(k), t_bf16(v), uneven_lists(1, H_Q, N, W, T)[:, flip], W, None, True, pv_fp8=pv_fp8)
        assert max_abs(to_np(other[:, flip])[:, :, :N // 32 * 32], out[:, :, :N // 32 * 32]) == 0


def test_one_position_given_many_times():
    """A list that repeats one position (as the clamp of positions past the prefix makes it) is longer than the prefix it
    stands in: eleven tiles of one head in front of the first window tile, after one INT8 tile."""
    q, k, v = make(1, 2, 1, 900, 64, 8)
    idx = torch.zeros(1, 2, 700, dtype=torch.int64, device=DEV)
    idx[0, 1] = 10 ** 6
    plan = su.PrefillPlan(t_bf16(q), t_bf16(k), t_bf16(v), idx, 64, None, True)
    out = to_np(plan.run())
    plan.check_status()
    rr = orc.hybrid_prefill_reference(q, k, v, idx.clamp(0, 900 - 64 - 1).cpu().numpy(), window_size=64, round_fn=orc.bf16_round)
    assert np.isfinite(out).all() and max_abs(out, rr) <= MAX_ABS


def test_plan_reuse_and_status_word():
    q, k, v = make(1, 8, 2, 900, 128, 17)
    vidx = hq.compute_vertical_indices(t_bf16(q), t_bf16(k), 128, 0.05, kv_repeat=4)
    plan = su.PrefillPlan(t_bf16(q), t_bf16(k), t_bf16(v), vidx, 128, None, True)
    a = to_np(plan.run()).copy()
    b = to_np(plan.run())
    plan.check_status()                      # no bounded wait expired on the device
    assert np.array_equal(a, b)              # deterministic
    check(a, orc.dense_causal_attention(q, k, v))


@pytest.mark.parametrize("H_Q,H_KV,N,dtype,pv_fp8", [(4, 2, 300, torch.bfloat16, False), (3, 1, 129, torch.float32, True), (2, 2, 64, torch.float16, False)])
def test_blocks_skipped_after_a_failed_wait_give_nan(H_Q, H_KV, N, dtype, pv_fp8):
    """The status word as a block that gave up leaves it: the blocks that find it set skip their work; their rows must not
    look like results.  The word cleared, the same plan computes."""
    q, k, v = [t_bf16(x).to(dtype) for x in make(2, H_Q, H_KV, N, 64, N)]
    plan = su.PrefillPlan(q, k, v, None, 64, None, True, pv_fp8=pv_fp8)
    plan.out.fill_(7.0)
    plan.status.fill_(2)
    assert plan.run().isnan().all()
    with pytest.raises(hq.HyQuantError):
        plan.check_status()
    plan.status.zero_()
    assert plan.run().isfinite().all()
    plan.check_status()


def test_window_only_full_and_int8_only_variants():
    q, k, v = make(1, 8, 2, 700, 128, 5)
    ref = orc.dense_causal_attention(q, k, v)
    tq, tk, tv = t_bf16(q), t_bf16(k), t_bf16(v)
    check(to_np(hq.sage_unified_attention(tq, tk, tv, window_size=128)), ref)
    check(to_np(hq.sage_unified_attention(tq, tk, tv, window_size=0)), ref)
    check(to_np(hq.sage_fp8_attention(tq, tk, tv, pv_fp8=False)), ref)
    # FP8 P V (the entry point's default, checked against its own oracle in test_gpu_fp8_pv.py) is an order of magnitude
    # further from exact attention: that is the format, not the kernel
    fp8 = to_np(hq.sage_fp8_attention(tq, tk, tv))
    assert np.isfinite(fp8).all() and 1e-4 < orc.rel_mse(fp8, ref) < 5e-3
    full = to_np(hq.full_attention_fp16_triton(tq, tk, tv))
    check(full, ref)
    assert orc.rel_mse(full, ref) < 2e-5          # no quantisation at all on this path
    nhd = hq.full_attention_fp16_triton(tq.transpose(1, 2), tk.transpose(1, 2), tv.transpose(1, 2), tensor_layout="NHD")
    assert max_abs(to_np(nhd.transpose(1, 2)), full) == 0
    # fp32 inputs come back as fp32
    o32 = hq.sage_unified_attention(tq.float(), tk.float(), tv.float(), window_size=128)
    assert o32.dtype == torch.float32
    check(to_np(o32), ref)


def test_vertical_lines_are_served_in_bf16():
    """A key with a huge outlier would wreck its INT8 block; as a vertical line it is exact."""
    q, k, v = make(1, 2, 1, 1024, 128, 9)
    k[0, 0, 300] *= 32.0        # a power of two keeps the row bf16-exact
    ref = orc.dense_causal_attention(q, k, v)
    vidx = torch.tensor([[[300, 5], [300, 7]]], device=DEV)
    out = hq.sage_vertical_attention_v2(t_bf16(q), t_bf16(k), t_bf16(v), vidx, window_size=128, smooth_k=False)
    check(to_np(out), ref)


def test_full_size_rows_against_fp32_reference():
    """BASELINE prefill shape (B=1, 32q/8kv, N=8192, W=128, rho=5%): sampled query blocks against an
    fp32 dense computation on the device."""
    t = __import__("hyquant_b200.synth", fromlist=["gen_torch"]).gen_torch(1, 32, 8, 8192, 128, 128, 0.05, 2013, device=DEV)
    q, k, v = t["q"], t["k"], t["v"]
    vidx = hq.compute_vertical_indices(q, k, 128, 0.05, kv_repeat=4)
    out = hq.sage_vertical_attention_v2(q, k, v, vidx, window_size=128).float()
    kf = k.float().repeat_interleave(4, dim=1); vf = v.float().repeat_interleave(4, dim=1)
    for blk in (0, 1, 31, 63):
        rows = slice(blk * 128, blk * 128 + 128)
        s = torch.einsum("bhqd,bhkd->bhqk", q[:, :, rows].float(), kf) * 128 ** -0.5
        pos = torch.arange(8192, device=DEV)
        s = s.masked_fill(pos[None, None, None, :] > pos[rows][None, None, :, None], float("-inf"))
        ref = torch.einsum("bhqk,bhkd->bhqd", torch.softmax(s, -1), vf)
        o = out[:, :, rows]
        assert (o - ref).abs().max().item() <= MAX_ABS
        assert ((o - ref) ** 2).sum().item() / (ref ** 2).sum().item() <= REL_MSE


@pytest.mark.parametrize("B,H_Q,H_KV,N,W,T,layout", [(1, 4, 2, 64, 0, 0, "rows"), (2, 6, 2, 129, 64, 3, "rows"), (2, 4, 2, 1000, 128, 65, "tokens"),
                                                     (1, 3, 1, 777, 777, 0, "tokens"), (2, 2, 2, 1, 1, 0, "rows"), (1, 8, 4, 515, 128, 64, "expanded")])
def test_v_read_where_it_lies_equals_v_transposed(B, H_Q, H_KV, N, W, T, layout):
    """The one-shot route takes V tiles as rows of keys (MN-major operands), a kept plan as V^T: the same products in the same
    order, so the same bits - at ragged ends (keys past N are zero, not the next head's rows, which are NaN here), with V
    strided by token, and with strides that only the transposed route takes."""
    from hyquant_b200.sage_unified import PrefillPlan, hybrid_prefill
    g = torch.Generator(device="cpu").manual_seed(N + T)
    rnd = lambda *s: torch.randn(*s, generator=g).to(torch.bfloat16).cuda()     # noqa: E731
    q, k, v = rnd(B, H_Q, N, 128), rnd(B, H_KV, N, 128), rnd(B, H_KV, N, 128)
    if H_KV > 1 and layout != "expanded":
        v[:, 1] = float("nan")
    if layout == "tokens":
        v = v.transpose(1, 2).contiguous().transpose(1, 2)
    elif layout == "expanded":
        v = v[:, :1].expand(B, H_KV, N, 128)
    idx = torch.stack([torch.randperm(N - W, generator=g)[:T] for _ in range(B * H_Q)]).reshape(B, H_Q, T).cuda() if T else None
    smooth = W < N
    a = hybrid_prefill(q, k, v, idx, W, None, smooth)
    b = PrefillPlan(q, k, v, idx, W, None, smooth).run()
    plan = PrefillPlan(q, k, v, idx, W, None, smooth)
    plan.args.struct_bytes, plan.args.v_rows = type(plan.args).v_sb.offset, 7          # the struct before V's strides: the flag is not read
    assert torch.equal(plan.run().view(torch.int16), b.view(torch.int16))
    head0 = a[:, :H_Q // H_KV]
    assert bool(torch.isfinite(head0.float()).all())
    assert torch.equal(a.view(torch.int16), b.view(torch.int16))
