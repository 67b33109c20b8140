"""The work a program built on hyquant_b200 has it do, as cases that can be timed: decode attention over a frozen
four-segment cache (one layer, a whole token as one CUDA graph, a short answer with its staging flush), the
prefill -> decode transition, and the prefill operators.

Inputs are the seeded synthetic tensors of ``hyquant_b200.synth`` (outlier K channels, vertical-line keys), in bf16.
Head shapes and sizes are those of this repository's benchmark and tests (32q/8kv, 64q/8kv, 32q/2kv, head_dim 128,
window 128 or 256, 5 % vertical lines) and, in the drawn cases, generic ones around them.
"""

from __future__ import annotations

import math

import torch

from hyquant_b200.d_stage_kv_cache import DStageLayerCache
from hyquant_b200.graph_decode import DecodeStepGraph
from hyquant_b200.patch._common import compute_vertical_indices
from hyquant_b200.sage_unified import (
    full_attention_fp16_triton, sage_fp8_attention, sage_unified_attention, sage_vertical_attention_v2,
)
from hyquant_b200.synth import gen_torch

D = 128
RATIO = 0.05


def listed():
    return [
        # one attention call of one layer in a generation loop, the shortest prefix of the benchmark's sweep: latency counts
        dict(name="decode_1k", kind="decode", B=1, hq=32, hkv=8, n=1024, staging=64, window=128, k_bits=4, v_bits=4, vert=True),
        # the benchmark's headline call: 32K prefix, batch 1
        dict(name="decode_32k", kind="decode", B=1, hq=32, hkv=8, n=32768, staging=64, window=128, k_bits=4, v_bits=4, vert=True),
        # batched serving: the whole chip is busy with one call
        dict(name="decode_batch16_32k", kind="decode", B=16, hq=64, hkv=8, n=32768, staging=64, window=128, k_bits=4, v_bits=4, vert=True),
        # long context with sixteen query heads per kv-head
        dict(name="decode_gqa16_128k", kind="decode", B=4, hq=32, hkv=2, n=131072, staging=31, window=128, k_bits=4, v_bits=4, vert=True),
        # another cache mode (8-bit codes, no vertical lines), odd sizes and an odd group of query heads
        dict(name="decode_k8v8_ragged", kind="decode", B=3, hq=28, hkv=4, n=5003, staging=101, window=256, k_bits=8, v_bits=8, vert=False),
        # one generated token of a whole model: every layer's attention as one graph replay, host buffers in and out
        dict(name="token_graph_8k", kind="token", B=1, hq=32, hkv=8, n=8192, layers=32, window=128, k_bits=4, v_bits=4, vert=True),
        # one layer's part of a short answer: freeze after a 2K prompt, then 160 tokens (one staging flush among them)
        dict(name="answer_2k", kind="answer", B=1, hq=32, hkv=8, n=2048, tokens=160, window=256, k_bits=4, v_bits=2, vert=True),
        # the end of a long prompt, one layer: vertical-line selection, reorganisation, quantisation
        dict(name="freeze_32k", kind="freeze", B=1, hq=32, hkv=8, n=32768, window=128, k_bits=4, v_bits=4, vert=True),
        # hybrid prefill with its vertical-line selection, an ordinary and the longest prompt of the benchmark
        dict(name="prefill_8k", kind="hybrid", B=1, hq=32, hkv=8, n=8192, window=128),
        dict(name="prefill_32k", kind="hybrid", B=1, hq=32, hkv=8, n=32768, window=128),
        # 16-bit causal prefill (the plain cache modes' prefill kernel), short ragged prompts in a batch
        dict(name="prefill_full_ragged", kind="full", B=2, hq=32, hkv=8, n=1973),
        # INT8 Q K^T with FP8 P V
        dict(name="prefill_fp8_16k", kind="fp8", B=1, hq=32, hkv=8, n=16384),
    ]


_HEADS = [(32, 8), (32, 8), (64, 8), (32, 2), (28, 4), (16, 8), (24, 8), (12, 2), (8, 8)]
_BITS = [(4, 4), (4, 4), (4, 4), (8, 8), (4, 2), (2, 4)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "decode", "token", "answer", "freeze", "hybrid", "hybrid", "unified", "full", "fp8"])
    hq, hkv = rng.choice(_HEADS)
    kb, vb = rng.choice(_BITS)
    vert, window = rng.random() < 0.75, rng.choice([128, 128, 256])
    if kind == "decode":
        B = rng.choice([1, 1, 2, 3, 4, 8, 16])
        most = min(131072, 4 * 1024 * 1024 // (B * hkv))            # no more cache than sixteen 32K prefixes of eight heads
        return dict(kind=kind, B=B, hq=hq, hkv=hkv, n=_log_int(rng, 700, most), staging=rng.randint(0, 126), window=window,
                    k_bits=kb, v_bits=vb, vert=vert)
    if kind == "token":
        return dict(kind=kind, B=rng.choice([1, 1, 2]), hq=hq, hkv=hkv, n=_log_int(rng, 1000, 16384), layers=rng.choice([8, 16, 28, 32]),
                    window=window, k_bits=kb, v_bits=vb, vert=vert)
    if kind == "answer":
        return dict(kind=kind, B=rng.choice([1, 1, 2]), hq=hq, hkv=hkv, n=_log_int(rng, 700, 8192), tokens=rng.randint(20, 200),
                    window=window, k_bits=kb, v_bits=vb, vert=vert)
    if kind == "freeze":
        B = rng.choice([1, 1, 2, 4])
        return dict(kind=kind, B=B, hq=hq, hkv=hkv, n=_log_int(rng, 700, 65536 // B), window=window, k_bits=kb, v_bits=vb, vert=vert)
    B = rng.choice([1, 1, 2])
    most = int(32768 / math.sqrt(B * hq / 32.0))                     # no more work than the longest listed prompt
    if kind == "fp8":
        most = min(most, 16384)
    n = _log_int(rng, 300, most)
    if kind in ("hybrid", "unified"):
        return dict(kind=kind, B=B, hq=hq, hkv=hkv, n=n, window=window)
    return dict(kind=kind, B=B, hq=hq, hkv=hkv, n=n)


# ---------------------------------------------------------------------------------------------------------------

def _new_layer(case, i=0):
    return DStageLayerCache(i, k_bits=case["k_bits"], v_bits=case["v_bits"], window_size=case["window"], top_ratio=RATIO,
                            use_vert=case["vert"])


def _inputs(case, seed, n_qry=None):
    return gen_torch(case["B"], case["hq"], case["hkv"], case["n"], W=case.get("window", 128), rho=RATIO, seed=seed, n_qry=n_qry)


def _freeze(case, g):
    layer = _new_layer(case)
    layer.update_prefill(g["k"], g["v"])
    layer.save_query_tail(g["q"])
    layer.freeze(kv_repeat=case["hq"] // case["hkv"])
    return layer


def _rows(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32).to(torch.bfloat16)


def prepare(case, seed):
    kind, B, hq, hkv = case["kind"], case["B"], case["hq"], case["hkv"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 7919)
    if kind == "decode":
        # the layer's cache as the prefill left it, with `staging` tokens generated since
        g = _inputs(case, seed, n_qry=case["window"])
        layer = _freeze(case, g)
        if case["staging"]:
            layer.append_staging(_rows(gen, B, hkv, case["staging"], D), _rows(gen, B, hkv, case["staging"], D))
        return dict(kind=kind, layer=layer, q=g["q_decode"], R=hq // hkv)
    if kind == "token":
        layers = [_freeze(case, _inputs(case, 1000 * seed + i, n_qry=case["window"])) for i in range(case["layers"])]
        graph = DecodeStepGraph(layers, B, hq, hkv)
        rows = _rows(gen, case["layers"], B, hq + 2 * hkv, 1, D).cpu()
        for i in range(case["layers"]):                             # what the model's projections hand over, in pinned memory
            graph.host_q[i].copy_(rows[i, :, :hq])
            graph.host_k[i].copy_(rows[i, :, hq:hq + hkv])
            graph.host_v[i].copy_(rows[i, :, hq + hkv:])
        return dict(kind=kind, graph=graph)
    if kind == "answer":
        g = _inputs(case, seed, n_qry=case["window"])
        t = case["tokens"]
        return dict(kind=kind, case=case, g=g, R=hq // hkv, q=_rows(gen, t, B, hq, 1, D), k=_rows(gen, t, B, hkv, 1, D),
                    v=_rows(gen, t, B, hkv, 1, D))
    if kind == "freeze":
        return dict(kind=kind, case=case, g=_inputs(case, seed, n_qry=case["window"]))
    g = _inputs(case, seed)
    return dict(kind=kind, case=case, q=g["q"], k=g["k"], v=g["v"], R=hq // hkv)


def run(state):
    kind = state["kind"]
    if kind == "decode":
        return state["layer"].decode_attention(state["q"], state["R"])
    if kind == "token":
        return state["graph"].step()
    if kind == "answer":
        layer, R, q, k, v = _freeze(state["case"], state["g"]), state["R"], state["q"], state["k"], state["v"]
        out = torch.empty_like(q)
        for i in range(q.shape[0]):
            layer.decode_step(q[i], k[i], v[i], R, out=out[i])
        return out
    if kind == "freeze":
        c = _freeze(state["case"], state["g"])
        return dict(k=c.k_quant_packed, v=c.v_quant_packed, ks=c.k_scale, vs=c.v_scale, kt=c.k_topk, vt=c.v_topk, kw=c.k_window,
                    vw=c.v_window, idx=c.vertical_indices)
    q, k, v = state["q"], state["k"], state["v"]
    if kind == "hybrid":
        W = state["case"]["window"]
        idx = compute_vertical_indices(q, k, W, RATIO, kv_repeat=state["R"])
        return sage_vertical_attention_v2(q, k, v, idx, window_size=W), idx
    if kind == "unified":
        return sage_unified_attention(q, k, v, window_size=state["case"]["window"])
    if kind == "full":
        return full_attention_fp16_triton(q, k, v)
    return sage_fp8_attention(q, k, v)


# ---------------------------------------------------------------------------------------------------------------

def _segments(case):
    """(quantised, vertical-line, window) tokens of a head after freeze."""
    n, W = case["n"], min(case["window"], case["n"])
    cand = max(0, n - 2 * W)
    T = min(max(1, math.ceil(cand * RATIO)), cand) if case["vert"] and cand else 0
    return n - W - T, T, W


def _decode_bytes(case, staging):
    nq, T, W = _segments(case)
    BH, per_tok = case["B"] * case["hkv"], 16 * case["k_bits"] + 16 * case["v_bits"] + 4
    return BH * (per_tok * nq + 512 * (T + W + staging)) + 512 * case["B"] * case["hq"]


def _freeze_bytes(case):
    nq, T, W = _segments(case)
    BH, per_tok = case["B"] * case["hkv"], 16 * case["k_bits"] + 16 * case["v_bits"] + 4
    tail = 256 * case["B"] * case["hq"] * W if T else 0
    return BH * (512 * case["n"] + per_tok * nq + 512 * (T + W) + 8 * T) + tail


def work(case):
    kind, B, hq, hkv, n = case["kind"], case["B"], case["hq"], case["hkv"], case["n"]
    if kind == "decode":
        return dict(bytes=_decode_bytes(case, case["staging"]), flops=4 * D * B * hq * (n + case["staging"]))
    if kind == "token":
        return dict(bytes=case["layers"] * _decode_bytes(case, 64), flops=case["layers"] * 4 * D * B * hq * (n + 64))
    if kind == "answer":
        t = case["tokens"]
        return dict(bytes=_freeze_bytes(case) + t * _decode_bytes(case, min(t, 64)), flops=t * 4 * D * B * hq * (n + t // 2))
    if kind == "freeze":
        return dict(bytes=_freeze_bytes(case), flops=2 * D * B * hkv * n)
    return dict(bytes=2 * D * B * n * (2 * hq + 2 * hkv), flops=4 * D * B * hq * (n * (n + 1) // 2))


def tolerance(case):
    kind = case["kind"]
    if kind == "freeze":
        return "exact"                     # codes, scales, copied rows and indices
    if kind == "fp8":
        return {"rel": 2e-2, "max": 0.5}   # P in e4m3 (2^-4 a value): another split into tiles rounds other values
    # bf16 outputs and bf16 / fp16 probabilities; the vertical-line indices are whole numbers (a tie may swap a few)
    return {"rel": 6e-3, "max": 0.1, "differ": 1e-3}


# ---------------------------------------------------------------------------------------------------------------
# The same calls in 64 bits, in plain torch: what the quantised cache and the attention over it are by definition.

def _quant64(x, bits):
    """[..., n, 128] -> the values that the per-token codes and fp16 scales stand for."""
    qmax = float(2 ** (bits - 1) - 1)
    scale = (x.float().abs().amax(-1, keepdim=True).clamp_min(1e-5) * (1.0 / torch.tensor(qmax)).to(x.device)).half().double()
    return (x.double() / scale).round().clamp(-qmax - 1, qmax) * scale


def _frozen64(case, g):
    """[B, hkv, m, 128] keys and values of a layer's cache after freeze, as the codes and rows it holds."""
    k, v, q = g["k"], g["v"], g["q"]
    B, hkv, n, R, W = k.shape[0], k.shape[1], k.shape[2], q.shape[1] // k.shape[1], min(case["window"], k.shape[2])
    kp, vp, kw, vw = k[:, :, :n - W], v[:, :, :n - W], k[:, :, n - W:].double(), v[:, :, n - W:].double()
    T = _segments(case)[1]
    kq, vq = _quant64(kp, case["k_bits"]), _quant64(vp, case["v_bits"])
    if T:
        tail = q[:, :, -W:].reshape(B, hkv, R, -1, D).mean(dim=2).double().mean(dim=2, keepdim=True)
        score = (kp[:, :, :n - 2 * W].double() @ tail.transpose(2, 3)).squeeze(3)
        idx = score.topk(T, dim=-1).indices[..., None].expand(-1, -1, -1, D)
        kq.scatter_(2, idx, kp.gather(2, idx).double())
        vq.scatter_(2, idx, vp.gather(2, idx).double())
    return torch.cat([kq, kw], dim=2), torch.cat([vq, vw], dim=2)


def _attend64(q, k, v):
    B, hq = q.shape[:2]
    s = q.double().reshape(B, k.shape[1], -1, D) @ k.transpose(2, 3) / math.sqrt(D)
    return (s.softmax(dim=-1) @ v).reshape(B, hq, 1, D)


def exact(case, seed):
    kind, B, hq, hkv = case["kind"], case["B"], case["hq"], case["hkv"]
    if kind == "freeze":
        return None                        # codes, copied rows and indices: whole numbers and bytes
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed + 7919)
    if kind == "decode":
        g = _inputs(case, seed, n_qry=case["window"])
        k, v = _frozen64(case, g)
        if case["staging"]:
            ks, vs = _rows(gen, B, hkv, case["staging"], D), _rows(gen, B, hkv, case["staging"], D)
            k, v = torch.cat([k, ks.double()], dim=2), torch.cat([v, vs.double()], dim=2)
        return _attend64(g["q_decode"], k, v)
    if kind == "token":
        rows, out = _rows(gen, case["layers"], B, hq + 2 * hkv, 1, D), []
        for i in range(case["layers"]):
            k, v = _frozen64(case, _inputs(case, 1000 * seed + i, n_qry=case["window"]))
            kn, vn = rows[i, :, hq:hq + hkv].double(), rows[i, :, hq + hkv:].double()
            out.append(_attend64(rows[i, :, :hq], torch.cat([k, kn], dim=2), torch.cat([v, vn], dim=2)))
        return torch.stack(out)
    if kind == "answer":
        g, t = _inputs(case, seed, n_qry=case["window"]), case["tokens"]
        q, kn, vn = _rows(gen, t, B, hq, 1, D), _rows(gen, t, B, hkv, 1, D), _rows(gen, t, B, hkv, 1, D)
        (k, v), out, first = _frozen64(case, g), [], 0
        for i in range(t):
            if i + 1 - first == 128:       # the staging buffer is full: its tokens are quantised before this attention
                ks, vs = torch.cat(list(kn[first:i + 1]), dim=2), torch.cat(list(vn[first:i + 1]), dim=2)
                k, v, first = torch.cat([k, _quant64(ks, case["k_bits"])], dim=2), torch.cat([v, _quant64(vs, case["v_bits"])], dim=2), i + 1
            ks, vs = [x.double() for x in kn[first:i + 1]], [x.double() for x in vn[first:i + 1]]
            out.append(_attend64(q[i], torch.cat([k] + ks, dim=2), torch.cat([v] + vs, dim=2)))
        return torch.stack(out)
    g, n, R = _inputs(case, seed), case["n"], hq // hkv
    out = torch.empty(B, hq, n, D, dtype=torch.float64, device="cuda")
    at = torch.arange(n, device="cuda")
    for b in range(B):
        for h in range(hq):
            k, v = g["k"][b, h // R].double(), g["v"][b, h // R].double()
            for i in range(0, n, 4096):
                j = min(i + 4096, n)
                s = (g["q"][b, h, i:j].double() / math.sqrt(D)) @ k[:j].T
                s.masked_fill_(at[None, :j] > at[i:j, None], float("-inf"))
                out[b, h, i:j] = s.softmax(dim=-1) @ v[:j]
    return (out, None) if kind == "hybrid" else out
