"""Workloads of the KIVI cache as a serving program meets them, on one GPU.

``listed()`` are the fixed ones, ``draw(rng)`` gives more from the same ranges.
``prepare`` makes what a program holds before the call, ``run`` is one pass
through the public entry points, ``exact`` restates the result in 64 bits.

Kinds of work:

``decode``    ``KiviCache.decode_attention`` of one layer, one query token per sequence
``steps``     the decode loop over caller-owned tensors: append a token, attend, until the window is full and flushes
              (``_C.append_and_flush`` / ``_C.decode_attention``)
``prefill``   a whole prompt into an empty cache (``_C.append_and_flush``)
``serve``     the dense fp32 cache for unmodified model code (``LayerStore.materialize``)
``operators`` the packed operators of the extension: quantize and dequantize keys and values
``roundtrip`` the fused quantize-dequantize operators of the extension
``sample``    the next-token choice over [batch, vocab] logits
"""
import torch

from intel_kivi_hybrid_b200 import KiviCache, cabi
from intel_kivi_hybrid_b200.extension.loader import kivi_native as _C

_DEV = "cuda"
_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16}


# ---- the cases -----------------------------------------------------------------
def _decode(name, batch, kv_heads, n_rep, tokens, dtype="bfloat16", head_dim=128, group=32, residual=128):
    return {"name": name, "kind": "decode", "batch": batch, "kv_heads": kv_heads, "n_rep": n_rep, "tokens": tokens,
            "dtype": dtype, "head_dim": head_dim, "group": group, "residual": residual}


def listed():
    return [
        # GPT-2-small, one sequence, fp32: 512-token prompt and 200 generated tokens; the smallest call, latency alone
        _decode("gpt2_b1_712_fp32", 1, 12, 1, 712, "float32", head_dim=64),
        # Llama-3-8B shapes, an ordinary batch at a 4k context
        _decode("gqa_b16_4k_bf16", 16, 8, 4, 4096),
        # the throughput workload: batch 64 at a 32k context
        _decode("gqa_b64_32k_bf16", 64, 8, 4, 32768),
        # few long sequences: 128k tokens of history
        _decode("gqa_b4_128k_bf16", 4, 8, 4, 131200),
        # Llama-2-7B shapes: every query head has its own KV head; a ragged context
        _decode("mha_b8_4k_bf16", 8, 32, 1, 4005),
        # fp32 activations at the GQA shapes
        _decode("gqa_b4_8k_fp32", 4, 8, 4, 8192, "float32"),
        # a chat turn: 32 decode steps of a small batch, the last of which flushes a group
        {"name": "steps_b4_2k_bf16", "kind": "steps", "batch": 4, "kv_heads": 8, "n_rep": 4, "quant": 1952, "dtype": "bfloat16",
         "head_dim": 128, "group": 32, "residual": 128},
        # bulk prefill of Llama-2-7B shapes, bf16 and (a ragged prompt) fp32
        {"name": "prefill_b8_8k_bf16", "kind": "prefill", "batch": 8, "kv_heads": 32, "tokens": 8192, "dtype": "bfloat16",
         "head_dim": 128, "group": 32, "residual": 128},
        {"name": "prefill_b2_5k_fp32", "kind": "prefill", "batch": 2, "kv_heads": 32, "tokens": 5003, "dtype": "float32",
         "head_dim": 128, "group": 32, "residual": 128},
        # dense fp32 past_key_values for a model that runs its own attention
        {"name": "serve_b4_8k", "kind": "serve", "batch": 4, "kv_heads": 8, "tokens": 8192, "dtype": "bfloat16",
         "head_dim": 128, "group": 32, "residual": 128},
        # the operators one by one, as a program does that keeps packed tensors itself
        {"name": "operators_b4_4k_fp32", "kind": "operators", "batch": 4, "kv_heads": 8, "tokens": 4096, "dtype": "float32",
         "head_dim": 128, "group": 32},
        # top-k sampling of a batch over a GPT-2 vocabulary
        {"name": "sample_b128_topk", "kind": "sample", "batch": 128, "vocab": 50257, "dtype": "float32", "temperature": 0.8,
         "top_k": 50, "do_sample": True},
    ]


_LARGEST = 64 * 8 * 32768              # (token, unit) pairs of the largest listed case, 128 bytes each


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread evenly over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    case = _any(rng)
    while work(case)["bytes"] > _LARGEST * 128:          # no dearer than the largest listed case
        case = _any(rng)
    return case


def _any(rng):
    kind = rng.choice(["decode"] * 5 + ["steps", "prefill", "prefill", "serve", "operators", "roundtrip", "sample"])
    dtype = rng.choice(["bfloat16", "bfloat16", "float32"])
    if kind == "sample":
        return {"kind": kind, "batch": _log(rng, 1, 256), "vocab": _log(rng, 1000, 130000), "dtype": dtype,
                "temperature": round(rng.uniform(0.3, 1.5), 2), "top_k": rng.choice([0, 1, _log(rng, 2, 500), _log(rng, 2, 500)]),
                "do_sample": rng.random() < 0.8}
    head_dim, group = rng.choice([(128, 32)] * 5 + [(64, 32), (64, 32), (128, 64), (64, 16), (128, 128)])
    if kind in ("operators", "roundtrip"):
        units = _log(rng, 1, 128)
        tokens = group * _log(rng, 1, max(1, 2 ** 19 // units // group))
        return {"kind": kind, "batch": 1, "kv_heads": units, "tokens": tokens, "dtype": dtype, "head_dim": head_dim, "group": group}
    residual = max(group, rng.choice([32, 64, 100, 128, 128, 128, 256]))
    case = {"kind": kind, "batch": _log(rng, 1, 64), "kv_heads": rng.choice([1, 2, 4, 8, 8, 8, 12, 32]), "dtype": dtype,
            "head_dim": head_dim, "group": group, "residual": residual}
    units = case["batch"] * case["kv_heads"]
    if kind == "decode":
        case["n_rep"] = rng.choice([1, 1, 2, 3, 4, 4, 4, 5, 7, 8])
        most = _LARGEST if dtype == "bfloat16" and (head_dim, group) == (128, 32) else _LARGEST // 8
        case["tokens"] = _log(rng, 24, max(25, min(131072, most // units)))
    elif kind == "steps":
        case["n_rep"] = rng.choice([1, 2, 4, 4, 8])
        case["quant"] = group * _log(rng, 1, max(1, min(16384, _LARGEST // 64 // units) // group))
    else:
        case["tokens"] = _log(rng, 130, max(131, min(32768, _LARGEST // 8 // units)))
    return case


# ---- inputs ----------------------------------------------------------------------
def _gen(seed, stream):
    return torch.Generator(device=_DEV).manual_seed(1000 * int(seed) + stream)


def _keys(case, tokens, seed):
    """N(0,1) keys with four outlier channels per head scaled by ten: [B, H, tokens, D]."""
    B, H, D = case["batch"], case["kv_heads"], case["head_dim"]
    g = _gen(seed, 1)
    k = torch.randn(B, H, tokens, D, generator=g, dtype=_DTYPES[case["dtype"]], device=_DEV)
    out = torch.rand(H, D, generator=g, device=_DEV).topk(4, dim=1).indices
    factor = torch.ones(H, D, device=_DEV).scatter_(1, out, 10.0)
    return k.mul_(factor[:, None, :].to(k.dtype))


def _values(case, tokens, seed):
    """N(0,1) values with two per cent of the tokens scaled by eight: [B, H, tokens, D]."""
    B, H, D = case["batch"], case["kv_heads"], case["head_dim"]
    g = _gen(seed, 2)
    v = torch.randn(B, H, tokens, D, generator=g, dtype=_DTYPES[case["dtype"]], device=_DEV)
    loud = torch.rand(B, H, tokens, 1, generator=g, device=_DEV) < 0.02
    return v.mul_(torch.where(loud, 8.0, 1.0).to(v.dtype))


def _queries(case, seed, steps=1):
    B, Hq, D = case["batch"], case["kv_heads"] * case["n_rep"], case["head_dim"]
    return torch.randn(steps, B, Hq, D, generator=_gen(seed, 3), dtype=_DTYPES[case["dtype"]], device=_DEV)


def _logits(case, seed):
    return 3.0 * torch.randn(case["batch"], case["vocab"], generator=_gen(seed, 4), dtype=_DTYPES[case["dtype"]], device=_DEV)


def _split(tokens, group, residual):
    """(quantized, in the window) after `tokens` tokens: whole groups leave while the window holds a full residual length."""
    flushed = (tokens - residual) // group + 1 if tokens >= residual else 0
    return flushed * group, tokens - flushed * group


def _steps(case):
    """Tokens before the first step and number of steps: the window grows from residual - group to residual, then flushes."""
    return case["quant"] + case["residual"] - case["group"], case["group"]


def _store_tensors(case, capacity):
    """Caller-owned packed store and window of one layer, in the order the extension's operators take them."""
    U, D, G, R = case["batch"] * case["kv_heads"], case["head_dim"], case["group"], case["residual"]
    capacity = -(-capacity // G) * G
    zeros = lambda *shape, dtype=torch.float32: torch.zeros(*shape, dtype=dtype, device=_DEV)  # noqa: E731
    return {"k_packed": zeros(U, capacity // G, D * G // 4, dtype=torch.uint8), "k_scales": zeros(U, capacity // G, D),
            "k_zeros": zeros(U, capacity // G, D), "v_packed": zeros(U, capacity, D // 4, dtype=torch.uint8),
            "v_scales": zeros(U, capacity, D // G), "v_zeros": zeros(U, capacity, D // G),
            "k_res": zeros(U, R, D, dtype=_DTYPES[case["dtype"]]), "v_res": zeros(U, R, D, dtype=_DTYPES[case["dtype"]])}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return {"case": case, "logits": _logits(case, seed), "seed": int(seed)}
    D, G = case["head_dim"], case["group"]
    if kind == "decode":
        cache = KiviCache(num_layers=1, head_dim=D, num_kv_heads=case["kv_heads"], device=_DEV, group_size=G,
                          residual_length=case["residual"], max_tokens=case["tokens"])
        cache.ingest_layer(0, _keys(case, case["tokens"], seed), _values(case, case["tokens"], seed))
        return {"case": case, "cache": cache, "q": _queries(case, seed)[0]}
    if kind == "steps":
        held, n = _steps(case)
        U = case["batch"] * case["kv_heads"]
        K, V = (f(case, held + n, seed).flatten(0, 1) for f in (_keys, _values))
        store = _store_tensors(case, case["quant"] + G)
        counters = _C.append_and_flush(K[:, :held], V[:, :held], *store.values(), 0, 0, 0, G)
        q = _queries(case, seed, n).reshape(n, U, case["n_rep"], D)
        need = _C.decode_attention_workspace(U, case["n_rep"], D)
        return {"case": case, "store": store, "counters": counters, "q": q, "new_k": K[:, held:].contiguous(),
                "new_v": V[:, held:].contiguous(), "out": torch.empty_like(q), "workspace": torch.empty(need, dtype=torch.uint8, device=_DEV)}
    K, V = _keys(case, case["tokens"], seed), _values(case, case["tokens"], seed)
    if kind == "prefill":
        return {"case": case, "store": _store_tensors(case, case["tokens"]), "K": K.flatten(0, 1), "V": V.flatten(0, 1)}
    if kind == "serve":
        st = cabi.LayerStore(case["batch"] * case["kv_heads"], D, G, case["residual"], case["tokens"], _DTYPES[case["dtype"]], _DEV)
        st.update(K.flatten(0, 1), V.flatten(0, 1))
        return {"case": case, "store": st}
    # operators: keys are handed over transposed, [B, H, D, S]
    state = {"case": case, "K": K.transpose(2, 3).contiguous(), "V": V}
    n = K.numel()
    for x in ("k", "v"):
        if kind == "operators":
            state[x + "_packed"] = torch.empty(n // 4, dtype=torch.uint8, device=_DEV)
            state[x + "_scales"] = torch.empty(n // G, device=_DEV)
            state[x + "_zeros"] = torch.empty(n // G, device=_DEV)
        state[x + "_out"] = torch.empty(n, device=_DEV)
    return state


# ---- one pass ----------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sample":
        return cabi.sample_tokens(s["logits"], case["temperature"], case["top_k"], case["do_sample"], seed=s["seed"], step=1)
    D, G = case["head_dim"], case["group"]
    if kind == "decode":
        return s["cache"].decode_attention(0, s["q"])
    if kind == "steps":
        arrays = tuple(s["store"].values())
        counters = s["counters"]
        for i in range(s["q"].shape[0]):
            counters = _C.append_and_flush(s["new_k"][:, i:i + 1], s["new_v"][:, i:i + 1], *arrays, *counters, G)
            _C.decode_attention(s["q"][i], *arrays, *counters, s["out"][i], G, s["workspace"])
        return {"out": s["out"], **s["store"]}
    if kind == "prefill":
        _C.append_and_flush(s["K"], s["V"], *s["store"].values(), 0, 0, 0, G)
        return s["store"]
    if kind == "serve":
        return s["store"].materialize()
    if kind == "operators":
        _C.quantize_keys_async(s["K"], s["k_packed"], s["k_scales"], s["k_zeros"], G)
        _C.quantize_values_async(s["V"], s["v_packed"], s["v_scales"], s["v_zeros"], D, G)
        _C.dequantize_keys_async(s["k_packed"], s["k_scales"], s["k_zeros"], s["k_out"], G)
        _C.dequantize_values_async(s["v_packed"], s["v_scales"], s["v_zeros"], s["v_out"], D, G)
        return {n: s[n] for n in ("k_packed", "k_scales", "k_zeros", "k_out", "v_packed", "v_scales", "v_zeros", "v_out")}
    _C.quant_dequant_roundtrip_keys_async(s["K"], s["k_out"], G)
    _C.quant_dequant_roundtrip_values_async(s["V"], s["v_out"], D, G)
    return {n: s[n] for n in ("k_out", "v_out")}


# ---- what a pass cannot do without ---------------------------------------------------
def _attention_work(case, quant, res):
    U, D, G, esz = case["batch"] * case["kv_heads"], case["head_dim"], case["group"], _DTYPES[case["dtype"]].itemsize
    return {"bytes": U * (quant * (D // 2 + 16 * D // G) + res * 2 * D * esz) + 2 * U * case["n_rep"] * D * esz,
            "flops": 4 * U * case["n_rep"] * (quant + res) * D}


def work(case):
    kind = case["kind"]
    esz = _DTYPES[case["dtype"]].itemsize
    if kind == "sample":
        return {"bytes": case["batch"] * (case["vocab"] * esz + 8), "flops": case["batch"] * case["vocab"] * (4 if case["do_sample"] else 1)}
    U, D, G = case["batch"] * case["kv_heads"], case["head_dim"], case["group"]
    if kind == "decode":
        return _attention_work(case, *_split(case["tokens"], G, case["residual"]))
    if kind == "steps":
        n = _steps(case)[1]
        w = [_attention_work(case, case["quant"], case["residual"] - G + i + 1) for i in range(n - 1)]
        w.append(_attention_work(case, case["quant"] + G, case["residual"] - G))
        flush = U * G * (2 * D * esz + D // 2 + 16 * D // G)
        return {"bytes": sum(x["bytes"] for x in w) + n * U * 4 * D * esz + flush, "flops": sum(x["flops"] for x in w)}
    elems = 2 * U * case["tokens"] * D
    if kind in ("prefill", "serve"):
        quant, res = _split(case["tokens"], G, case["residual"])
        packed, window = U * quant * (D // 2 + 16 * D // G), U * res * 2 * D * esz
        if kind == "prefill":
            return {"bytes": elems * esz + packed + window, "flops": 6 * elems}
        return {"bytes": packed + window + elems * 4, "flops": 2 * elems}
    if kind == "operators":          # the packed tensors are written, and read again by the second pair of calls
        return {"bytes": elems * esz + 2 * (elems // 4 + elems // G * 8) + elems * 4, "flops": 8 * elems}
    return {"bytes": elems * esz + elems * 4, "flops": 8 * elems}


def tolerance(case):
    kind = case["kind"]
    if kind in ("decode", "steps"):
        # fp32: sums of thousands of terms in another order; bf16: the output's own rounding on both sides
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 1e-2}
    if kind == "sample":
        return {"differ": 0.01}      # a draw that lands on the boundary between two tokens
    return "exact"                   # quantization and dequantization are defined to the bit


# ---- 64-bit restatement ----------------------------------------------------------------
def _codes(x, group):
    """(codes, scale, zero) of consecutive runs of `group` elements of fp32 x; the codes are defined by fp32 arithmetic."""
    g = x.reshape(-1, group)
    zero = g.amin(1, keepdim=True)
    scale = (g.amax(1, keepdim=True) - zero) / torch.full((), 3.0, device=x.device) + 1e-10
    t = (g - zero) / scale
    low = torch.floor(t)
    return (low + (t - low >= 0.5)).clamp_(0, 3), scale, zero


def _dense(x, group, over_tokens):
    """What the cache serves for [H, T, D] fp32 tokens that have been quantized, in 64 bits."""
    y = x.transpose(1, 2).contiguous() if over_tokens else x.contiguous()
    code, scale, zero = _codes(y, group)
    y = (code.double() * scale.double() + zero.double()).reshape(y.shape)
    return y.transpose(1, 2) if over_tokens else y


def _attend(q, k, v):
    """q [H, n_rep, D], k and v [H, T, D], all 64-bit."""
    w = torch.softmax(q @ k.transpose(1, 2) * q.shape[-1] ** -0.5, dim=-1)
    return w @ v


def exact(case, seed):
    kind = case["kind"]
    if kind == "sample":
        return None
    D, G = case["head_dim"], case["group"]
    B, H = case["batch"], case["kv_heads"]
    if kind == "steps":
        held, n = _steps(case)
        K, V, q = _keys(case, held + n, seed), _values(case, held + n, seed), _queries(case, seed, n)
        out = torch.empty(n, B * H, case["n_rep"], D, dtype=torch.float64, device=_DEV)
        for b in range(B):
            k, v = K[b].float(), V[b].float()
            last = case["quant"] + G
            kq, vq = _dense(k[:, :last], G, True), _dense(v[:, :last], G, False)
            for i in range(n):
                quant = last if i == n - 1 else case["quant"]
                kk, vv = (torch.cat([x[:, :quant], y[:, quant:held + i + 1].double()], 1) for x, y in ((kq, k), (vq, v)))
                out[i, b * H:(b + 1) * H] = _attend(q[i, b].double().reshape(H, -1, D), kk, vv)
        return {"out": out, **{name: None for name in ("k_packed", "k_scales", "k_zeros", "v_packed", "v_scales", "v_zeros", "k_res", "v_res")}}
    K, V = _keys(case, case["tokens"], seed), _values(case, case["tokens"], seed)
    if kind in ("operators", "roundtrip"):
        got = {}
        for name, x in (("k", K.transpose(2, 3).contiguous()), ("v", V)):
            code, scale, zero = _codes(x.float(), G)
            dense = (code.double() * scale.double() + zero.double()).reshape(-1)
            got.update({name + "_packed": None, name + "_scales": scale.double().reshape(-1), name + "_zeros": zero.double().reshape(-1), name + "_out": dense})
        return got if kind == "operators" else {n: got[n] for n in ("k_out", "v_out")}
    quant, _ = _split(case["tokens"], G, case["residual"])
    if kind == "prefill":
        # key scales and zeros; the codes are bytes, and the values' have an order of the store's own
        scales = torch.zeros(B * H, -(-case["tokens"] // G), D, dtype=torch.float64, device=_DEV)
        zeros = torch.zeros_like(scales)
        for u in range(B * H if quant else 0):
            _, scale, zero = _codes(K[u // H, u % H, :quant].float().t().contiguous(), G)
            scales[u, :quant // G], zeros[u, :quant // G] = (x.reshape(D, quant // G).t().double() for x in (scale, zero))
        return {"k_scales": scales, "k_zeros": zeros, **{n: None for n in ("k_packed", "v_packed", "v_scales", "v_zeros", "k_res", "v_res")}}

    def whole(x, over_tokens):
        x = x.float()
        if not quant:
            return x.double()
        return torch.cat([_dense(x[:, :quant], G, over_tokens), x[:, quant:].double()], 1)

    if kind == "serve":
        return tuple(torch.cat([whole(x[b], over) for b in range(B)]) for x, over in ((K, True), (V, False)))
    q = _queries(case, seed)[0]
    out = torch.empty(B, H * case["n_rep"], D, dtype=torch.float64, device=_DEV)
    for b in range(B):
        out[b] = _attend(q[b].double().reshape(H, -1, D), whole(K[b], True), whole(V[b], False)).reshape(-1, D)
    return out
