"""The work that users of this framework have it do, as timed cases.

Each case is one pass through the public entry points on synthetic data of the benchmark's distributions:
``W4A4Linear`` in its three configurations, the W4A8 pair, the activation quantisers, the MoE layer and the
Qwen3-shaped prefill.  ``listed()`` names typical points, ``draw()`` spreads over the ranges around them.
"""
import torch

GROUP = 128
HIDDEN, INTER, EXPERTS, TOP_K = 2048, 768, 128, 8      # the MoE layer of the benchmark configuration


def listed():
    return [
        # one user decoding: a token through the fused QKV projection; launches and host work count
        {"name": "decode_1", "kind": "linear", "mode": "group", "M": 1, "K": 4096, "N": 6144},
        # a decoding batch through gate+up, the widest matrix of the model; the weights' bytes count
        {"name": "decode_16", "kind": "linear", "mode": "group", "M": 16, "K": 4096, "N": 24576},
        # a larger batch, or a short prompt, of odd length through the long-K down projection
        {"name": "batch_100", "kind": "linear", "mode": "group", "M": 100, "K": 12288, "N": 4096},
        # a prompt of ordinary, odd length
        {"name": "prompt_1000", "kind": "linear", "mode": "group", "M": 1000, "K": 4096, "N": 6144},
        # a prefill batch, the largest linear of the sweep
        {"name": "prefill_8192", "kind": "linear", "mode": "group", "M": 8192, "K": 4096, "N": 24576},
        # the per-channel configuration on a prompt
        {"name": "channel_2048", "kind": "linear", "mode": "channel", "M": 2048, "K": 4096, "N": 4096},
        # the best-quality configuration: asymmetric codes, clipping at 0.95 and SmoothQuant factors
        {"name": "enhanced_1500", "kind": "linear", "mode": "enhanced", "M": 1500, "K": 4096, "N": 6144},
        # int8 activations against int4 weights held as int8
        {"name": "w4a8_512", "kind": "linear", "mode": "w4a8", "M": 512, "K": 12288, "N": 4096},
        # activation quantisation by itself, for callers that run their own GEMM
        {"name": "quantise_16384", "kind": "quantise", "mode": "group", "M": 16384, "K": 12288},
        # the MoE layer while decoding: few tokens, nearly every expert touched
        {"name": "moe_decode_64", "kind": "moe", "T": 64},
        # the MoE layer of the benchmark configuration
        {"name": "moe_4096", "kind": "moe", "T": 4096},
        # a model's layer end to end, after the embedding: norms, attention and the four linears
        {"name": "prefill_8x512", "kind": "prefill", "batch": 8, "seq": 512, "layers": 1},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choices(["linear", "quantise", "moe", "prefill"], [6, 1, 2, 1])[0]
    if kind == "linear":
        mode = rng.choices(["group", "channel", "enhanced", "w4a8"], [4, 2, 2, 2])[0]
        # the model's own widths at times, else any K of whole groups and any N; some N are not even multiples of 8
        if rng.random() < 0.4:
            K, N = rng.choice([(4096, 6144), (4096, 4096), (4096, 24576), (12288, 4096), (2560, 9728), (9728, 2560)])
        else:
            K, N = GROUP * _log(rng, 8, 96), _log(rng, 1000, 16000)
            N = N if rng.random() < 0.2 else (N + 7) // 8 * 8
        return {"kind": "linear", "mode": mode, "M": _log(rng, 1, 8192), "K": K, "N": N}
    if kind == "quantise":
        return {"kind": "quantise", "mode": rng.choice(["group", "channel", "enhanced", "w4a8"]), "M": _log(rng, 64, 16384),
                "K": GROUP * _log(rng, 8, 96)}
    if kind == "moe":
        return {"kind": "moe", "T": _log(rng, 8, 4096)}
    return {"kind": "prefill", "batch": rng.randint(1, 8), "seq": _log(rng, 64, 512), "layers": 1}


def _activations(gen, M, K):
    """N(0, 1) with 8 channels per 4096 scaled by 20 (at least one)."""
    x = torch.randn(M, K, device="cuda", generator=gen)
    hot = torch.randperm(K, device="cuda", generator=gen)[: max(1, round(K * 8 / 4096))]
    x[:, hot] *= 20.0
    return x.to(torch.bfloat16)


def _weights(gen, *shape):
    return (torch.randn(*shape, device="cuda", generator=gen) * 0.02).to(torch.bfloat16)


def prepare(case, seed):
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.linear import W4A4Linear
    from fp8_inference_toolkit_b200.moe import MoEWeights, moe_route
    from fp8_inference_toolkit_b200.qwen3 import Qwen3Config, Qwen3Prefill

    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if case["kind"] in ("linear", "quantise"):
        M, K, mode = case["M"], case["K"], case["mode"]
        x = _activations(gen, M, K)
        if mode == "enhanced":
            x += 0.75                                     # what asymmetric codes are for
        state["x"] = x
    if case["kind"] == "linear":
        N = case["N"]
        w = _weights(gen, N, K)
        if mode == "w4a8":
            packed, scale = ops.static_int4_weight_quant(w)
            state["w"], state["w_scale"] = ops.unpack_int4_to_int8(packed, K), scale
        else:
            kwargs = {}
            if mode == "enhanced":
                kwargs = {"asymmetric": True, "clip_ratio": 0.95, "layer_name": "proj",
                          "calibration_stats": {"proj": {"input_absmax": x.abs().amax(0).float()}}}
            lin = W4A4Linear(K, N, per_channel=mode == "channel", device="cuda", **kwargs)
            lin.weight.data.copy_(w)
            state["linear"] = lin.quantize_()
    elif case["kind"] == "moe":
        state["x"] = torch.randn(case["T"], HIDDEN, device="cuda", generator=gen).to(torch.bfloat16)
        logits = torch.randn(case["T"], EXPERTS, device="cuda", generator=gen)
        state["ids"], state["w"] = moe_route(logits, TOP_K)
        state["experts"] = MoEWeights.quantize(_weights(gen, EXPERTS, 2 * INTER, HIDDEN), _weights(gen, EXPERTS, HIDDEN, INTER))
    elif case["kind"] == "prefill":
        model = Qwen3Prefill(Qwen3Config(layers=case["layers"]), device="cuda", seed=seed)
        model.embed.weight.data.normal_(generator=gen)
        state["model"] = model
        state["ids"] = torch.randint(0, model.cfg.vocab, (case["batch"], case["seq"]), device="cuda", generator=gen)
    return state


def run(state):
    from fp8_inference_toolkit_b200 import ops
    from fp8_inference_toolkit_b200.moe import moe_layer

    case = state["case"]
    if case["kind"] == "prefill":
        return state["model"](state["ids"])
    if case["kind"] == "moe":
        return moe_layer(state["x"], state["ids"], state["w"], state["experts"])
    x, mode = state["x"], case["mode"]
    if case["kind"] == "quantise":
        if mode == "group":
            return ops.dynamic_int4_quant_grouped(x, GROUP)
        if mode == "channel":
            return ops.dynamic_int4_quant(x)
        if mode == "enhanced":
            return ops.dynamic_int4_quant_asymmetric_clipped_grouped(x, GROUP, 0.95)
        return ops.dynamic_int8_quant(x)
    if mode == "w4a8":
        M, K, N = case["M"], case["K"], case["N"]
        q, scale = ops.dynamic_int8_quant(x)
        out = torch.empty((M, N), dtype=torch.bfloat16, device=x.device)
        ops.cutlass_w4a8_scaled_mm(q, state["w"], scale, state["w_scale"], out, M, N, K)
        return out
    return state["linear"](x)


def _quantised_bytes(rows, K, mode):
    """Codes and scales of `rows` rows."""
    G = K // GROUP
    return {"group": rows * K // 2 + 4 * rows * G, "channel": rows * K // 2 + 4 * rows,
            "enhanced": rows * K // 2 + 8 * rows * G, "w4a8": rows * K + 4 * rows}[mode]


def work(case):
    if case["kind"] == "linear":
        M, K, N = case["M"], case["K"], case["N"]
        return {"bytes": 2 * M * K + _quantised_bytes(N, K, case["mode"]) + 2 * M * N, "flops": 2 * M * N * K}
    if case["kind"] == "quantise":
        M, K = case["M"], case["K"]
        return {"bytes": 2 * M * K + _quantised_bytes(M, K, case["mode"]), "flops": 4 * M * K}
    if case["kind"] == "moe":
        T = case["T"]
        touched = EXPERTS * (1 - (1 - TOP_K / EXPERTS) ** T)      # experts that at least one token goes to
        weights = _quantised_bytes(2 * INTER, HIDDEN, "group") + _quantised_bytes(HIDDEN, INTER, "group")
        return {"bytes": 4 * T * HIDDEN + 8 * T * TOP_K + touched * weights, "flops": 2 * T * TOP_K * 3 * INTER * HIDDEN}
    tokens, seq, layers = case["batch"] * case["seq"], case["seq"], case["layers"]
    shapes = [(4096, 6144), (4096, 4096), (4096, 24576), (12288, 4096)]
    weights = sum(_quantised_bytes(n, k, "group") for k, n in shapes)
    linears = sum(2 * tokens * k * n for k, n in shapes)
    attention = 2 * tokens * (seq + 1) * 32 * 128                  # causal scores and weighted sum, 32 heads of 128
    return {"bytes": 8 * tokens + 4 * tokens * 4096 + layers * weights, "flops": layers * (linears + attention)}


def tolerance(case):
    if case["kind"] == "quantise":
        return "exact"
    if case["kind"] in ("linear", "moe"):
        # one rounding to bf16 of sums that fp32 holds, which may be added in another order: 1.7e-3 against the same sums
        # in float64 (the MoE layer's SwiGLU and second quantiser taken along in float64 too)
        return {"rel": 7e-3}
    # int4 codes of intermediate activations that sit on a rounding boundary move with the last bit of what comes before
    # them, and attention passes that on: 0.04 between the layer with fused and with separate quantisers, and with the
    # norms' sums in float64
    return {"rel": 0.16}
