"""What a user of this framework has it do, as cases to time.

The framework is the quantised matrix path of an inference engine, so the cases are the calls and call sequences such
an engine makes: one matrix-vector product, a recorded decode token of a dense and of two mixture-of-experts models,
a prompt's matrix products with bf16 and with f32 activations, the batched matrix-vector product of short prompts,
and the routed experts of a prompt. Weights are random GGUF blocks with the value ranges of real ones; activations
are N(0, 1).

One context, stream and dispatch object serve every case of a process, as one engine would own them.
"""
import torch

import zinc_b200 as zb
from zinc_b200 import synth
from zinc_b200.decode_step import DecodeStep, StepShape
from zinc_b200.moe_step import MoeDecode, MoePrefill, MoeShape

TYPES = {"q4_k": zb.Q4_K, "q5_k": zb.Q5_K, "q6_k": zb.Q6_K, "q8_0": zb.Q8_0, "mxfp4": zb.MXFP4}


def listed():
    return [
        # The smallest products of a token: a Q8_0 shared-expert gate of a 2048-wide model, called on its own.
        {"name": "matvec_q8_0_512x2048", "op": "matvec", "type": "q8_0", "M": 512, "K": 2048},
        # One attention projection of an 8B model, called on its own.
        {"name": "matvec_q4_k_4096x4096", "op": "matvec", "type": "q4_k", "M": 4096, "K": 4096},
        # Every projection of one token of an 8B dense model, Q4_K_M mix, recorded once and replayed per token.
        {"name": "decode_dense_8b", "op": "decode", "hidden": 4096, "layers": 36, "q_dim": 4096, "kv_dim": 1024,
         "ffn": 12288, "vocab": 151936},
        # The expert layers of one token: 256 experts, top-8 and a shared one, Q4_K / Q6_K.
        {"name": "moe_decode_kquant", "op": "moe_decode", "arch": "kquant", "hidden": 2048, "experts": 256, "top_k": 8,
         "ffn": 512, "layers": 40},
        # The expert layers of one token: 32 experts, top-4, MXFP4, with biases.
        {"name": "moe_decode_mxfp4", "op": "moe_decode", "arch": "mxfp4", "hidden": 2880, "experts": 32, "top_k": 4,
         "ffn": 2880, "layers": 24},
        # A short prompt's key projection: few rows, a ragged number of tokens.
        {"name": "gemm_q4_k_1024x4096_t77", "op": "gemm", "type": "q4_k", "act": "bf16", "M": 1024, "K": 4096, "T": 77},
        # A prompt's gate or up projection.
        {"name": "gemm_q4_k_12288x4096_t512", "op": "gemm", "type": "q4_k", "act": "bf16", "M": 12288, "K": 4096,
         "T": 512},
        # A long prompt's down projection: the largest dense product.
        {"name": "gemm_q6_k_4096x12288_t2048", "op": "gemm", "type": "q6_k", "act": "bf16", "M": 4096, "K": 12288,
         "T": 2048},
        # A prompt's projection with the activations left in f32.
        {"name": "gemm_f32_q4_k_4096x4096_t658", "op": "gemm", "type": "q4_k", "act": "f32", "M": 4096, "K": 4096,
         "T": 658},
        # The same for a short prompt through the batched matrix-vector call.
        {"name": "batch_q4_k_12288x4096_c105", "op": "batch", "type": "q4_k", "M": 12288, "K": 4096, "T": 105},
        # The routed experts of a prompt, many experts with few tokens each.
        {"name": "moe_prefill_kquant_t512", "op": "moe_prefill", "arch": "kquant", "hidden": 2048, "experts": 256,
         "top_k": 8, "ffn": 512, "T": 512},
        # The routed experts of a prompt, few experts with many tokens each.
        {"name": "moe_prefill_mxfp4_t1024", "op": "moe_prefill", "arch": "mxfp4", "hidden": 2880, "experts": 32,
         "top_k": 4, "ffn": 2880, "T": 1024},
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def _cols(rng, name, lo, hi):
    """A number of columns that the type's blocks divide."""
    b = synth.BLOCK[TYPES[name]][0]
    return b * _log(rng, max(1, lo // b), hi // b)


def draw(rng):
    op = rng.choice(["matvec", "matvec", "decode", "moe_decode", "gemm", "gemm", "gemm", "batch", "moe_prefill"])
    if op == "matvec":
        t = rng.choice(sorted(TYPES))
        return {"op": op, "type": t, "M": _log(rng, 128, 65536), "K": _cols(rng, t, 512, 14336)}
    if op == "decode":
        return {"op": op, "hidden": 256 * rng.randint(4, 16), "layers": _log(rng, 2, 36),
                "q_dim": 256 * rng.randint(4, 16), "kv_dim": 128 * rng.randint(2, 8), "ffn": 256 * rng.randint(6, 48),
                "vocab": _log(rng, 16001, 151936)}
    if op in ("gemm", "batch"):
        t = rng.choice(["q4_k", "q4_k", "q6_k", "q6_k", "q5_k", "q8_0"])
        c = {"op": op, "type": t, "M": _log(rng, 256, 12288), "K": _cols(rng, t, 1024, 12288),
             "T": _log(rng, 16, 2048) if op == "gemm" else _log(rng, 2, 300)}
        if op == "gemm":
            c["act"] = rng.choice(["bf16", "bf16", "f32"])
        # no larger than the largest listed product of its kind
        most = 12288 * 4096 * 105 if op == "batch" else 4096 * 12288 * 2048 if c["act"] == "bf16" else 4096 * 4096 * 658
        c["T"] = min(c["T"], max(2, most // (c["M"] * c["K"])))
        return c
    if rng.random() < 0.5:
        c = {"op": op, "arch": "kquant", "hidden": 256 * rng.randint(4, 16), "experts": rng.choice([64, 96, 128, 256]),
             "top_k": rng.randint(4, 8), "ffn": 256 * rng.randint(2, 4)}
    else:
        c = {"op": op, "arch": "mxfp4", "hidden": 64 * rng.randint(16, 45), "experts": rng.choice([16, 24, 32]),
             "top_k": rng.randint(2, 4), "ffn": 64 * rng.randint(16, 45)}
    if op == "moe_decode":
        c["layers"] = _log(rng, 2, 24)
        if c["arch"] == "kquant":   # the selected experts of a token: no more than the listed 40 layers read
            c["layers"] = max(1, min(c["layers"], 40 * 2048 * 512 * 9 // (c["hidden"] * c["ffn"] * (c["top_k"] + 1))))
    else:
        c["T"] = _log(rng, 16, 1024)
        if c["arch"] == "kquant":   # no more weights than the listed layer has
            while c["hidden"] * c["ffn"] * c["experts"] > 2048 * 512 * 256:
                c["experts"] //= 2
    return c


# ---- what a program has in hand before the call ------------------------------------------------------
_engine = None


class Engine:
    """The stream, context and dispatch object of the process."""

    def __init__(self):
        self.stream = torch.cuda.Stream()
        self.ctx = zb.Context(torch.cuda.current_device(), stream=self.stream.cuda_stream)
        self.dd = zb.DmmvDispatch(self.ctx)


def engine():
    global _engine
    if _engine is None:
        _engine = Engine()
    return _engine


class Recording:
    """A sequence of calls recorded once; freed with the state that owns it."""

    def __init__(self, ctx, record):
        self.ctx = ctx
        record()   # every kernel variant has run once before it is recorded
        ctx.begin_record()
        record()
        self.handle = ctx.end_record()

    def __del__(self):
        torch.cuda.synchronize()
        self.ctx.free_recording(self.handle)


def _moe_shape(case, layers):
    k = case["arch"] == "kquant"
    return MoeShape(hidden=case["hidden"], n_experts=case["experts"], top_k=case["top_k"], ffn=case["ffn"],
                    t_gate_up=zb.Q4_K if k else zb.MXFP4, t_down=zb.Q6_K if k else zb.MXFP4,
                    rule=zb.ROUTE_SOFTMAX_ALL_RENORM if k else zb.ROUTE_TOPK_THEN_SOFTMAX, shared=k, oai=not k,
                    n_layers=layers, biases=not k)


def prepare(case, seed):
    e = engine()
    dev = torch.device("cuda", torch.cuda.current_device())
    s = {"op": case["op"], "dd": e.dd, "ctx": e.ctx, "case": case}
    with torch.cuda.stream(e.stream):
        gen = torch.Generator(device=dev).manual_seed(7919 * seed + 1)

        def normal(*shape):
            return torch.randn(*shape, device=dev, generator=gen)

        if case["op"] in ("matvec", "gemm", "batch"):
            t, M, K = TYPES[case["type"]], case["M"], case["K"]
            s["type"] = t
            s["W"] = synth.torch_quant_matrix(t, M, K, dev, 104729 * seed + 2)
            if case["op"] == "matvec":
                s["x"], s["y"] = normal(K), torch.zeros(M, device=dev)
            else:
                T = case["T"]
                s["X"] = normal(T, K)
                s["act"] = zb.F32
                if case.get("act") == "bf16":
                    s["X"], s["act"] = s["X"].to(torch.bfloat16), zb.BF16
                s["Y"] = torch.zeros(T, M, device=dev)
        elif case["op"] == "decode":
            step = DecodeStep.build(torch, e.dd, StepShape(
                hidden=case["hidden"], n_layers=case["layers"], q_dim=case["q_dim"], kv_dim=case["kv_dim"],
                ffn=case["ffn"], vocab=case["vocab"]), seed=seed)
            for buf in (step.x_norm, step.attn_out, step.ffn_act_in):
                buf.copy_(normal(*buf.shape))
            s["step"], s["recording"] = step, Recording(e.ctx, step.record)
            s["out"] = [step.hidden, step.logits, step.q, step.k, step.v, step.act]
        elif case["op"] == "moe_decode":
            shape = _moe_shape(case, case["layers"])
            step = MoeDecode.build(torch, e.dd, shape, seed=seed)
            s["step"], s["recording"] = step, Recording(e.ctx, step.record)
            slots = step.routing.numel() // 2
            s["out"] = [step.hidden, step.logits, step.routing[:slots], step.routing[slots:].view(torch.float32)]
        else:
            s["step"] = MoePrefill.build(torch, e.dd, _moe_shape(case, 1), case["T"], seed=seed)
    e.ctx.submit_and_wait()
    return s


# ---- one pass ----------------------------------------------------------------------------------------
def run(state):
    op, dd = state["op"], state["dd"]
    if op in ("decode", "moe_decode"):
        state["ctx"].replay(state["recording"].handle)
        return state["out"]
    if op == "moe_prefill":
        dd.setWorkspace(state["step"].workspace)
        state["step"].record()
        return state["step"].hidden
    c = state["case"]
    M, K = c["M"], c["K"]
    if op == "matvec":
        dd.recordDispatch(state["type"], state["W"], state["x"], state["y"], M, K)
        return state["y"]
    if op == "gemm":
        dd.recordMulMm(state["type"], state["W"], state["X"], state["Y"], M, c["T"], K, K, M, act_type=state["act"])
    else:
        dd.recordBatchDispatchPush(state["type"], state["W"], state["X"], state["Y"], M, K, 0, 0, 0, c["T"])
    return state["Y"]


# ---- what a pass cannot do without -------------------------------------------------------------------
def _mat(t, M, K):
    return M * zb.row_bytes(t, K)


def work(case):
    op = case["op"]
    if op in ("matvec", "gemm", "batch"):
        M, K, T = case["M"], case["K"], case.get("T", 1)
        x = 2 if case.get("act") == "bf16" else 4
        return {"bytes": _mat(TYPES[case["type"]], M, K) + T * (x * K + 4 * M), "flops": 2 * M * K * T}
    H = case["hidden"]
    if op == "decode":
        q, kv, f, L, v = case["q_dim"], case["kv_dim"], case["ffn"], case["layers"], case["vocab"]
        weights = L * (_mat(zb.Q4_K, q + 2 * kv, H) + _mat(zb.Q4_K, H, q) + _mat(zb.Q4_K, 2 * f, H) +
                       _mat(zb.Q6_K, H, f)) + _mat(zb.Q6_K, v, H)
        elements = L * ((q + 2 * kv) * H + H * q + 3 * f * H) + v * H
        return {"bytes": weights + 4 * (3 * H + q + 2 * f + v + q + 2 * kv), "flops": 2 * elements}
    E, k, f = case["experts"], case["top_k"], case["ffn"]
    shape = _moe_shape(case, case.get("layers", 1))
    one = shape.expert_bytes()
    if op == "moe_decode":
        n = k + (1 if shape.shared else 0)
        biases = 4 * (E + k * (2 * f + H)) if shape.biases else 0
        return {"bytes": shape.n_layers * (shape.layer_weight_bytes() + biases) + 4 * (3 * H + E + 4 * n),
                "flops": shape.n_layers * 2 * (n * 3 * H * f + E * H)}
    T = case["T"]
    # experts that T tokens' top-k of independent uniform choices reach
    reached = E * (1 - (1 - k / E) ** T)
    return {"bytes": int(reached * one) + 4 * T * (3 * H + 2 * k), "flops": 2 * T * k * 3 * H * f}


def tolerance(case):
    # bf16 operands: weights and activations carry 8 bits, rounded once each; sums are f32
    if case["op"] == "moe_prefill" or (case["op"] == "gemm" and case["act"] == "bf16"):
        return {"rel": 5e-3, "max": 5e-2}
    # f32 activations and sums over quantised weights
    return {"rel": 1e-5, "max": 1e-4}
