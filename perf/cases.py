"""What a user of flh_b200 has it do, as measurable cases.

The framework is the W4A4 inference path: quantise the activations of a linear (with or without the online Hadamard
transform), multiply packed int4 codes with packed int4 weights, and do that for every linear of a decoder in prefill and
decode.  Three kinds of case stand for it, all through the classes a program uses:

  linear    ActQuantizer -> LinearFLH, the unit the package is dropped in for: one token, decode batches, ragged chunks,
            whole prompts; both activation modes (group_sym: FLH's own contract, group-128 scales on both sides;
            token_asym: per-token scale and zero-point, per-channel weight scales, full-width transform in front of the
            down projection); float16 and bfloat16; with and without bias and the int8 copy of the weights
  quant     ActQuantizer alone, the memory-bound half, at sizes where it is timed by itself
  decoder   Decoder.forward with its KV cache: prefill, and decode steps replayed from a CUDA graph as a server does

Sizes are the linears of the 7B- and 70B-shaped decoders of flh_b200.model (and the shards of the latter over 8 ranks), the
width 14336 of the tests and the benchmark, and token counts from 1 to 16,384.  Calibration and weight conversion run once
per model, mostly in torch's linear algebra, and are not part of the path.
"""
import math

import torch

from flh_b200.model import Decoder, DecoderConfig, LLAMA2_7B, LLAMA3_70B
from flh_b200.nn import ActQuantizer, LinearFLH

GROUP = 128
VOCAB = 32000
# (K, N, the activation is SiLU(gate) * up: the online transform goes in front of this linear in token_asym mode)
LINEARS = (
    (4096, 12288, False), (4096, 4096, False), (4096, 22016, False), (11008, 4096, True),        # 7B: qkv, o, gate_up, down
    (8192, 10240, False), (8192, 8192, False), (8192, 57344, False), (28672, 8192, True),        # 70B: qkv, o, gate_up, down
    (8192, 1280, False), (1024, 8192, False), (8192, 7168, False), (3584, 8192, True),           # 70B over 8 ranks
    (14336, 4096, True),
)
QUANT_WIDTHS = (3584, 4096, 8192, 11008, 14336, 28672)
MAX_LINEAR = 8192 * 4096 * 22016       # largest M * K * N of a linear
MAX_QUANT = 16384 * 4096               # largest M * K of a quantiser alone


def linear(name, mode, m, k, n, hadamard, dtype="float16", bias=False, prepack=False):
    return dict(name=name, kind="linear", mode=mode, m=m, k=k, n=n, hadamard=hadamard, dtype=dtype, bias=bias, prepack=prepack)


def quant(name, mode, m, k, hadamard, dtype="float16"):
    return dict(name=name, kind="quant", mode=mode, m=m, k=k, hadamard=hadamard, dtype=dtype)


def decoder(name, shape, mode, layers, batch, seq, ctx, prepack=False):
    return dict(name=name, kind="decoder", shape=shape, mode=mode, layers=layers, batch=batch, seq=seq, ctx=ctx, prepack=prepack)


def listed():
    return [
        # one token of one conversation, a fused q/k/v projection in FLH's own scale layout: the smallest call
        linear("token1_group_qkv", "group_sym", 1, 4096, 12288, False),
        # a small decode batch through the down projection with the online 172 x 64 transform
        linear("decode16_token_down", "token_asym", 16, 11008, 4096, True),
        # a decode batch of 64 through the largest kind of weight (half of the 70B gate/up projection), FLH's scale layout
        linear("decode64_group_70b", "group_sym", 64, 8192, 28672, False),
        # a ragged chunk of mixed requests (chunked prefill), bfloat16, with a bias
        linear("chunk333_token_bf16", "token_asym", 333, 4096, 22016, False, dtype="bfloat16", bias=True),
        # a whole prompt through q/k/v, FLH's scale layout (the GEMM of the reference's own benchmark)
        linear("prompt2048_group_qkv", "group_sym", 2048, 4096, 12288, False),
        # four prompts through gate/up, per-token and per-channel scales, no prepared copy of the weights
        linear("prompts8192_token_up", "token_asym", 8192, 4096, 22016, False),
        # the quantiser with the full-width transform at its headline size
        quant("quant_token_16384", "token_asym", 16384, 4096, True),
        # the same at the factored width 28 x 512, bfloat16, a ragged token count
        quant("quant_token_1531_bf16", "token_asym", 1531, 14336, True, dtype="bfloat16"),
        # group-128 transform and symmetric codes (FLH's kernel contract), ragged
        quant("quant_group_6007", "group_sym", 6007, 4096, True),
        # prefill of one prompt, 7B-shaped, the default wiring (group_sym), into its KV cache
        decoder("prefill_7b_group", "7b", "group_sym", 2, 1, 2048, 0),
        # prefill of four prompts, 70B-shaped, per-token wiring with the int8 copy of the weights kept: the largest case
        decoder("prefill_70b_token", "70b", "token_asym", 1, 4, 2048, 0, prepack=True),
        # one decode step of 16 conversations at 1,024 tokens of context, 7B-shaped, a recorded step replayed
        decoder("decode_7b_token", "7b", "token_asym", 4, 16, 1, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("linear", "quant", "decoder"), (6, 3, 2))[0]
    mode = rng.choice(("group_sym", "token_asym"))
    dtype = rng.choice(("float16", "bfloat16")) if mode == "token_asym" else "float16"
    if kind == "linear":
        k, n, silu = rng.choice(LINEARS)
        m = _log_int(rng, 1, min(8192, MAX_LINEAR // (k * n)))
        had = silu if mode == "token_asym" else rng.random() < 0.25
        case = linear("", mode, m, k, n, had, dtype, rng.random() < 0.2, mode == "token_asym" and rng.random() < 0.3)
    elif kind == "quant":
        k = rng.choice(QUANT_WIDTHS)
        case = quant("", mode, _log_int(rng, 1, MAX_QUANT // k), k, rng.random() < 0.75, dtype)
    else:
        shape = rng.choice(("7b", "70b"))
        layers = rng.randint(1, 2) if shape == "7b" else 1
        if rng.random() < 0.5:
            case = decoder("", shape, mode, layers, _log_int(rng, 1, 4), _log_int(rng, 16, 1024), 0, mode == "token_asym" and rng.random() < 0.5)
        else:
            case = decoder("", shape, mode, layers, _log_int(rng, 1, 64), 1, _log_int(rng, 64, 1536))
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------------------- preparation
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _activations(g, m, k, dtype):
    """N(0, 1) with 0.1 % of the channels x 20, the value law of the framework's tests and benchmark."""
    x = torch.randn(m, k, device="cuda", generator=g)
    x[:, torch.randperm(k, device="cuda", generator=g)[:max(1, round(k * 0.001))]] *= 20.0
    return x.to(getattr(torch, dtype))


def _quantizer(case):
    sym = case["mode"] == "group_sym"
    return ActQuantizer(bits=4, group_size=GROUP if sym else -1, sym=sym, use_hadamard=case["hadamard"], packed_output=True)


def _linear(g, case):
    k, n, group = case["k"], case["n"], GROUP if case["mode"] == "group_sym" else -1
    lin = LinearFLH(k, n, bias=case["bias"], dtype=torch.float16, device="cuda", group_size=group)
    lin.w_packed.copy_(torch.randint(0, 256, lin.w_packed.shape, dtype=torch.uint8, device="cuda", generator=g))
    lin.w_scale.copy_(torch.rand(lin.w_scale.shape, device="cuda", generator=g) * 0.015 + 0.005)
    if case["bias"]:
        lin.bias.copy_(torch.randn(n, device="cuda", generator=g))
    return lin.prepack_int8() if case["prepack"] else lin


def _config(case):
    shape = dict(LLAMA2_7B if case["shape"] == "7b" else LLAMA3_70B, n_layers=case["layers"])
    return DecoderConfig(**shape, vocab=VOCAB, act_mode=case["mode"])


def prepare(case, seed):
    g = _gen(seed)
    if case["kind"] == "quant":
        return dict(kind="quant", quant=_quantizer(case), x=_activations(g, case["m"], case["k"], case["dtype"]))
    if case["kind"] == "linear":
        return dict(kind="linear", quant=_quantizer(case), lin=_linear(g, case),
                    x=_activations(g, case["m"], case["k"], case["dtype"]), out=getattr(torch, case["dtype"]))
    model = Decoder(_config(case), torch.device("cuda"), seed=seed)
    if case["prepack"]:
        model.prepack_int8()
    b, s, ctx = case["batch"], case["seq"], case["ctx"]
    cache = model.new_cache(b, ctx + s)
    ids = torch.randint(0, VOCAB, (b, s), device="cuda", generator=g)
    state = dict(kind="decoder", model=model, cache=cache, ids=ids, start=ctx, graph=None)
    if s == 1:
        for c in cache:                      # what an earlier prefill left there
            c[0][:, :, :ctx].normal_(generator=g)
            c[1][:, :, :ctx].normal_(generator=g)
        # a decode step is many short launches: record it once, replay it with new token ids
        state["tokens"] = ids.clone()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):
                model(state["tokens"], cache=cache, start=ctx)
        torch.cuda.current_stream().wait_stream(side)
        state["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(state["graph"], stream=side):
            state["logits"] = model(state["tokens"], cache=cache, start=ctx)
    return state


# ------------------------------------------------------------------------------------------------------------- one pass
def run(state):
    if state["kind"] == "quant":
        return [t for t in state["quant"](state["x"]) if t is not None]
    if state["kind"] == "linear":
        scale, zero, codes = state["quant"](state["x"])
        return state["lin"](codes, scale, zero, out_dtype=state["out"])
    if state["graph"] is not None:
        state["tokens"].copy_(state["ids"])
        state["graph"].replay()
        logits = state["logits"]
    else:
        logits = state["model"](state["ids"], cache=state["cache"], start=state["start"])
    return [logits] + [t for c in state["cache"] for t in c[:2]]


# ---------------------------------------------------------------------------------------- what a pass cannot do without
def _weight_bytes(case, k, n):
    prepacked = case["prepack"] and case["mode"] == "token_asym"
    return k * n * (1.0 if prepacked else 0.5) + 2 * n * (k // GROUP if case["mode"] == "group_sym" else 1)


def work(case):
    if case["kind"] == "quant":
        m, k = case["m"], case["k"]
        side = 2 * k // GROUP if case["mode"] == "group_sym" else 4
        return {"bytes": m * (2 * k + k // 2 + side), "flops": m * k * 3}
    if case["kind"] == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * m * (k + n) + _weight_bytes(case, k, n), "flops": 2 * m * k * n}
    c = _config(case)
    b, s, ctx, hd = case["batch"], case["seq"], case["ctx"], c.hidden // c.n_heads
    rows, kv = b * s, c.n_kv_heads * hd
    shapes = ((c.hidden, c.hidden + 2 * kv), (c.hidden, c.hidden), (c.hidden, 2 * c.ffn), (c.ffn, c.hidden))
    keys = ctx + (s + 1) / 2                                                       # seen by an average query
    flops = sum(2.0 * rows * k * n for k, n in shapes) + 4.0 * rows * c.hidden * keys
    nbytes = sum(_weight_bytes(case, k, n) for k, n in shapes) + 2 * 2.0 * b * kv * (ctx + s)
    head = c.hidden * VOCAB
    return {"bytes": c.n_layers * nbytes + 2.0 * head + 2.0 * rows * c.hidden + 2.0 * b * VOCAB,
            "flops": c.n_layers * flops + 2.0 * b * head}


def tolerance(case):
    """Four times what was seen between the path and itself with the K-groups summed in reverse order and the transform in
    the sequential order (12 listed and 24 drawn cases on a B200)."""
    online = case.get("hadamard") and case["mode"] == "token_asym"
    if case["kind"] == "quant":
        # the online transform may be summed in any order: 5e-7 of the bytes were seen to differ, and a narrow call may hold one
        # such byte; everything else is fixed to the last bit
        return {"rel": 1e-4, "max": 1e-3, "differ": 1e-5 + 8.0 / (case["m"] * case["k"])} if online else "exact"
    if case["kind"] == "linear":
        if online:      # a code that moves by one step moves its row of the output by up to 8 steps of about 1000
            return {"rel": 1e-3, "max": 5e-2}
        # whole-number sums and one binary32 chain: 1.4e-5 in norm from last-bit roundings of the result, one of them at most a value
        return {"rel": 5e-5, "max": 2e-3} if case["dtype"] == "float16" else {"rel": 4e-4, "max": 1.6e-2}
    # codes of the second linear onward follow last bits of the one before, and a code moves by whole steps: 0.009 in norm and
    # 0.22 at worst in the caches of a second layer
    return {"rel": 3e-2, "max": 9e-1}
