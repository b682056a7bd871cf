"""The work that users of this framework have it do, as cases that can be timed.

A case is a dict of plain values. ``kind`` says which public entry point one pass goes through:

``linear``
    ``QCudaLinear.forward`` on activations that are on the device: a GGUF weight of format ``fmt`` and shape ``[n, k]``,
    ``m`` activation rows of type ``act``, with or without a bias.
``decode``
    One greedy token for each of ``batch`` sequences through ``QLlama.decode`` (the captured graph), ``context`` tokens being
    in the KV cache.
``prefill``
    ``QLlama.prefill`` of ``batch`` prompts of ``context`` tokens.

The decoder has the dimensions of the 7B configuration and ``layers`` of its 32 layers, with both ends (embedding, LM head).
Every layer is the same work; after more than two or three layers the rounding of activations to 8 bits has made two correct
results differ by more than a comparison can use.
"""
import math

import torch

from xn_b200.dtypes import GgmlDType
from xn_b200.llama import LlamaConfig, QLlama
from xn_b200.quantized import QCudaLinear, QCudaTensor

FORMATS = {"q4_0": GgmlDType.Q4_0, "q4_1": GgmlDType.Q4_1, "q5_0": GgmlDType.Q5_0, "q5_1": GgmlDType.Q5_1, "q8_0": GgmlDType.Q8_0,
           "q2_k": GgmlDType.Q2K, "q3_k": GgmlDType.Q3K, "q4_k": GgmlDType.Q4K, "q5_k": GgmlDType.Q5K, "q6_k": GgmlDType.Q6K}
ACTS = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
# where the blocks of the formats without a device quantizer hold their f16 scales, and the scales' magnitudes
F16_FIELDS = {"q4_1": ((0, 0.02), (2, 0.08)), "q5_0": ((0, 0.01),), "q5_1": ((0, 0.01), (2, 0.08)), "q2_k": ((80, 0.01), (82, 0.01)),
              "q3_k": ((108, 0.01),), "q5_k": ((0, 0.005), (2, 0.005))}


def _linear(name, fmt, n, k, m, act="f32", bias=False):
    return {"name": name, "kind": "linear", "fmt": fmt, "n": n, "k": k, "m": m, "act": act, "bias": bias}


def _model(name, kind, batch, context, max_seq, layers=2, fmt="q4_k"):
    return {"name": name, "kind": kind, "batch": batch, "context": context, "max_seq": max_seq, "layers": layers, "fmt": fmt}


def listed():
    return [
        # one token at a time, called layer by layer from a program of the user's: launch and host latency count
        _linear("q4_0_4096_row1", "q4_0", 4096, 4096, 1),              # the smallest projection
        _linear("q4_k_ffn_row1", "q4_k", 14336, 4096, 1),              # an MLP up projection
        _linear("q6_k_head_row1", "q6_k", 128256, 4096, 1),            # an LM head with a large vocabulary
        # a few sequences, or a draft of tokens to verify, at once
        _linear("q5_k_4096_rows7", "q5_k", 4096, 4096, 7),             # a format that is held as the file's blocks
        _linear("q4_k_down_rows16_bf16", "q4_k", 4096, 14336, 16, "bf16"),  # an MLP down projection in a bf16 model
        _linear("q8_0_rows45_f16_bias", "q8_0", 11008, 4096, 45, "f16", True),  # a ragged batch, f16 model with biases
        _linear("q6_k_head_rows32", "q6_k", 128256, 4096, 32),         # logits of a batch of 32
        # prompts
        _linear("q8_0_rows512", "q8_0", 11008, 4096, 512),
        _linear("q4_k_gate_up_rows2000_bf16", "q4_k", 28672, 4096, 2000, "bf16"),  # a long ragged prompt through a fused gate / up projection
        # the decoder: what all of the above adds up to
        _model("decode_batch1", "decode", 1, 512, 1024),
        _model("decode_batch16", "decode", 16, 200, 512),
        _model("prefill_512", "prefill", 1, 512, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.random()
    if what < 0.12:
        return _draw_model(rng, "decode", rng.choice([1, 1, 2, 3, 4, 6, 8, 11, 16]), rng.randint(16, 480), 512)
    if what < 0.2:
        batch = rng.choice([1, 1, 2, 3])
        return _draw_model(rng, "prefill", batch, _log_int(rng, 40, 512 // batch), 1024)
    fmt = rng.choice(["q4_0", "q8_0", "q4_k", "q4_k", "q6_k"]) if rng.random() < 0.85 else rng.choice(sorted(F16_FIELDS))
    block = FORMATS[fmt].block_size
    most = 28672 * 4096 * 2000 if fmt not in F16_FIELDS else 4096 * 4096 * 24
    while True:
        n = _log_int(rng, 256, 32768)
        if rng.random() < 0.6:
            n = max(128, n // 128 * 128)
        step = 256 if block == 256 else 64
        k = max(1, _log_int(rng, 512, 14336) // step) * step
        m = 1 if rng.random() < 0.25 else _log_int(rng, 2, 2048)
        if n * k * m <= most:
            break
    case = _linear("", fmt, n, k, m, rng.choice(["f32", "f32", "f16", "bf16"]), rng.random() < 0.25)
    del case["name"]
    return case


def _draw_model(rng, kind, batch, context, max_seq):
    case = _model("", kind, batch, context, max_seq, rng.choice([1, 2, 2]), rng.choice(["q4_k", "q4_k", "q8_0", "q4_0"]))
    del case["name"]
    return case


def _blocks(fmt, n, k, gen):
    """Valid blocks of a format that has no device quantizer: random codes, scales from |N(0, 1)|."""
    dt = FORMATS[fmt]
    nb = n * k // dt.block_size
    out = torch.randint(0, 256, (nb, dt.type_size), dtype=torch.uint8, device="cuda", generator=gen)
    for at, scale in F16_FIELDS[fmt]:
        v = (torch.randn(nb, 1, device="cuda", generator=gen).abs() * scale).to(torch.float16)
        out[:, at:at + 2] = v.view(torch.uint8)
    return out.view(-1)


def _config(case):
    return LlamaConfig(n_layers=case["layers"], linear_dtype=FORMATS[case["fmt"]])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "linear":
        fmt, n, k = case["fmt"], case["n"], case["k"]
        if fmt in F16_FIELDS:
            weight = QCudaTensor.from_device_rows(FORMATS[fmt], _blocks(fmt, n, k, gen), n, k, 0, n)
        else:
            weight = QCudaTensor.from_dense(torch.randn(n, k, device="cuda", generator=gen) * 0.02, FORMATS[fmt])
        act = ACTS[case["act"]]
        bias = (torch.randn(n, device="cuda", generator=gen) * 0.1).to(act) if case["bias"] else None
        x = torch.randn(case["m"], k, device="cuda", generator=gen).to(act)
        return {"case": case, "layer": QCudaLinear.new(weight, bias), "x": x}
    cfg = _config(case)
    model = QLlama(cfg, torch.device("cuda:0"), batch=case["batch"], max_seq=case["max_seq"], seed=seed)
    prompt = torch.randint(0, cfg.vocab, (case["batch"], case["context"]), device="cuda", generator=gen)
    state = {"case": case, "model": model, "prompt": prompt}
    if case["kind"] == "decode":
        model.prefill(prompt)
        model.capture_decode()
        state["pos"], state["tokens"] = model.pos.clone(), torch.randint(0, cfg.vocab, (case["batch"],), device="cuda", generator=gen)
    return state


def run(state):
    kind = state["case"]["kind"]
    if kind == "linear":
        return state["layer"].forward(state["x"])
    model = state["model"]
    if kind == "prefill":
        logits = model.prefill(state["prompt"])
    else:
        model.pos.copy_(state["pos"])
        model.tokens.copy_(state["tokens"])
        model.decode(1)
        logits = model.last_logits
    return {"logits": logits, "cache": [(layer.k_cache, layer.v_cache) for layer in model.layers]}


def work(case):
    if case["kind"] == "linear":
        n, k, m = case["n"], case["k"], case["m"]
        size = ACTS[case["act"]].itemsize
        return {"bytes": n * FORMATS[case["fmt"]].row_bytes(k) + size * (m * k + m * n + (n if case["bias"] else 0)), "flops": 2 * m * n * k}
    c = _config(case)
    batch, context = case["batch"], case["context"]
    per_token = 2 * c.n_layers * c.d_model * ((c.n_heads + 2 * c.n_kv_heads) * c.head_dim + c.n_heads * c.head_dim + 3 * c.ffn)
    attn = 4 * c.n_layers * c.n_heads * c.head_dim          # per query and key
    cache = 4 * c.n_layers * c.n_kv_heads * c.head_dim      # bytes of one position's k and v in bf16
    if case["kind"] == "prefill":
        keys = context * (context + 1) // 2
        return {"bytes": c.weight_bytes_per_step() + batch * context * (cache + 2 * c.d_model) + 4 * batch * c.vocab,
                "flops": batch * (context * per_token + keys * attn + 2 * c.d_model * c.vocab)}
    return {"bytes": c.weight_bytes_per_step() + batch * ((context + 2) * cache + 2 * c.d_model + 4 * c.vocab),
            "flops": batch * (per_token + (context + 1) * attn + 2 * c.d_model * c.vocab)}


def tolerance(case):
    # Four times what was seen between the path and itself in 64 bits or with its sums in another order.
    if case["kind"] != "linear":
        # A difference in the last bit of a sum moves some of the next linear's 8-bit activation codes by one: 1.2 % of the logits'
        # norm after two layers, whatever made the difference, and no more than that after one where nothing differs.
        return {"rel": 3e-2, "max": 0.25}
    rows = case["m"]
    half_operands = case["fmt"] not in F16_FIELDS and rows > (16 if case["fmt"] == "q6_k" else 64)   # 3e-4 to 8e-4 on weights and rows rounded to f16
    if case["act"] == "bf16":    # the result is rounded to 8 bits, once or (with a bias) twice: 1.6e-3
        return {"rel": 7e-3, "max": 3e-2}
    if half_operands:
        return {"rel": 3e-3, "max": 1.5e-2}
    if case["act"] == "f16":     # the result is rounded to 11 bits, once or (with a bias) twice: 3.6e-4
        return {"rel": 1.5e-3, "max": 4e-3}
    return {"rel": 1e-6, "max": 1e-5}   # exact integer sums in each block, blocks added in f32: 9e-8
