"""The work that a user of this library has it do, as cases that can be timed and whose outputs can be compared.

Four kinds, each through the public entry point that a program calls:

* ``matmul``     - ``QMatMul.forward``: one projection of a quantized model, from one decoded token to a long prompt, over the
  Llama-3-8B projection shapes of the benchmark and generic ones around them;
* ``dequantize`` - ``QTensor.dequantize``: a matrix expanded on its device (dense fallback of a model, weight inspection);
* ``moe``        - ``FusedMoeGGUF.forward``: the mixture-of-experts block of a layer, decode and prompt;
* ``decoder``    - ``LlamaShapedDecoder``: a prompt and the decode steps after it, with given tokens.

Weights are GGUF blocks made on the device: uniformly random codes and sub-scales, super-scales such that the weights have the
spread of a trained projection.  Activations are normal with a spread between channels.
"""
from __future__ import annotations

import math

import torch

from candle_b200.decoder import DecoderConfig, LlamaShapedDecoder
from candle_b200.fused_moe import FusedMoeGGUF
from candle_b200.quantized import GgmlDType, QMatMul, QTensor

_DEVICE = "cuda:0"
_ELEM = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}

# f16 fields of a block: (byte offset, typical magnitude)
_SCALES = {
    "Q4_0": [(0, 0.06 / 8)], "Q4_1": [(0, 0.12 / 15), (2, -0.06)], "Q5_0": [(0, 0.06 / 16)], "Q5_1": [(0, 0.12 / 31), (2, -0.06)],
    "Q8_0": [(0, 0.06 / 127)], "Q2K": [(80, 0.12 / (15 * 3)), (82, 0.06 / 15)], "Q3K": [(108, 0.06 / (32 * 4))],
    "Q4K": [(0, 0.12 / (63 * 15)), (2, 0.06 / 63)], "Q5K": [(0, 0.12 / (63 * 31)), (2, 0.06 / 63)], "Q6K": [(208, 0.06 / (127 * 32))],
}


def listed():
    return [
        # --- one projection, decode: a token of one sequence, the head of one sequence, a batch of eight sequences
        # attention output projection of an 8B model, one token: the smallest call, where launches and host time count
        dict(name="decode_q4k_4096x4096_b1", kind="matmul", dtype="Q4K", k=4096, n=4096, rows=1, elem="f32"),
        # vocabulary head of the same model, one token: the longest stream of weights
        dict(name="decode_q6k_head_b1", kind="matmul", dtype="Q6K", k=4096, n=128256, rows=1, elem="f32"),
        # gate / up projection for eight sequences decoded together, 16-bit activations
        dict(name="decode_q4k_4096x14336_b8", kind="matmul", dtype="Q4K", k=4096, n=14336, rows=8, elem="bf16"),
        # --- one projection, prompt
        # gate / up projection of a long prompt in the usual 16-bit type
        dict(name="prompt_q4k_4096x14336_m2048", kind="matmul", dtype="Q4K", k=4096, n=14336, rows=2048, elem="bf16"),
        # down projection (Q6_K in the usual mixes) of an ordinary prompt, f32 activations
        dict(name="prompt_q6k_14336x4096_m512", kind="matmul", dtype="Q6K", k=14336, n=4096, rows=512, elem="f32"),
        # 8-bit model, a prompt whose length fits no tile
        dict(name="prompt_q8_0_4096x4096_m333", kind="matmul", dtype="Q8_0", k=4096, n=4096, rows=333, elem="f16"),
        # a 5-bit model's prompt: the formats between the common ones
        dict(name="prompt_q5k_4096x14336_m512", kind="matmul", dtype="Q5K", k=4096, n=14336, rows=512, elem="f32"),
        # --- a matrix expanded to f16 (what a model with the dense fallback does at load)
        dict(name="dequantize_q4k_14336x4096_f16", kind="dequantize", dtype="Q4K", k=4096, n=14336, elem="f16"),
        # --- the expert block of a Qwen3-30B-A3B-shaped layer: eight decoded tokens, and a prompt of 1024
        dict(name="moe_q4k_decode_t8", kind="moe", dtype="Q4K", hidden=2048, ffn=768, experts=128, topk=8, tokens=8, prefill=False),
        dict(name="moe_q4k_prompt_t1024", kind="moe", dtype="Q4K", hidden=2048, ffn=768, experts=128, topk=8, tokens=1024, prefill=True),
        # --- four layers of a Llama-3-8B-shaped decoder with its head: a chat turn (short prompt, then decode steps replayed
        # from a graph), and the prompt phase of two longer sequences
        dict(name="decoder_b1_p64_s32", kind="decoder", layers=4, d_model=4096, heads=32, kv_heads=8, ffn=14336, vocab=128256,
             batch=1, prompt=64, steps=32),
        dict(name="decoder_b2_p512_s0", kind="decoder", layers=4, d_model=4096, heads=32, kv_heads=8, ffn=14336, vocab=128256,
             batch=2, prompt=512, steps=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


_WIDE = ("Q4_1", "Q5_0", "Q5_1", "Q2K", "Q3K", "Q5K")


def draw(rng):
    kind = rng.choices(["matmul", "dequantize", "moe", "decoder"], [10, 1, 2, 2])[0]
    if kind == "matmul":
        dtype = rng.choices(["Q4K", "Q6K", "Q8_0", "Q4_0", "Q5K", "Q4_1", "Q5_0", "Q5_1", "Q2K", "Q3K"], [8, 6, 4, 3, 3, 1, 1, 1, 1, 1])[0]
        k = 256 * _log_int(rng, 4, 56)
        if rng.random() < 0.4:      # decode: up to eight sequences, now and then a head-sized matrix
            rows, n = rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]), _log_int(rng, 512, 48000)
            n = min(n, 4096 * 128256 // k)
        else:                       # several tokens of a few sequences up to long prompts
            rows, n = _log_int(rng, 9, 2048), _log_int(rng, 512, 14336)
            cap = (512 if dtype in _WIDE else 2048) * 4096 * 14336
            rows = max(9, min(rows, cap // (k * n)))
        if rng.random() < 0.7:
            n = max(512, n // 64 * 64)
        return dict(kind=kind, dtype=dtype, k=k, n=n, rows=rows, elem=rng.choice(["f32", "bf16", "f16"]))
    if kind == "dequantize":
        dtype = rng.choice(sorted(_SCALES))
        return dict(kind=kind, dtype=dtype, k=256 * _log_int(rng, 4, 56), n=_log_int(rng, 512, 4096), elem=rng.choice(["f32", "f16", "bf16"]))
    if kind == "moe":
        tokens = _log_int(rng, 1, 1024)
        return dict(kind=kind, dtype=rng.choice(["Q4K", "Q4K", "Q6K", "Q8_0"]) if tokens <= 64 else rng.choice(["Q4K", "Q6K"]),
                    hidden=256 * _log_int(rng, 4, 8), ffn=256 * rng.choice([2, 3]), experts=rng.choice([16, 32, 64, 128]),
                    topk=rng.choice([2, 4, 8]), tokens=tokens, prefill=tokens > 64)
    heads = rng.choice([8, 16, 32])
    batch = rng.choice([1, 1, 2, 4])
    return dict(kind=kind, layers=rng.choice([2, 3, 4]), d_model=heads * 128, heads=heads, kv_heads=8, ffn=2048 * rng.choice([1, 2, 4, 7]),
                vocab=rng.choice([32000, 49152, 65536]), batch=batch, prompt=max(1, _log_int(rng, 16, 1024) // batch),
                steps=rng.choice([0, 0, 4, 16, 32]))


def _blocks(dtype: str, n: int, k: int, gen) -> torch.Tensor:
    t = GgmlDType[dtype]
    count, size = n * (k // t.block_size()), t.type_size()
    b = torch.randint(0, 256, (count, size), dtype=torch.uint8, device=_DEVICE, generator=gen)
    for off, mag in _SCALES[dtype]:
        d = (torch.rand(count, device=_DEVICE, generator=gen) * 0.5 + 0.75) * mag
        b[:, off:off + 2] = d.to(torch.float16).view(torch.uint8).view(count, 2)
    return b.view(-1)


def _qtensor(dtype: str, shape, gen) -> QTensor:
    return QTensor.from_device_blocks(_blocks(dtype, math.prod(shape[:-1]), shape[-1], gen), GgmlDType[dtype], shape)


def _activations(rows: int, k: int, elem: str, gen) -> torch.Tensor:
    spread = torch.exp(0.5 * torch.randn(k, device=_DEVICE, generator=gen))
    return (torch.randn((rows, k), device=_DEVICE, generator=gen) * spread).to(_ELEM[elem])


def prepare(case, seed):
    gen = torch.Generator(device=_DEVICE)
    gen.manual_seed(seed)
    kind = case["kind"]
    if kind == "matmul":
        w = QMatMul.from_qtensor(_qtensor(case["dtype"], (case["n"], case["k"]), gen))
        return kind, w, _activations(case["rows"], case["k"], case["elem"], gen)
    if kind == "dequantize":
        return kind, _qtensor(case["dtype"], (case["n"], case["k"]), gen), _ELEM[case["elem"]]
    if kind == "moe":
        e, f, d = case["experts"], case["ffn"], case["hidden"]
        router = torch.randn((e, d), device=_DEVICE, generator=gen) * 0.05
        block = FusedMoeGGUF(router, _qtensor(case["dtype"], (e, f, d), gen), _qtensor(case["dtype"], (e, f, d), gen),
                             _qtensor(case["dtype"], (e, d, f), gen), case["topk"])
        x = _activations(case["tokens"], d, "f32", gen)
        return kind, block, x.view(1, case["tokens"], d), case["prefill"]
    p, s = case["prompt"], case["steps"]
    cfg = DecoderConfig(layers=case["layers"], d_model=case["d_model"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn=case["ffn"],
                        vocab=case["vocab"], max_pos=-(-(p + s + 3) // 128) * 128)      # + 3: the steps run while a graph is recorded
    model = LlamaShapedDecoder(cfg, _DEVICE, batch=case["batch"], seed=seed)
    tokens = torch.randint(0, cfg.vocab, (case["batch"], p + s), device=_DEVICE, generator=gen)
    if s:
        model.capture_decode_step()
    return kind, model, tokens[:, :p].contiguous(), [tokens[:, p + i].contiguous() for i in range(s)]


def run(state):
    kind = state[0]
    if kind == "matmul":
        return state[1].forward(state[2])
    if kind == "dequantize":
        return state[1].dequantize(state[2])
    if kind == "moe":
        return state[1].forward(state[2], state[3])
    _, model, prompt, steps = state
    model.reset()
    tokens = [model.forward(prompt)]
    logits = [model.last_logits]
    if steps:
        logits = [model.last_logits.clone()]
        for tok in steps:       # given tokens, so that one near-tie does not change everything after it
            tokens.append(model.decode_step(tok).clone())
            logits.append(model.last_logits.clone())
    return {"tokens": torch.stack(tokens, dim=1), "logits": torch.stack(logits, dim=1)}


def _row_bytes(dtype: str, k: int) -> int:
    t = GgmlDType[dtype]
    return k // t.block_size() * t.type_size()


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        es = _ELEM[case["elem"]].itemsize
        k, n, rows = case["k"], case["n"], case["rows"]
        return {"bytes": n * _row_bytes(case["dtype"], k) + rows * (k + n) * es, "flops": 2 * rows * n * k}
    if kind == "dequantize":
        return {"bytes": case["n"] * (_row_bytes(case["dtype"], case["k"]) + case["k"] * _ELEM[case["elem"]].itemsize), "flops": case["n"] * case["k"]}
    if kind == "moe":
        e, f, d, t, top = case["experts"], case["ffn"], case["hidden"], case["tokens"], case["topk"]
        used = e * (1.0 - (1.0 - top / e) ** t)         # experts that see a token
        expert = 2 * f * _row_bytes(case["dtype"], d) + d * _row_bytes(case["dtype"], f)
        return {"bytes": int(used * expert) + e * d * 4 + 2 * t * d * 4, "flops": 2 * t * (top * 3 * f * d + e * d)}
    d, q, kv, f = case["d_model"], case["heads"] * 128, case["kv_heads"] * 128, case["ffn"]
    layer = (q + kv) * _row_bytes("Q4K", d) + kv * _row_bytes("Q6K", d) + d * _row_bytes("Q4K", q) + 2 * f * _row_bytes("Q4K", d) + d * _row_bytes("Q6K", f)
    weights = case["layers"] * layer + case["vocab"] * _row_bytes("Q6K", d)
    params = case["layers"] * ((q + 2 * kv) * d + d * q + 3 * f * d)
    b, p, s = case["batch"], case["prompt"], case["steps"]
    keys = p * (p + 1) // 2 + sum(range(p + 1, p + s + 1))          # (query, key) pairs of one sequence and head
    step_kv = sum(range(p + 1, p + s + 1)) * 2 * kv * 4             # a decode step reads its whole context
    return {"bytes": (1 + s) * weights + case["layers"] * b * (step_kv + 2 * (p + s) * kv * 4) + b * (1 + s) * case["vocab"] * 4,
            "flops": 2 * b * (p + s) * params + 2 * b * (1 + s) * case["vocab"] * d + case["layers"] * b * keys * q * 4}


def tolerance(case):
    kind = case["kind"]
    if kind == "dequantize":
        return "exact"              # one formula per element, rounded once
    if kind == "matmul":
        # exact integer products, f32 sums.  With the 256-element blocks of K in another order: 6e-8 .. 5e-7 (f32 results),
        # up to 1.1e-5 (f16) and 3.4e-5 (bf16), where a sum near a rounding boundary takes the neighbouring value
        return {"rel": {"f32": 2e-6, "f16": 5e-5, "bf16": 1.5e-4}[case["elem"]]}
    if kind == "moe":
        # another order of the f32 sums moves a few of the 8-bit (prompt: also 16-bit) roundings between the matmuls; inputs moved
        # by one f32 rounding: 5e-7 (decode, no rounding moved - a single one is worth about 2e-5), 4.6e-4 (prompt)
        return {"rel": 2e-3 if case["prefill"] else 1e-4}
    # The same through several layers of activation quantization, which is a step function: embeddings moved by one f32 rounding
    # give logits 1.3e-2 .. 4.2e-2 away, and the arg-max of 32000 .. 128256 logits then changes for up to 9 % of the tokens
    # (the second term leaves room for one token where few come back).
    count = case["batch"] * (1 + case["steps"])
    return {"rel": 0.16, "differ": min(1.0, 0.36 + 1.0 / count)}
