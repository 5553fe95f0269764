"""Workloads whose speed is watched: what a user of the compressed linears has the package do.

Five kinds of work, all through the public entry points:

  linear    one ``CobaltSparseLinear`` call on ``M`` tokens: the module that replaces an ``nn.Linear``.  Up to 16 tokens
            is a decode step (bandwidth-bound), more is a prompt or a chunk of one (tensor-bound).  ``bias`` and
            ``scale2`` (the fp16 scale per input column of the reference's dual-scaled matrices) are the module's options.
  block     the seven projections of ``layers`` decoder blocks on ``M`` tokens: q|k|v and gate|up as fused launches, o and
            down as modules, called eagerly as a patched model does.
  generate  ``CobaltDecoder.generate``: a prompt, then ``new`` tokens through the captured decode step, teacher-forced
            so that two runs can be compared step by step.
  prefill   ``CobaltDecoder.prefill``: the prompt alone (time to first token, scoring).
  convert   ``CobaltSparseLinear.from_linear`` (keep mask, rounding, packing) followed by ``unpack`` and ``dequantize``: what it
            costs to bring a checkpoint in and to look at what became of it.

Shapes are those of a Mistral-7B block and a Gemma-3-27B block; models have few layers, because every layer does the same
work.  All data is synthetic and seeded: weights N(0, 0.02), activation norms |N(0, 1)| + 0.1, activations N(0, 1).
"""
import math

import torch

from cobalt_b200 import CobaltSparseLinear
from cobalt_b200.compress import quantize_survivors
from cobalt_b200.decoder import PROJ, CobaltDecoder, compress_head, proj_shapes
from cobalt_b200.linear import FusedProjections

DEV = "cuda"
GROUP = 128
VOCAB = 32000


# ----------------------------------------------------------------------------- the cases
def _linear(name, K, N, M, bits, sparsity, bias=False, scale2=False):
    return {"name": name, "op": "linear", "K": K, "N": N, "M": M, "bits": bits, "sparsity": sparsity, "bias": bias,
            "scale2": scale2}


def _model(name, op, family, hidden, heads, kv, inter, layers, batch, prompt, new, bits, sparsity, head_bits, window=0):
    return {"name": name, "op": op, "family": family, "hidden": hidden, "heads": heads, "kv": kv, "inter": inter,
            "layers": layers, "batch": batch, "prompt": prompt, "new": new, "bits": bits, "sparsity": sparsity,
            "head_bits": head_bits, "window": window}


def listed():
    return [
        # the smallest matrix of a 7B block in one decode step of an eagerly run model: latency of one call
        _linear("linear_kv_1tok", 1024, 4096, 1, 4, 0.5),
        # the single-linear configuration: a square projection, 3-bit, 70 % sparse, one token
        _linear("linear_q_1tok", 4096, 4096, 1, 3, 0.7),
        # a dual-scaled matrix with bias, a few sequences decoded together
        _linear("linear_q_5tok_scaled", 4096, 4096, 5, 4, 0.5, bias=True, scale2=True),
        # the largest matrix of a 27B block at the batch size served there
        _linear("linear_gate27b_8tok", 21504, 5376, 8, 3, 0.6),
        # a short, ragged prompt through a square projection
        _linear("linear_q_100tok", 4096, 4096, 100, 2, 0.5),
        # a full prompt through the widest contraction of a 7B block
        _linear("linear_down_2048tok", 4096, 14336, 2048, 3, 0.7),
        # all projections of 7B blocks in a decode step, one sequence and a full batch
        {"name": "block_7b_1tok", "op": "block", "hidden": 4096, "kv_width": 1024, "inter": 14336, "layers": 2, "M": 1, "bits": 4,
         "sparsity": 0.5},
        {"name": "block_7b_16tok", "op": "block", "hidden": 4096, "kv_width": 1024, "inter": 14336, "layers": 2, "M": 16, "bits": 4,
         "sparsity": 0.5},
        # a chat turn: a prompt of 1024 tokens and 64 new ones, 7B blocks, dense head
        _model("generate_7b", "generate", "llama", 4096, 32, 8, 14336, 2, 1, 1024, 64, 4, 0.5, 0),
        # eight sequences served together, 27B blocks (sliding and full attention), compressed head
        _model("generate_27b_8seq", "generate", "gemma", 5376, 32, 16, 21504, 2, 8, 200, 48, 3, 0.6, 4, 1024),
        # time to first token of a 2048-token prompt, 7B blocks
        _model("prefill_7b", "prefill", "llama", 4096, 32, 8, 14336, 2, 1, 2048, 0, 4, 0.5, 0),
        # a projection of a checkpoint compressed and checked
        {"name": "convert_q", "op": "convert", "K": 4096, "N": 4096, "bits": 3, "sparsity": 0.7},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of ``step`` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(max(int(round(v / step)) * step, lo), hi)


def draw(rng):
    op = rng.choice(["linear", "linear", "linear", "prompt", "prompt", "block", "generate", "prefill", "convert"])
    bits = rng.choice([2, 3, 4])
    sparsity = round(rng.uniform(0.3, 0.8), 2)
    if op in ("linear", "prompt"):
        K, N = _log_int(rng, 64, 21504), _log_int(rng, 512, 21504, GROUP)           # any row count, whole groups
        while K * N > 21504 * 5376:
            K = max(64, K // 2)
        M = rng.randint(1, 16)
        if op == "prompt":
            M = _log_int(rng, 17, 2048)
            while M * K * N > 2048 * 4096 * 14336:
                M = max(17, M // 2)
        return {"op": "linear", "K": K, "N": N, "M": M, "bits": bits, "sparsity": sparsity, "bias": rng.random() < 0.25,
                "scale2": rng.random() < 0.2}
    if op == "block":
        hidden = _log_int(rng, 512, 5376, GROUP)
        return {"op": "block", "hidden": hidden, "kv_width": rng.choice([1, 2, 4]) * GROUP * max(1, hidden // 2048),
                "inter": _log_int(rng, hidden, min(4 * hidden, 14336), GROUP), "layers": rng.randint(1, 2), "M": rng.randint(1, 16),
                "bits": bits, "sparsity": sparsity}
    if op == "convert":
        return {"op": "convert", "K": _log_int(rng, 256, 4096), "N": _log_int(rng, 512, 4096, GROUP), "bits": bits,
                "sparsity": sparsity}
    kv = rng.choice([2, 4, 8])
    heads = kv * rng.choice([1, 2, 4])
    hidden = _log_int(rng, 512, 4096, 256)
    family = rng.choice(["llama", "gemma"])
    case = {"op": op, "family": family, "hidden": hidden, "heads": heads, "kv": kv,
            "inter": _log_int(rng, hidden, 3 * hidden, GROUP), "layers": 2, "batch": 1, "prompt": _log_int(rng, 17, 2048), "new": 0,
            "bits": bits, "sparsity": sparsity, "head_bits": rng.choice([0, 4]), "window": rng.choice([256, 1024]) if family == "gemma" else 0}
    if op == "generate":
        case["batch"] = rng.choice([1, 1, 2, 4, 8])
        case["prompt"] = _log_int(rng, 17, 1024 if case["batch"] == 1 else 200)
        case["new"] = rng.randint(8, 48)
    return case


# ----------------------------------------------------------------------------- preparation
def _gen(seed, salt=0):
    return torch.Generator(device=DEV).manual_seed(1_000_003 * (seed % 1_000_003) + salt)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _module(g, K, N, bits, sparsity, bias=False, scale2=False):
    """One compressed matrix.  The keep mask follows the column-balanced score |W| * norm^(1/2) with a global threshold that is
    taken from a sample of the scores (the exact order statistic takes longer than everything else here)."""
    W = (_randn(g, K, N) * 0.02).half().float()
    norm = _randn(g, N).abs() + 0.1
    score = W.abs() * norm.sqrt()
    sample = score.reshape(-1)[:: max(1, K * N // 500_000)]
    keep = score > torch.kthvalue(sample, max(1, int(sample.numel() * sparsity))).values
    del score
    q, scale, zero = quantize_survivors(W, keep, bits)
    b = (_randn(g, K) * 0.1).to(torch.bfloat16) if bias else None
    s2 = torch.exp(_randn(g, N) * 0.25).half() if scale2 else None
    return CobaltSparseLinear(q, scale, zero, keep, s2, b, {"nbits": bits})


def _config(case):
    cfg = dict(model_type="mistral", hidden_size=case["hidden"], num_hidden_layers=case["layers"],
               num_attention_heads=case["heads"], num_key_value_heads=case["kv"], head_dim=128,
               intermediate_size=case["inter"], vocab_size=VOCAB, rms_norm_eps=1e-5, rope_theta=1e6, sliding_window=None)
    if case["family"] == "gemma":
        cfg.update(model_type="gemma3_text", rms_norm_eps=1e-6, rope_local_base_freq=1e4, sliding_window=case["window"],
                   sliding_window_pattern=2, query_pre_attn_scalar=128,
                   rope_scaling={"rope_type": "linear", "factor": 8.0})
    return cfg


def _dense(g, cfg):
    H, V, gemma = cfg["hidden_size"], cfg["vocab_size"], cfg["model_type"] == "gemma3_text"

    def norm(n):
        w = _randn(g, n) * 0.05
        return (w if gemma else 1.0 + w).to(torch.bfloat16)

    # a head that follows the embedding (Gemma: the same matrix; else the same rows, one token on) gives the peaked
    # distributions of a trained model, whose greedy tokens do not hang on the last bit of a sum
    E = _randn(g, V, H) * (0.02 if gemma else 1.0)
    P = {"model.embed_tokens.weight": E.to(torch.bfloat16), "model.norm.weight": norm(H)}
    names = ["input_layernorm", "post_attention_layernorm"]
    if gemma:
        names += ["pre_feedforward_layernorm", "post_feedforward_layernorm"]
    else:
        P["lm_head.weight"] = (E.roll(1, 0) * 0.02).to(torch.bfloat16)
    for i in range(cfg["num_hidden_layers"]):
        for nm in names:
            P[f"model.layers.{i}.{nm}.weight"] = norm(H)
        if gemma:
            P[f"model.layers.{i}.self_attn.q_norm.weight"] = norm(cfg["head_dim"])
            P[f"model.layers.{i}.self_attn.k_norm.weight"] = norm(cfg["head_dim"])
    return P


def _decoder(case, seed):
    g = _gen(seed, 2)
    cfg = _config(case)
    lin = {(i, name): _module(g, K, N, case["bits"], case["sparsity"])
           for i in range(case["layers"]) for name, (K, N) in ((n, proj_shapes(cfg)[n]) for n in PROJ)}
    dense = _dense(g, cfg)
    head = compress_head(dense, cfg, case["head_bits"]) if case["head_bits"] else None
    return CobaltDecoder(cfg, lin, dense, case["prompt"] + case["new"], torch.device(DEV), batch=case["batch"], head=head)


def prepare(case, seed):
    state = dict(case)
    g = _gen(seed, 1)
    if case["op"] == "linear":
        state["module"] = _module(g, case["K"], case["N"], case["bits"], case["sparsity"], case["bias"], case["scale2"])
        state["x"] = _randn(g, case["M"], case["N"]).to(torch.bfloat16)
    elif case["op"] == "block":
        H, kv, inter = case["hidden"], case["kv_width"], case["inter"]
        state["layers_"] = []
        for _ in range(case["layers"]):
            m = [_module(g, K, N, case["bits"], case["sparsity"])
                 for K, N in ((H, H), (kv, H), (kv, H), (H, H), (inter, H), (inter, H), (H, inter))]
            state["layers_"].append((FusedProjections(m[:3]), m[3], FusedProjections(m[4:6]), m[6]))
        state["x"] = [_randn(g, case["M"], n).to(torch.bfloat16) for n in (H, H, H, inter)]
    elif case["op"] == "convert":
        linear = torch.nn.Linear(case["N"], case["K"], bias=False, device=DEV, dtype=torch.bfloat16)
        linear.weight.data.copy_(_randn(g, case["K"], case["N"]) * 0.02)
        state["linear"] = linear
        state["norms"] = _randn(g, case["N"]).abs() + 0.1
    else:
        dec = state["decoder"] = _decoder(case, seed)
        shape = (case["prompt"],) if case["batch"] == 1 else (case["batch"], case["prompt"])
        state["prompt"] = torch.randint(0, VOCAB, shape, generator=g, device=DEV)
        if case["op"] == "generate":
            shape = (case["new"],) if case["batch"] == 1 else (case["new"], case["batch"])
            state["teacher"] = torch.randint(0, VOCAB, shape, generator=g, device=DEV)
            dec.generate(state["prompt"], 2, teacher=state["teacher"])              # a serving process captures its step once
    return state


# ----------------------------------------------------------------------------- one pass
@torch.no_grad()
def run(state):
    op = state["op"]
    if op == "linear":
        return state["module"](state["x"])
    if op == "block":
        x_qkv, x_o, x_up, x_down = state["x"]
        outs = []
        for qkv, o, gate_up, down in state["layers_"]:
            outs += qkv(x_qkv)
            outs.append(o(x_o))
            outs += gate_up(x_up)
            outs.append(down(x_down))
        return outs
    if op == "convert":
        module = CobaltSparseLinear.from_linear(state["linear"], state["norms"], bits=state["bits"], sparsity=state["sparsity"])
        codes, keep = module.unpack()
        return {"codes": codes, "keep": keep, "dense": module.dequantize()}
    dec = state["decoder"]
    if op == "prefill":
        logits = dec.prefill(state["prompt"])
        return {"logits": logits, "k": dec.k_cache, "v": dec.v_cache}
    tokens, logits = dec.generate(state["prompt"], state["new"], teacher=state["teacher"])
    return {"tokens": tokens, "logits": logits, "k": dec.k_cache, "v": dec.v_cache}


# ----------------------------------------------------------------------------- what a pass cannot do without
def _matrix_bytes(K, N, bits, sparsity):
    return K * N / 8 + K * N * (1.0 - sparsity) * bits / 8 + K * (N // GROUP) * 4


def _add(total, nbytes, flops):
    total["bytes"] += nbytes
    total["flops"] += flops


def _forward_work(case, total, tokens, first, sequences):
    """One forward of ``tokens`` new tokens per sequence that sit at positions ``first`` ..., for ``sequences`` sequences at once.
    Contractions are counted dense: an unstructured mask leaves the tensor cores no less to do."""
    cfg = _config(case)
    H, D, heads, kv = case["hidden"], 128, case["heads"], case["kv"]
    rows = tokens * sequences
    seen = sum(range(first + 1, first + tokens + 1)) * sequences                      # (token, cache slot) pairs, full attention
    near = seen
    if case["window"]:
        near = sum(min(p, case["window"]) for p in range(first + 1, first + tokens + 1)) * sequences
    for i in range(case["layers"]):
        for K, N in proj_shapes(cfg).values():
            _add(total, _matrix_bytes(K, N, case["bits"], case["sparsity"]), 2.0 * rows * K * N)
        sliding = case["window"] and (i + 1) % 2
        pairs, slots = (near, min(first + tokens, case["window"] + tokens)) if sliding else (seen, first + tokens)
        _add(total, 2 * kv * D * 2.0 * slots * sequences, 4.0 * heads * D * pairs)
    if case["head_bits"]:
        _add(total, _matrix_bytes(VOCAB, H, case["head_bits"], 0.0), 2.0 * rows * VOCAB * H)
    else:
        _add(total, 2.0 * VOCAB * H, 2.0 * rows * VOCAB * H)
    _add(total, rows * (H + VOCAB) * 2.0, 0.0)                                       # embedding rows in, logits out


def work(case):
    total = {"bytes": 0.0, "flops": 0.0}
    op = case["op"]
    if op == "linear":
        K, N, M = case["K"], case["N"], case["M"]
        options = 2 * K * case["bias"] + 2 * N * case["scale2"]
        _add(total, _matrix_bytes(K, N, case["bits"], case["sparsity"]) + 2.0 * M * (N + K) + options, 2.0 * M * K * N)
    elif op == "block":
        H, kv, inter, M = case["hidden"], case["kv_width"], case["inter"], case["M"]
        for K, N in ((H, H), (kv, H), (kv, H), (H, H), (inter, H), (inter, H), (H, inter)):
            _add(total, case["layers"] * (_matrix_bytes(K, N, case["bits"], case["sparsity"]) + 2.0 * M * K), case["layers"] * 2.0 * M * K * N)
        _add(total, 2.0 * M * (3 * H + inter), 0.0)
    elif op == "convert":
        K, N = case["K"], case["N"]
        # dense weight and norms in; packed image out, read back twice; codes, mask and dense weight out
        _add(total, 2.0 * K * N + 4.0 * N + 3 * _matrix_bytes(K, N, case["bits"], case["sparsity"]) + 4.0 * K * N, 0.0)
    else:
        for _ in range(case["batch"]):
            _forward_work(case, total, case["prompt"], 0, 1)
        for i in range(1, case["new"]):
            _forward_work(case, total, 1, case["prompt"] + i - 1, case["batch"])
    return total


def tolerance(case):
    """Four times what a change of summation order alone does: the same path with every linear done as an fp64 matmul of the
    dequantised weight.  Outputs are bf16 roundings of fp32 sums, so now and then two correct orders fall on either side of a
    rounding boundary."""
    op = case["op"]
    if op == "convert":
        return "exact"
    if op in ("linear", "block"):                            # up to 1.7e-4 and one bf16 spacing (7.8e-3) seen
        return {"rel": 7e-4, "max": 0.032}
    return {"rel": 2.8e-2, "max": 0.17, "differ": 0.01}      # logits and caches of two layers: 7.0e-3 and 4.2e-2 seen, no token moved
