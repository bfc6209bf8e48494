"""What is timed: the calls that a program built on this package makes, over the range of sizes it makes them at.

The package multiplies fp16 activations with 4-bit codebook weights.  A serving program quantizes its
weights once when a model is loaded (`quantize`), then issues GEMMs: one `matmul` per linear layer in the
decode steps (1 to 64 tokens, bound by the weights' bytes) and in the prefill steps (up to 4096 tokens, bound
by the tensor cores), `matmul_batched` / `matmul_sequence` for the experts of a mixture, a `MatmulSequence`
for GEMMs that do not depend on each other, a `HostSequence` where activations come from host memory, and
`dequant` where another kernel wants fp16 weights.  m = output features, n = tokens, k = reduction length;
the sizes are those of the layers the repository's own tables and benchmark name (hidden 4096 with a 14336-wide
MLP, hidden 8192 with a 28672-wide MLP, eight experts) or generic ones that no tile size divides.

Weights are normal, quantized row-wise with the default NF4 codebook; activations are normal.
"""

import random

import torch

import tuna_b200

MAX_FLOPS = 2 * 57344 * 4096 * 8192   # of the largest listed GEMM
MAX_BYTES = 2_900_000_000             # of the largest listed sequence


def listed():
    return [
        # a decode step of one sequence: the smallest layer (attention output), where latency and launch cost count
        {"name": "decode_1_attn", "op": "matmul", "m": 4096, "n": 1, "k": 4096},
        # a decode step of a batch of 16: gate+up projection
        {"name": "decode_16_gateup", "op": "matmul", "m": 28672, "n": 16, "k": 4096},
        # a decode step of 43 sequences on a layer whose sizes no tile divides
        {"name": "decode_43_ragged", "op": "matmul", "m": 11000, "n": 43, "k": 4104},
        # a short prompt, or a step that mixes prompts and decoding: QKV projection
        {"name": "prefill_256_qkv", "op": "matmul", "m": 6144, "n": 256, "k": 4096},
        # a prompt of a length that no tile divides, hidden size 8192
        {"name": "prefill_777_qkv", "op": "matmul", "m": 10240, "n": 777, "k": 8192},
        # the largest GEMM: gate+up of hidden size 8192 over a 4096-token prompt chunk
        {"name": "prefill_4096_gateup", "op": "matmul", "m": 57344, "n": 4096, "k": 8192},
        # independent GEMMs in one call: the MLP projections of 32 layers at 16 tokens (the benchmark's sweep)
        {"name": "sequence_mlp_32", "op": "sequence", "hidden": 4096, "inter": 14336, "layers": 32, "n": 16},
        # gate+up of a mixture's eight experts, 16 sequences with two experts each: new token lists in every step
        {"name": "experts_gateup", "op": "experts", "m": 28672, "k": 4096, "experts": 8, "tokens": 32, "routing": 3},
        # the down projections of the eight experts with 16 tokens each in one batched call
        {"name": "batched_down_16", "op": "batched", "m": 4096, "n": 16, "k": 14336, "batch": 8},
        # a layer's weights back to fp16
        {"name": "dequant_gateup", "op": "dequant", "m": 28672, "k": 4096},
        # a layer's weights quantized at load time
        {"name": "quantize_gateup", "op": "quantize", "m": 28672, "k": 4096},
        # activations and outputs in pinned host memory, weights resident: the MLP projections of 16 layers
        {"name": "host_mlp_16", "op": "host", "hidden": 4096, "inter": 14336, "layers": 16, "n": 16},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def _feature_size(rng, lo, hi):
    """A multiple of 8 (the packed layout's unit); half of the time one of 128, as most layers are."""
    step = 128 if rng.random() < 0.5 else 8
    return max(step, _log_int(rng, lo, hi) // step * step)


def draw(rng):
    """One more case of the ranges above: sizes log-uniform, redrawn until they cost no more than the largest listed case."""
    while True:
        op = rng.choice(["matmul"] * 10 + ["sequence", "experts", "batched", "dequant", "quantize", "host"])
        m, k = _feature_size(rng, 512, 57344), _feature_size(rng, 512, 28672)
        case = {"op": op, "m": m, "k": k}
        if op == "matmul":
            case["n"] = _log_int(rng, 1, 64) if rng.random() < 0.5 else _log_int(rng, 65, 4096)
        elif op == "batched":
            case.update(n=_log_int(rng, 1, 64), batch=rng.randint(2, 16))
        elif op == "experts":
            case.update(experts=rng.randint(4, 16), tokens=_log_int(rng, 4, 1024), routing=rng.randint(0, 1 << 20))
        elif op in ("sequence", "host"):
            hidden = _feature_size(rng, 1024, 8192)
            case = {"op": op, "hidden": hidden, "inter": _feature_size(rng, hidden, 4 * hidden), "layers": rng.randint(2, 32),
                    "n": _log_int(rng, 1, 64)}
        w = work(case)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= MAX_BYTES:
            return case


def _token_counts(case):
    """Tokens per expert: every token goes to one of the experts, popular ones get more (some may get none)."""
    rng = random.Random(case["routing"])
    weights = [rng.random() + 0.1 for _ in range(case["experts"])]
    counts = [0] * case["experts"]
    for e in rng.choices(range(case["experts"]), weights, k=case["tokens"]):
        counts[e] += 1
    return counts


def _gemm_shapes(case):
    """[(m, n, k), ...] of the case's GEMMs, without experts that got no token."""
    if case["op"] == "matmul":
        return [(case["m"], case["n"], case["k"])]
    if case["op"] == "batched":
        return [(case["m"], case["n"], case["k"])] * case["batch"]
    if case["op"] == "experts":
        return [(case["m"], n, case["k"]) for n in _token_counts(case) if n]
    return [(2 * case["inter"], case["n"], case["hidden"]), (case["hidden"], case["n"], case["inter"])] * case["layers"]


def work(case):
    """Packed weights (half a byte each), scales, codebook, activations and outputs once each; two operations per product."""
    if case["op"] in ("dequant", "quantize"):
        m, k = case["m"], case["k"]
        return {"bytes": m * k // 2 + 2 * m * k + 4 * m + 64, "flops": 0}
    shapes = _gemm_shapes(case)
    return {"bytes": 64 + sum(m * k // 2 + 4 * m + 2 * n * (m + k) for m, n, k in shapes),
            "flops": sum(2 * m * n * k for m, n, k in shapes)}


def tolerance(case):
    """Codes and dequantized weights are exact.  A GEMM accumulates in fp32 and rounds once to fp16: against sums in
    64 bits the GEMMs above show rel 2.1e-4 and max 5e-4 (two roundings differ by up to 1e-3); four times that."""
    if case["op"] in ("dequant", "quantize"):
        return "exact"
    return {"rel": 1e-3, "max": 4e-3}


def _weights(gen, m, k):
    w = torch.randn((m, k), generator=gen, device="cuda", dtype=torch.float16).mul_(k ** -0.5)
    q, (absmax, code) = tuna_b200.quantize(w)
    return q, absmax, code


def _activations(gen, *shape):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float16)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    op = case["op"]
    state = {"case": case}
    if op == "quantize":
        state["w"] = torch.randn((case["m"], case["k"]), generator=gen, device="cuda", dtype=torch.float16).mul_(case["k"] ** -0.5)
    elif op == "dequant":
        state["q"], state["s"], state["c"] = _weights(gen, case["m"], case["k"])
        state["o"] = torch.empty((case["m"], case["k"]), device="cuda", dtype=torch.float16)
    elif op == "matmul":
        m, n, k = case["m"], case["n"], case["k"]
        state["q"], state["s"], state["c"] = _weights(gen, m, k)
        state["x"] = _activations(gen, n, k)
        state["o"] = torch.empty((n, m), device="cuda", dtype=torch.float16)
    elif op == "batched":
        m, n, k, batch = case["m"], case["n"], case["k"], case["batch"]
        parts = [_weights(gen, m, k) for _ in range(batch)]
        state["q"] = torch.stack([p[0] for p in parts])
        state["s"] = torch.stack([p[1] for p in parts])
        state["c"] = parts[0][2]
        state["x"] = _activations(gen, batch, n, k)
        state["o"] = torch.empty((batch, n, m), device="cuda", dtype=torch.float16)
    elif op == "experts":
        # the tokens of all experts lie expert by expert in one buffer, as routing leaves them
        m, k, counts = case["m"], case["k"], _token_counts(case)
        x = _activations(gen, case["tokens"], k)
        o = torch.empty((case["tokens"], m), device="cuda", dtype=torch.float16)
        state["experts"] = [_weights(gen, m, k) for _ in counts]
        state["counts"], state["x"], state["o"] = counts, x, o
    else:
        host = op == "host"
        shapes = _gemm_shapes(case)
        xs = _activations(gen, sum(n * k for m, n, k in shapes))
        os_ = torch.empty(sum(n * m for m, n, k in shapes), dtype=torch.float16, device="cuda")
        if host:  # one pinned buffer each way
            xs, os_ = xs.cpu().pin_memory(), torch.empty(os_.shape, dtype=torch.float16, pin_memory=True)
        gemms, x0, o0 = [], 0, 0
        for m, n, k in shapes:
            q, s, c = _weights(gen, m, k)
            gemms.append((xs[x0:x0 + n * k].view(n, k), q, s, os_[o0:o0 + n * m].view(n, m), m, n, k))
            x0, o0 = x0 + n * k, o0 + n * m
        state["handle"] = tuna_b200.HostSequence(gemms, c) if host else tuna_b200.MatmulSequence(gemms, c)
        state["o"] = os_
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "quantize":
        q, (absmax, code) = tuna_b200.quantize(state["w"])
        return {"q": q, "absmax": absmax, "code": code}
    if op == "dequant":
        tuna_b200.dequant(state["q"], state["s"], state["c"], state["o"], case["m"], case["k"])
    elif op == "matmul":
        tuna_b200.matmul(state["x"], state["q"], state["s"], state["c"], state["o"], case["m"], case["n"], case["k"])
    elif op == "batched":
        tuna_b200.matmul_batched(state["x"], state["q"], state["s"], state["c"], state["o"], case["m"], case["n"], case["k"])
    elif op == "experts":
        m, k, x, o = case["m"], case["k"], state["x"], state["o"]
        gemms, first = [], 0
        for (q, s, c), n in zip(state["experts"], state["counts"]):
            gemms.append((x[first:first + n], q, s, o[first:first + n], m, n, k))
            first += n
        tuna_b200.matmul_sequence(gemms, c)
    else:
        state["handle"].run()
    return state["o"]
