"""Performance cases of the rosa_soft operator family.

Each case is one pass of work that users of this package do, through its public entry points:
a training step of the operator (dense or packed batches), scoring without gradients, batched
hard inference, and streaming sessions of the runtime (prompt and token-by-token generation).

``listed()``   the fixed cases
``draw(rng)``  one more case of the same ranges
``prepare``    inputs on the GPU from a seed, and the runtime object of a streaming session
``run``        one pass; returns everything the pass computes
``work``       bytes and operations a pass cannot do without
``tolerance``  how far a correct implementation of the same precision may be off
"""
from __future__ import annotations

import random

import torch

import rosa_soft_b200 as rosa

DEVICE = "cuda"
ELEMENT = {"float32": 4, "float16": 2, "bfloat16": 2}


# ------------------------------------------------------------------------------------- cases
def _train(name, B, T, H, D, Hv, Dv, W, p, m, dtype, data="normal"):
    return {"name": name, "kind": "train", "B": B, "T": T, "H": H, "D": D, "Hv": Hv, "Dv": Dv, "W": W,
            "p": p, "m": m, "dtype": dtype, "data": data}


def _packed(name, N, Lmin, Lmax, mix, H, D, Hv, Dv, W, p, m, dtype, data="normal"):
    return {"name": name, "kind": "packed", "N": N, "Lmin": Lmin, "Lmax": Lmax, "mix": mix, "H": H,
            "D": D, "Hv": Hv, "Dv": Dv, "W": W, "p": p, "m": m, "dtype": dtype, "data": data}


def listed():
    return [
        # Smallest training step: the configuration that a unit test or a first experiment runs.
        _train("train_tiny_f32", 1, 256, 4, 4, 4, 8, 32, 0.0, 3.0, "float32"),
        # The README training shape in both training precisions.
        _train("train_readme_f32", 2, 1024, 64, 8, 16, 8, 128, 0.1, 3.0, "float32"),
        _train("train_readme_bf16", 2, 1024, 64, 8, 16, 8, 128, 0.1, 3.0, "bfloat16"),
        # The headline long-context training step, whole batch on one GPU: the largest case.
        _train("train_long_bf16", 16, 8192, 64, 8, 16, 8, 128, 0.1, 3.0, "bfloat16"),
        # Low-entropy stream with repeated segments: matches run into the horizon, no dropout.
        _train("train_repeats_bf16", 4, 8192, 64, 2, 64, 16, 256, 0.0, 3.0, "bfloat16", "repeats"),
        # Symbols wider than 16 bits and an odd length.
        _train("train_wide_f16", 1, 2047, 16, 24, 4, 32, 64, 0.05, 9.0, "float16"),
        # Packed pre-training batch: sequences of 64..4096 tokens in 32768.
        _packed("train_packed_f16", 32768, 64, 4096, 1, 32, 16, 8, 32, 64, 0.05, 9.0, "float16"),
        # Packed fine-tuning batch of many short ragged sequences.
        _packed("train_ragged_bf16", 3001, 1, 257, 2, 16, 8, 4, 8, 32, 0.1, 3.0, "bfloat16", "repeats"),
        # Scoring of a batch without gradients.
        {"name": "score_bf16", "kind": "score", "B": 4, "T": 4095, "H": 32, "D": 8, "Hv": 8, "Dv": 8,
         "W": 128, "dtype": "bfloat16", "data": "repeats"},
        # Batched hard inference over 32-bit symbols with float payload.
        {"name": "inference_32bit", "kind": "inference", "B": 64, "T": 16384, "H": 64, "Hp": 64, "Dp": 8,
         "W": 32},
        # Prompts of many streams fed to the runtime in chunks.
        {"name": "stream_prompts", "kind": "stream", "B": 64, "T": 16384, "H": 64, "Hp": 64, "bits": 8,
         "payload_bits": 8, "W": 32, "chunk": 2048},
        # Generation: a prompt of logits, then single tokens per slot, results as +-1 values.
        {"name": "stream_generate", "kind": "generate", "B": 8, "T": 2001, "H": 32, "Hp": 8, "bits": 8,
         "payload_bits": 8, "W": 32, "steps": 24, "dtype": "bfloat16"},
    ]


def _log_int(rng, lo, hi):
    """An integer between lo and hi, spread over its logarithm."""
    return min(hi, max(lo, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(("train", "train", "train", "packed", "packed", "score", "inference", "stream",
                       "generate"))
    H = rng.choice((4, 8, 12, 16, 32, 64))
    Hv = H // rng.choice((1, 2, 4))
    W = rng.choice((16, 32, 64, 128, 256))
    data = rng.choice(("normal", "repeats"))
    if kind in ("train", "packed"):
        D, Dv = rng.choice(((2, 16), (4, 8), (8, 8), (8, 8), (8, 16), (12, 8), (16, 32), (20, 24), (24, 32),
                            (8, 64)))
        p, m = rng.choice((0.0, 0.05, 0.1)), rng.choice((3.0, 9.0))
        dtype = rng.choice(("bfloat16", "bfloat16", "float16", "float32"))
    if kind == "train":
        T = _log_int(rng, 64, 8192)
        most = max(1, min(32, 2 ** 31 // (H * T * T), 2 ** 22 // (H * T)))
        return {"kind": kind, "B": _log_int(rng, 1, most), "T": T, "H": H, "D": D, "Hv": Hv, "Dv": Dv,
                "W": W, "p": p, "m": m, "dtype": dtype, "data": data}
    if kind == "packed":
        Lmax = _log_int(rng, 64, 4096)
        N = _log_int(rng, 512, max(1024, min(32768, 2 ** 30 // (H * Lmax))))
        return {"kind": kind, "N": N, "Lmin": rng.randint(1, 64), "Lmax": Lmax, "mix": rng.randrange(1000),
                "H": H, "D": D, "Hv": Hv, "Dv": Dv, "W": W, "p": p, "m": m, "dtype": dtype, "data": data}
    if kind == "score":
        T = _log_int(rng, 64, 8192)
        return {"kind": kind, "B": _log_int(rng, 1, max(1, min(32, 2 ** 20 // (H * T)) * 4)), "T": T, "H": H,
                "D": rng.choice((2, 4, 8, 16, 24)), "Hv": Hv, "Dv": rng.choice((8, 12, 16, 32)), "W": W,
                "dtype": rng.choice(("bfloat16", "float16", "float32")), "data": data}
    T = _log_int(rng, 128, 16384)
    B = _log_int(rng, 1, max(1, min(64, 2 ** 25 // (H * T))))
    if kind == "inference":
        return {"kind": kind, "B": B, "T": T, "H": H, "Hp": Hv, "Dp": rng.choice((1, 4, 8, 16)), "W": W}
    bits, payload_bits = rng.choice((4, 6, 8, 8)), rng.choice((1, 4, 8))
    if kind == "stream":
        return {"kind": kind, "B": B, "T": T, "H": H, "Hp": Hv, "bits": bits, "payload_bits": payload_bits,
                "W": W, "chunk": max(1 + T // 16, _log_int(rng, 64, 4096))}
    return {"kind": kind, "B": B, "T": T, "H": H, "Hp": Hv, "bits": bits, "payload_bits": payload_bits, "W": W,
            "steps": rng.randint(4, 24), "dtype": rng.choice(("bfloat16", "float32"))}


def _lengths(case):
    """Sequence lengths of a packed case: uniform in [Lmin, Lmax] until the tokens are used up."""
    rng = random.Random(case["mix"])
    lengths, left = [], case["N"]
    while left > 0:
        lengths.append(min(left, rng.randint(min(case["Lmin"], case["Lmax"]), case["Lmax"])))
        left -= lengths[-1]
    return lengths


# ------------------------------------------------------------------------------------ inputs
def _repeating_tokens(rows, tokens, bits, rng, gen):
    """[rows, tokens] symbols of `bits` bits in which segments of 16..256 tokens repeat earlier ones
    30 % of the time."""
    out = torch.randint(0, 1 << bits, (rows, tokens), generator=gen, device=DEVICE, dtype=torch.int32)
    at = 0
    while at < tokens:
        n = min(rng.randint(16, 256), tokens - at)
        if rng.random() < 0.3 and at > n:
            src = rng.randint(0, at - n)
            out[:, at:at + n] = out[:, src:src + n]
        at += n
    return out


def _copied_windows(q, k, rng):
    """q, k [B, T, H]: every now and then both streams go on with a copy of an earlier window of
    8..512 positions, so that long matches exist."""
    B, T = q.shape[:2]
    for b in range(B):
        t = min(600, T // 4 + 8)
        while t < T - 9:
            if rng.random() < 0.1:
                n = min(rng.randint(8, 512), T - 1 - t, t)
                src = rng.randint(0, t - n)
                k[b, t:t + n] = k[b, src:src + n]
                q[b, t + 1:t + 1 + n] = k[b, src + 1:src + 1 + n]
                t += n
            t += rng.randint(1, 19)


def _operator_inputs(case, lead, seed, gen):
    """Query, key, value logits and the upstream gradient: standard normal, or for "repeats" +-1
    sign patterns of a token stream that repeats itself (query and key carry the same stream)."""
    dtype = getattr(torch, case["dtype"])
    H, D, Hv, Dv = case["H"], case["D"], case["Hv"], case["Dv"]
    normal = lambda *tail: torch.randn(*lead, *tail, generator=gen, device=DEVICE).to(dtype)  # noqa: E731
    if case["data"] == "repeats":
        rows = H * (lead[0] if len(lead) == 2 else 1)
        tokens = _repeating_tokens(rows, lead[-1], D, random.Random(seed), gen)
        bits = (tokens.unsqueeze(-1) >> torch.arange(D, device=DEVICE, dtype=torch.int32)) & 1
        logits = (2 * bits - 1).to(dtype).reshape(*lead[:-1], H, lead[-1], D).movedim(-3, -2)
        q = logits.contiguous()
        k = q.clone()
    else:
        q, k = normal(H, D), normal(H, D)
    return q, k, normal(Hv, Dv), normal(H, Dv)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind in ("train", "packed", "score"):
        lead = (case["N"],) if kind == "packed" else (case["B"], case["T"])
        q, k, v, go = _operator_inputs(case, lead, seed, gen)
        state = {"kind": kind, "q": q, "k": k, "v": v}
        if kind == "score":
            state["controls"] = {"max_suffix_length": case["W"]}
            return state
        for t in (q, k, v):
            t.requires_grad_(True)
        state["go"] = go
        state["dropout_seed"] = seed
        state["controls"] = {"max_suffix_length": case["W"], "scale": 1.0, "dropout_p": case["p"],
                             "mismatch_scale": case["m"]}
        if kind == "packed":
            offsets = [0]
            for n in _lengths(case):
                offsets.append(offsets[-1] + n)
            state["cu_seqlens"] = torch.tensor(offsets, dtype=torch.int32, device=DEVICE)
        return state
    B, T, H, Hp = case["B"], case["T"], case["H"], case["Hp"]
    rng = random.Random(seed)
    if kind == "inference":
        q = torch.randint(-2 ** 31, 2 ** 31, (B, T, H), generator=gen, device=DEVICE).to(torch.int32)
        k = torch.randint(-2 ** 31, 2 ** 31, (B, T, H), generator=gen, device=DEVICE).to(torch.int32)
        _copied_windows(q, k, rng)
        payload = torch.randn(B, T, Hp, case["Dp"], generator=gen, device=DEVICE)
        return {"kind": kind, "q": q, "k": k, "payload": payload, "W": case["W"]}
    runtime = rosa.RosaRuntime(H, Hp, case["bits"], case["payload_bits"], case["W"])
    total = T + case.get("steps", 0)
    draw_symbols = lambda heads, bits: torch.randint(0, 1 << bits, (B, total, heads), generator=gen,  # noqa: E731
                                                     device=DEVICE, dtype=torch.uint8)
    q, k, pay = draw_symbols(H, case["bits"]), draw_symbols(H, case["bits"]), draw_symbols(Hp, case["payload_bits"])
    _copied_windows(q, k, rng)
    if kind == "stream":
        cuts = list(range(0, T, case["chunk"]))
        return {"kind": kind, "runtime": runtime,
                "chunks": [tuple(t[:, a:a + case["chunk"]].contiguous() for t in (q, k, pay)) for a in cuts]}
    # generation: the logits of the prompt and of every later token, as the projections give them
    dtype = getattr(torch, case["dtype"])

    def logits(symbols, bits):
        ones = (symbols.to(torch.int32).unsqueeze(-1) >> torch.arange(bits, device=DEVICE)) & 1
        size = torch.rand(ones.shape, generator=gen, device=DEVICE) + 0.05
        return ((2 * ones - 1) * size).to(dtype)

    q, k, pay = logits(q, case["bits"]), logits(k, case["bits"]), logits(pay, case["payload_bits"])
    cuts = [(0, T)] + [(t, t + 1) for t in range(T, total)]
    return {"kind": kind, "runtime": runtime,
            "chunks": [tuple(t[:, a:b].contiguous() for t in (q, k, pay)) for a, b in cuts]}


# --------------------------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind in ("train", "packed"):
        q, k, v = state["q"], state["k"], state["v"]
        # the dropout masks follow the device generator, as they do under activation checkpointing
        torch.cuda.manual_seed(state["dropout_seed"])
        if kind == "train":
            out = rosa.rosa_soft(q, k, v, **state["controls"])
        else:
            out = rosa.rosa_soft_varlen(q, k, v, state["cu_seqlens"], **state["controls"])
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["go"])
        return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}
    if kind == "score":
        with torch.no_grad():
            return rosa.rosa_soft(state["q"], state["k"], state["v"], **state["controls"])
    if kind == "inference":
        out, end = rosa.rosa_hard_inference(state["q"], state["k"], state["payload"],
                                            max_suffix_length=state["W"])
        return {"out": out, "end": end}
    runtime = state["runtime"]
    runtime.reset()
    update = runtime.update_packed if kind == "stream" else runtime.update
    return [update(q, k, payload) for q, k, payload in state["chunks"]]


# ---------------------------------------------------------------------------------- accounts
def _pairs(case):
    if case["kind"] == "packed":
        return case["H"] * sum(n * (n - 1) // 2 for n in _lengths(case))
    return case["H"] * case["B"] * (case["T"] * (case["T"] - 1) // 2)


def work(case):
    kind = case["kind"]
    if kind in ("train", "packed", "score"):
        N = case["N"] if kind == "packed" else case["B"] * case["T"]
        s = ELEMENT[case["dtype"]]
        qk, v, out = 2 * case["H"] * case["D"], case["Hv"] * case["Dv"], case["H"] * case["Dv"]
        if kind == "score":
            return {"bytes": N * s * (qk + v + out), "flops": 0}
        # inputs and upstream gradient in, output and gradients out; the dense contraction of the
        # backward: 6 D + 4 Dv operations per causal pair
        return {"bytes": N * s * (2 * qk + 2 * v + 2 * out),
                "flops": (6 * case["D"] + 4 * case["Dv"]) * _pairs(case)}
    N = case["B"] * (case["T"] + case.get("steps", 0))
    H, Hp = case["H"], case["Hp"]
    if kind == "inference":
        return {"bytes": N * (2 * 4 * H + 4 * Hp * case["Dp"] + 4 * H * case["Dp"] + 8 * H), "flops": 0}
    if kind == "stream":
        return {"bytes": N * (2 * H + Hp + H + 8 * H), "flops": 0}
    s = ELEMENT[case["dtype"]]
    return {"bytes": N * (s * (2 * H * case["bits"] + Hp * case["payload_bits"] + H * case["payload_bits"])
                          + 8 * H), "flops": 0}


def tolerance(case):
    if case["kind"] in ("train", "packed"):
        # gradients: float32 sums, or the rounding of the input type (the bfloat16 contraction keeps
        # eight bits of the weighted probabilities)
        return {"rel": {"float32": 2e-5, "float16": 2e-3, "bfloat16": 1e-2}[case["dtype"]]}
    return "exact"      # routed signs, payload copies, symbols and positions
