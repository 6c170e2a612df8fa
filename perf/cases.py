"""Performance cases: what users of this package have it do, through its public entry points.

Two families of calls.  Attention: `adasplash_v2` (causal, alpha = 1.5: training steps, forward-only
prefill, grouped heads with ragged lengths, long context) and `adasplash_v1` (any alpha, causal or full
attention), mostly 16-bit, fp32 for small models and checks.  Row-wise: `triton_entmax` as the activation of
a dense layer or of attention scores, from a few rows to a vocabulary-sized output layer.

Inputs are seeded normal tensors with the spreads of this repository's benchmark and tests: queries and keys
of standard deviation 1.0 to 1.5, row-wise inputs of 2 to 4.
"""
import math

import torch

import adasplash_b200 as adasplash

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}


def _attn(name, B, Hq, Hkv, N, D, dtype="bf16", scale=1.5, ragged=False, backward=True, alpha=1.5, causal=True,
          niter=1):
    return dict(name=name, op="attention", B=B, Hq=Hq, Hkv=Hkv, N=N, D=D, dtype=dtype, scale=scale, ragged=ragged,
                backward=backward, alpha=alpha, causal=causal, niter=niter)


def _rows(name, rows, cols, dtype="fp32", alpha=1.5, scale=4.0, backward=True):
    return dict(name=name, op="rowwise", rows=rows, cols=cols, dtype=dtype, alpha=alpha, scale=scale,
                backward=backward)


def listed():
    return [
        # The smallest training step: one short sequence, two heads.  Host work and launches.
        _attn("attn_step_n256", 1, 2, 2, 256, 64, scale=1.0),
        # Forward-only prefill of one medium prompt (inference, no gradients).
        _attn("attn_prefill_n2048", 1, 8, 8, 2048, 128, backward=False),
        # The headline training step: a batch of 8192-token sequences, 32 heads.
        _attn("attn_step_n8192", 4, 32, 32, 8192, 128),
        # Training with grouped key heads and right-padded sequences of many lengths; unit-variance
        # queries and keys, i.e. flat rows with dozens of non-zero probabilities.
        _attn("attn_step_gqa_ragged_n16384", 8, 32, 8, 16384, 128, scale=1.0, ragged=True),
        # Long context: one GPU's share of a long-document job (two sequences, one key head of eight).
        _attn("attn_step_n65536", 2, 8, 1, 65536, 128),
        # Sparsemax attention without a mask (an encoder), first-generation entry point.
        _attn("attn_sparsemax_full_n8192", 4, 32, 32, 8192, 64, alpha=2.0, causal=False, niter=10),
        # Another alpha, an odd length, fp16, padded batch: a fine-tuning step of a mid-sized decoder.
        _attn("attn_a1333_ragged_n1500", 4, 16, 16, 1500, 64, dtype="fp16", ragged=True, alpha=1.333, niter=10),
        # fp32 attention: small research models and gradient checks.
        _attn("attn_step_fp32_n2048", 1, 8, 8, 2048, 64, dtype="fp32", scale=1.0),
        # Row-wise entmax over a tall matrix (dense attention scores, routing): bound by memory.
        _rows("rows_16384x4096", 16384, 4096),
        # A few short rows: a classifier's output layer.  Host work and launches.
        _rows("rows_64x1000_sparsemax", 64, 1000, alpha=2.0, scale=2.0),
        # Output layer over a vocabulary with an odd number of entries.
        _rows("rows_2048x50001", 2048, 50001),
        # 16-bit dense attention probabilities of a short context with another alpha.
        _rows("rows_65536x1000_a1333_bf16", 65536, 1000, dtype="bf16", alpha=1.333, scale=2.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges."""
    if rng.random() < 0.35:
        cols = _log_int(rng, 32, 60000)
        if rng.random() < 0.5:
            cols = max(32, cols // 8 * 8)
        rows = _log_int(rng, 16, max(32, min(200000, 100_000_000 // cols)))
        c = _rows("", rows, cols, dtype=rng.choice(["fp32", "fp32", "bf16", "fp16"]),
                  alpha=rng.choice([1.5, 1.5, 2.0, 1.333]), scale=round(rng.uniform(2.0, 4.0), 2),
                  backward=rng.random() < 0.8)
    elif rng.random() < 0.7:
        dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])
        D = rng.choice([64, 128])
        G = rng.choice([1, 1, 4, 8])
        ragged = rng.random() < 0.5
        n_max = 2048 if dtype == "fp32" else 32768
        N = _log_int(rng, 128, n_max) if ragged else 2 ** rng.randint(7, int(math.log2(n_max)))
        # heads x batch so that the dense work stays well below the largest listed case
        room = (2 ** 28 if dtype == "fp32" else 2 ** 36) // (N * N * D // 64)
        Hkv = max(1, min(8, _log_int(rng, 1, 8), room // G))
        B = max(1, min(8, _log_int(rng, 1, 8), room // (G * Hkv)))
        c = _attn("", B, Hkv * G, Hkv, N, D, dtype=dtype, scale=round(rng.uniform(1.0, 1.5), 2), ragged=ragged,
                  backward=rng.random() < 0.75, niter=rng.choice([1, 1, 1, 2, 4]))
    else:
        N = _log_int(rng, 100, 8192)
        H = rng.choice([2, 4, 8, 16])
        B = max(1, min(4, 2 ** 32 // (N * N * H)))
        c = _attn("", B, H, H, N, 64, dtype=rng.choice(["bf16", "fp16"]), scale=round(rng.uniform(1.0, 1.5), 2),
                  ragged=rng.random() < 0.5, backward=rng.random() < 0.75, alpha=rng.choice([2.0, 1.333, 1.75]),
                  causal=rng.random() < 0.5, niter=10)
    del c["name"]
    return c


def _lengths(case, seed):
    if not case.get("ragged"):
        return [case["N"]] * case["B"]
    g = torch.Generator().manual_seed(seed)
    return [int(x) for x in torch.randint(max(1, case["N"] // 4), case["N"] + 1, (case["B"],), generator=g)]


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(seed)
    dt = DTYPES[case["dtype"]]

    def normal(shape, scale):
        t = torch.empty(shape, dtype=dt, device=dev)
        for i in range(shape[0]) if len(shape) == 4 else (slice(None),):   # bounds the fp32 temporary
            t[i] = (torch.randn(t[i].shape, generator=g, device=dev) * scale).to(dt)
        return t

    s = {"case": case}
    if case["op"] == "rowwise":
        shape = (case["rows"], case["cols"])
        s["x"] = normal(shape, case["scale"])
        if case["backward"]:
            s["x"].requires_grad_(True)
            s["dy"] = normal(shape, 1.0)
        return s
    B, N, D = case["B"], case["N"], case["D"]
    s["q"] = normal((B, case["Hq"], N, D), case["scale"])
    s["k"] = normal((B, case["Hkv"], N, D), case["scale"])
    s["v"] = normal((B, case["Hkv"], N, D), case["scale"])
    s["varlen"] = None
    if case["ragged"]:
        s["varlen"] = torch.tensor(_lengths(case, seed), dtype=torch.int32, device=dev)
    if case["backward"]:
        for n in "qkv":
            s[n].requires_grad_(True)
        s["do"] = normal((B, case["Hq"], N, D), 1.0)
        if case["ragged"]:   # the loss does not see padded positions
            s["do"].mul_((torch.arange(N, device=dev) < s["varlen"][:, None])[:, None, :, None])
    return s


def run(state):
    case = state["case"]
    if case["op"] == "rowwise":
        y = adasplash.triton_entmax(state["x"], alpha=case["alpha"])
        if not case["backward"]:
            return {"y": y}
        (dx,) = torch.autograd.grad(y, state["x"], state["dy"])
        return {"y": y, "dx": dx}
    q, k, v = state["q"], state["k"], state["v"]
    if case["alpha"] == 1.5 and case["causal"]:
        out = adasplash.adasplash_v2(q, k, v, niter=case["niter"], varlen=state["varlen"])
    else:
        out = adasplash.adasplash_v1(q, k, v, alpha=case["alpha"], is_causal=case["causal"],
                                     varlen=state["varlen"], niter=case["niter"])
    if not case["backward"]:
        return {"out": out}
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["do"])
    return {"out": out, "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Row-wise: x in and y out, and for the backward dy in and dx out.  Attention: q, k, v in, out out, and for
    the backward dO in, dq, dk, dv out; the operations are one product of every query with every key it
    may see (what the threshold of a row depends on) -- the few non-zero probabilities add little to that."""
    w = SIZE[case["dtype"]]
    if case["op"] == "rowwise":
        return {"bytes": (4 if case["backward"] else 2) * w * case["rows"] * case["cols"],
                "flops": (8 if case["backward"] else 4) * case["rows"] * case["cols"]}
    B, N, D = case["B"], case["N"], case["D"]
    q, kv = B * case["Hq"] * N * D * w, B * case["Hkv"] * N * D * w
    nbytes = 2 * q + 2 * kv + ((2 * q + 2 * kv) if case["backward"] else 0)
    n2 = N * N * (7.0 / 16.0) if case["ragged"] else float(N * N)   # mean of L^2 for L uniform on [N/4, N]
    return {"bytes": nbytes, "flops": 2.0 * D * B * case["Hq"] * n2 * (0.5 if case["causal"] else 1.0)}


def tolerance(case):
    if case["dtype"] == "fp32":
        # 32-bit sums, a fixed number of threshold steps: a score that a rounding moves over the edge of a
        # histogram bin starts its row's steps elsewhere
        return {"rel": 1e-4, "max": 2e-2}
    if case["op"] == "attention" and case["alpha"] > 1.5:
        # Above alpha = 1.5 a key enters the support with a Jacobian weight that does not start from zero:
        # a score within a 16-bit rounding of the threshold may be in or out, with its whole gradient.
        return {"rel": 1e-2, "max": 0.99}
    return {"rel": 1e-2}
