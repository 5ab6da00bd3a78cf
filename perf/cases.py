"""The work that a user of this library has it do, as cases whose time and results can be measured.

Every case goes through the public entry points (``GreedySampler``, ``StochasticSampler``, ``sample``, ``draft_q``, ``verify``,
``lm_head``). Sizes are those of the benchmark configurations and of the tests: vocabularies of 151,936 / 248,320 / 262,144 (and the
odd 50,257), one row to 4096 rows, BF16 and FP32 logits, the 8 rows of a speculative round, a hidden size of 4096. Logits are
N(0, 2^2), with a few spikes where the configuration has them; histories are uniform token ids.
"""
from __future__ import annotations

import math

import torch

import lithos_metal_b200 as lm

RHO, PI = 1.1, 0.5                       # repetition and presence penalty of the batched configurations
MIX_TOP_K = (0, 20, 50, 1000)            # per-row top_k of the batched configurations


def listed():
    return [
        # One stream, greedy: the smallest call of a decode loop.
        dict(name="greedy-1", kind="greedy", rows=1, vocab=151936, dtype="bf16", spikes=0),
        # One stream, temperature / top-k / top-p on FP32 logits with injected uniforms (the single-row configuration).
        dict(name="topk-topp-1-fp32", kind="sample", rows=1, vocab=151936, dtype="fp32", temperature=0.7, top_k=20, top_p=0.95, min_p=0.0,
             hist=0, draw="inverse_cdf", spikes=8),
        # A handful of chat streams in one step: nucleus sampling without a top_k, the reference's counter-based draw and module.
        dict(name="nucleus-4", kind="module", rows=4, vocab=248320, dtype="bf16", temperature=0.8, top_k=0, top_p=0.95, min_p=0.0, spikes=8),
        # The verification of seven sampled drafts given as probabilities (the speculative configuration).
        dict(name="verify-7", kind="verify", n_draft=7, vocab=151936, dtype="bf16", temperature=1.0, mode="stochastic"),
        # One speculative round: the drafter's draws, the target's thresholds, the verification fed with both rows of statistics.
        dict(name="round-7", kind="round", n_draft=7, vocab=151936, temperature=0.8, top_k=50, top_p=0.95),
        # A serving batch of FP32 logits, every request with its own knobs, counter-based draws.
        dict(name="mixed-64-fp32", kind="mixed", rows=64, vocab=151936, dtype="fp32", hist=0, draw="gumbel"),
        # A batch over a vocabulary that is no multiple of anything: rows start at odd addresses. Penalties over the tokens so far.
        dict(name="mixed-48-odd-vocab", kind="mixed", rows=48, vocab=50257, dtype="bf16", hist=512, draw="gumbel"),
        # Whole rows of the large-vocabulary configuration, one set of knobs.
        dict(name="topk-topp-64-262144", kind="sample", rows=64, vocab=262144, dtype="bf16", temperature=0.8, top_k=50, top_p=0.9, min_p=0.0,
             hist=0, draw="inverse_cdf", spikes=0),
        # The batched penalised configuration.
        dict(name="mixed-256-penalised", kind="mixed", rows=256, vocab=151936, dtype="bf16", hist=2048, draw="inverse_cdf"),
        # The large batch that the benchmark is quoted on.
        dict(name="mixed-4096-penalised", kind="mixed", rows=4096, vocab=151936, dtype="bf16", hist=2048, draw="inverse_cdf"),
        # The kept-token probability vectors of a few rows (log-probabilities for a client, distribution checks).
        dict(name="probs-4-fp32", kind="probs", rows=4, vocab=151936, dtype="fp32", temperature=0.7, top_k=20, top_p=0.95, min_p=0.0, spikes=8),
        # The vocabulary projection in front of all this, final norm fused, for the 8 rows of a speculative round.
        dict(name="lm-head-8", kind="head", rows=8, hidden=4096, vocab=151936, norm=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vocab(rng, lo=16384, hi=262144):
    """Any size between the bounds; half of them a multiple of 64, as padded vocabularies are."""
    v = _log_int(rng, lo, hi)
    return v if rng.random() < 0.5 else max(lo, min(hi, (v + 63) // 64 * 64))


def _rows_within(rng, vocab, width, lo=1, hi=4096, budget=300 << 20):
    return max(lo, min(_log_int(rng, lo, hi), budget // (vocab * width)))


def draw(rng):
    kind = rng.choice(["greedy", "sample", "sample", "module", "verify", "round", "mixed", "mixed", "mixed", "probs", "head"])
    dtype = rng.choice(["bf16", "bf16", "fp32"])
    width = 2 if dtype == "bf16" else 4
    vocab = _vocab(rng)
    knobs = dict(temperature=round(rng.uniform(0.3, 1.5), 3), top_k=rng.choice([0, 0, rng.randint(1, 64), rng.randint(65, 1000)]),
                 top_p=rng.choice([0.0, round(rng.uniform(0.5, 0.99), 3), round(rng.uniform(0.8, 0.99), 3)]), min_p=rng.choice([0.0, 0.0, 0.0, 0.02]))
    if kind == "greedy":
        return dict(kind=kind, rows=_rows_within(rng, vocab, width), vocab=vocab, dtype=dtype, spikes=rng.choice([0, 8]))
    if kind == "sample":
        return dict(kind=kind, rows=_rows_within(rng, vocab, width, hi=512), vocab=vocab, dtype=dtype, hist=rng.choice([0, 0, _log_int(rng, 16, 2048)]),
                    draw=rng.choice(["inverse_cdf", "gumbel"]), spikes=rng.choice([0, 8]), **knobs)
    if kind == "module":
        return dict(kind=kind, rows=_rows_within(rng, vocab, width, hi=32), vocab=vocab, dtype=dtype, spikes=rng.choice([0, 8]), **knobs)
    if kind == "verify":
        return dict(kind=kind, n_draft=rng.randint(1, 15), vocab=vocab, dtype=dtype, temperature=knobs["temperature"], mode=rng.choice(["greedy", "stochastic", "stochastic"]))
    if kind == "round":
        return dict(kind=kind, n_draft=rng.randint(2, 15), vocab=vocab, temperature=knobs["temperature"], top_k=rng.randint(1, 64), top_p=round(rng.uniform(0.8, 0.99), 3))
    if kind == "mixed":
        return dict(kind=kind, rows=_rows_within(rng, vocab, width, lo=8, hi=1024), vocab=vocab, dtype=dtype, hist=rng.choice([0, _log_int(rng, 64, 2048)]),
                    draw=rng.choice(["inverse_cdf", "gumbel"]))
    if kind == "probs":
        return dict(kind=kind, rows=rng.randint(1, 16), vocab=vocab, dtype=dtype, spikes=rng.choice([0, 8]), **knobs)
    return dict(kind=kind, rows=rng.randint(1, 8), hidden=64 * _log_int(rng, 8, 96), vocab=_vocab(rng, 16384, 131072), norm=rng.random() < 0.7)


# ---- inputs ---------------------------------------------------------------------------------------------------------------------

def _logits(g, rows, vocab, dtype, spikes=0):
    dev = torch.device("cuda")
    out = torch.empty(rows, vocab, dtype=torch.bfloat16 if dtype == "bf16" else torch.float32, device=dev)
    step = max(1, (64 << 20) // vocab)
    for r0 in range(0, rows, step):                                          # bounded temporaries
        n = min(step, rows - r0)
        out[r0:r0 + n] = torch.randn(n, vocab, generator=g, device=dev) * 2.0
    if spikes:
        at = torch.randint(0, vocab, (rows, spikes), generator=g, device=dev)
        out.scatter_(1, at, 12.0)
    return out


def _history(g, rows, vocab, n):
    return torch.randint(0, vocab, (rows, n), generator=g, device="cuda", dtype=torch.int32) if n else None


def prepare(case, seed):
    dev = torch.device("cuda")
    g = torch.Generator(device=dev)
    g.manual_seed(int(seed))
    kind = case["kind"]
    s = {"kind": kind, "seed": int(seed) & 0x7FFFFFFF}
    if kind == "head":
        H, V = case["hidden"], case["vocab"]
        s["hidden"] = torch.randn(case["rows"], H, generator=g, device=dev).to(torch.bfloat16)
        s["weight"] = (torch.randn(V, H, generator=g, device=dev, dtype=torch.bfloat16) * 0.02)
        s["norm"] = (torch.randn(H, generator=g, device=dev) * 0.1).to(torch.bfloat16) if case["norm"] else None
        return s
    if kind in ("verify", "round"):
        n, V, T = case["n_draft"], case["vocab"], case["temperature"]
        s["temperature"] = T
        s["target"] = _logits(g, n + 1, V, case.get("dtype", "bf16"))
        noisy = s["target"][:n].float() + torch.randn(n, V, generator=g, device=dev) * 0.5
        s["u_accept"] = torch.rand(n, generator=g, device=dev)
        s["u_final"] = torch.rand(1, generator=g, device=dev)
        if kind == "verify":
            s["mode"] = case["mode"]
            s["drafts"] = torch.randint(0, V, (n,), generator=g, device=dev, dtype=torch.int32)
            if case["mode"] == "greedy":                                     # drafts of a good drafter: the first few agree
                s["drafts"][: n // 2] = s["target"][: n // 2].float().argmax(-1).to(torch.int32)
            s["probs"] = torch.softmax(noisy / T, -1) if case["mode"] == "stochastic" else None
        else:
            s["draft_logits"] = noisy.to(torch.bfloat16)
            s["params"] = lm.SamplingParams(temperature=T, top_k=case["top_k"], top_p=case["top_p"], seed=s["seed"], draw="gumbel")
        return s
    rows, V = case["rows"], case["vocab"]
    s["logits"] = _logits(g, rows, V, case["dtype"], case.get("spikes", 0))
    if kind == "greedy":
        s["sampler"] = lm.GreedySampler()
        return s
    if kind == "module":
        s["sampler"] = lm.StochasticSampler(temperature=case["temperature"], top_k=case["top_k"], top_p=case["top_p"], min_p=case["min_p"], seed=s["seed"])
        return s
    if kind == "mixed":
        knobs = dict(temperature=torch.rand(rows, generator=g, device=dev) * 1.2 + 0.3,
                     top_k=torch.tensor(MIX_TOP_K, dtype=torch.int32, device=dev)[torch.randint(0, len(MIX_TOP_K), (rows,), generator=g, device=dev)],
                     top_p=torch.rand(rows, generator=g, device=dev) * 0.2 + 0.8)
    else:
        knobs = {k: case[k] for k in ("temperature", "top_k", "top_p", "min_p")}
    hist = case.get("hist", 0)
    s["history"] = _history(g, rows, V, hist)
    s["uniforms"] = torch.rand(rows, generator=g, device=dev) if case.get("draw") == "inverse_cdf" else None
    s["params"] = lm.SamplingParams(seed=s["seed"], draw=case.get("draw", "gumbel"), repetition_penalty=RHO if hist else 1.0,
                                    presence_penalty=PI if hist else 0.0, **knobs)
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------------------

def run(state):
    kind = state["kind"]
    if kind in ("greedy", "module"):
        return state["sampler"].forward(state["logits"])
    if kind == "head":
        return lm.lm_head(state["hidden"], state["weight"], state["norm"])
    if kind == "verify":
        return lm.verify(state["target"], state["drafts"], state["probs"], state["u_accept"], state["u_final"], state["mode"],
                         temperature=state["temperature"], return_p_draft=True)
    if kind == "round":
        T, seed = state["temperature"], state["seed"]
        d = lm.draft_q(state["draft_logits"], temperature=T, seed=seed, step=1)
        t = lm.sample(state["target"], state["params"], step=1, return_tau=True, return_vmax=True)
        v = lm.verify(state["target"], d.tokens[: state["draft_logits"].shape[0]], None, state["u_accept"], state["u_final"], "stochastic", temperature=T,
                      tau=t.tau, draft_logits=state["draft_logits"], draft_stats=d, target_vmax=t.vmax, target_mass=t.mass)
        return {"drafts": d.tokens, "lse": d.lse, "q_vmax": d.vmax, "q_mass": d.mass, "target": t.tokens, "tau": t.tau, "vmax": t.vmax, "mass": t.mass,
                "accept": v[0], "final": v[1], "tokens": v[2]}
    if kind == "probs":
        r = lm.sample(state["logits"], state["params"], return_tau=True, return_stats=True, return_probs=True)
        return {"tokens": r.tokens, "tau": r.tau, "stats": r.stats, "probs": r.probs}
    r = lm.sample(state["logits"], state["params"], history=state["history"], uniforms=state["uniforms"], return_tau=True)
    return {"tokens": r.tokens, "tau": r.tau}


def work(case):
    """Every input read once, every output written once; a few operations per logit (an exponential, a compare, two sums)."""
    kind, V = case["kind"], case["vocab"]
    if kind == "head":
        r, H = case["rows"], case["hidden"]
        return {"bytes": 2.0 * (V * H + r * H + (H if case["norm"] else 0) + r * V), "flops": 2.0 * r * V * H}
    if kind in ("verify", "round"):
        n, width = case["n_draft"], 4 if case.get("dtype") == "fp32" else 2
        if kind == "round":                                                  # the drafter's and the target's rows, once each
            return {"bytes": float((2 * n + 1) * V * 2), "flops": 4.0 * (2 * n + 1) * V}
        if case["mode"] == "greedy":
            return {"bytes": float((n + 1) * V * width), "flops": 1.0 * (n + 1) * V}
        # every target row (its normaliser), one row of the drafter's probabilities (the residual) and the drafts' own entries of the others
        return {"bytes": float((n + 1) * V * width + V * 4), "flops": 4.0 * (n + 1) * V}
    rows, width = case["rows"], 2 if case["dtype"] == "bf16" else 4
    nbytes = rows * (V * width + 4 * case.get("hist", 0) + 20)
    if kind == "probs":
        nbytes += rows * V * 4
    return {"bytes": float(nbytes), "flops": (1.0 if kind == "greedy" else 4.0) * rows * V}


def tolerance(case):
    kind = case["kind"]
    if kind in ("greedy", "module"):
        return "exact"                                                       # token ids
    if kind == "head":
        return {"rel": 5e-3}                                                 # BF16 results of FP32 sums: half a unit in the last place is 2^-9
    return {"rel": 1e-5}                                                     # FP32 results of FP64 sums; token ids and integer masses the same
