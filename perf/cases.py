"""The sampling calls whose time matters to a user of this package.

`listed()` names twelve of them and says what each stands for, `draw(rng)` gives further ones from the same ranges,
`prepare(case, seed)` makes what a decode loop has on the GPU before the call, `run(state)` is one call through the
package's public functions, `work(case)` the bytes it cannot do without and `tolerance(case)` how far another correct
implementation's results may lie from this one's.

A case is a dict:

  call     "plain"       batch_sampling_temperature_topk_topp(_any)
           "penalties"   batch_sampling_repetition_temperature_topk_topp(_any)
           "rows"        batch_sampling_rows: temperature / top_k / top_p of every row in tensors
           "vocab"       VocabParallelSampler.sample, the local part of a vocab-parallel group
  B, T, V  rows, positions per row (only the last one is sampled), vocabulary; V is a multiple of 4
  dtype    "f32", "f16" or "bf16" logits
  dist     "uniform"     U[0, 1): a flat row, nearly everything is kept below top_p
           "normal"      N(0, sigma^2)
           "peaked"      N(0, 2^2) with 32 ids per row raised by 10: a confident model
           "boosted"     N(0, 1) with 1 % of the ids raised by 8: a wide head over a long tail
  temperature, top_k, top_p, presence, repetition, decay   as the calls take them
  penalised, with_prob   "rows" only: with a penalties tensor; with the id's probability and the kept mass returned
"""
import math

import torch

import rapid_sampling_b200 as sampler
from rapid_sampling_b200.vocab_parallel import VocabParallelSampler

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}

# ranges of draw(): the smallest and largest batch and vocabulary of the package's own sweep, and the largest row the
# calls take; B * V stays within the largest listed case's
B_MAX = 512
V_MIN, V_MAX = 256, 1048576
ELEMENTS_MAX = 256 * 151936


def _case(name, call, B, V, dist, **more):
    c = dict(name=name, call=call, B=B, T=1, V=V, dtype="f32", dist=dist, temperature=1.0, top_k=-1, top_p=1.0)
    if dist == "normal":
        c["sigma"] = 3.0
    if call in ("penalties", "rows"):
        c.update(presence=0.1, repetition=0.1, decay=0.95)
    if call == "rows":
        c.update(penalised=True, with_prob=True)
    c.update(more)
    return c


def listed():
    return [
        # a byte-level vocabulary, one stream: nothing but the latency of a call
        _case("bytes_b1", "plain", 1, 256, "normal", top_p=0.9),
        # one chat stream with a large vocabulary and a tight nucleus: the package's headline workload
        _case("single_stream", "plain", 1, 262144, "normal", top_p=0.3),
        # the README example: four flat rows, so that half of the vocabulary is kept
        _case("flat_b4", "plain", 4, 131072, "uniform", top_p=0.5),
        # a few streams with repetition penalties and an odd batch: interactive decoding
        _case("penalties_b7", "penalties", 7, 100256, "peaked", temperature=0.7, top_k=40, top_p=0.9),
        # batched serving, one setting for all rows
        _case("serving_b64", "plain", 64, 151936, "peaked", temperature=0.8, top_k=50, top_p=0.9),
        # batched serving where every request brings its own setting, bf16 logits straight from the head, log-probabilities on
        _case("mixed_requests", "rows", 48, 151936, "peaked", dtype="bf16"),
        # plain nucleus sampling of a full batch, no top-k: kept sets of thousands of ids
        _case("nucleus_b128", "plain", 128, 50304, "normal", top_p=0.9),
        # a large batch of bf16 logits whose rows are no multiple of a stripe
        _case("bf16_b160", "plain", 160, 100256, "normal", sigma=2.5, dtype="bf16", temperature=0.7, top_k=100, top_p=0.95),
        # large-batch decoding with in-place penalties: the most bytes per call
        _case("penalties_b256", "penalties", 256, 65536, "normal", sigma=2.5, temperature=0.8, top_k=50, top_p=0.9),
        # rollouts for training: a large batch at temperature 1 with no cutoff at all
        _case("rollout_b256", "plain", 256, 151936, "peaked"),
        # the longest row the calls take, sampled from the last of four positions
        _case("longest_rows", "plain", 32, 1048576, "boosted", T=4, top_p=0.95),
        # one rank's columns of a vocabulary split over eight GPUs
        _case("vocab_shard", "vocab", 32, 131072, "boosted", top_p=0.95),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    call = rng.choices(["plain", "penalties", "rows", "vocab"], [9, 5, 3, 1])[0]
    B = max(1, min(B_MAX, round(_log_uniform(rng, 1, B_MAX))))
    elements = ELEMENTS_MAX if call == "plain" else 256 * 65536      # the penalties travel beside the logits, twice
    lo, hi = V_MIN, min(V_MAX, elements // B)
    if call == "vocab":                      # an eighth to a half of a language model's vocabulary
        lo, hi = 4096, min(hi, 131072)
    V = 4 * (int(_log_uniform(rng, lo, hi)) // 4)
    T = rng.randint(2, 4) if call == "plain" and rng.random() < 0.2 else 1
    dist = rng.choices(["peaked", "normal", "boosted", "uniform"], [4, 4, 1, 0 if call == "vocab" else 1])[0]
    dtype = "f32" if call == "vocab" else rng.choices(["f32", "bf16", "f16"], [6, 3, 1])[0]
    more = {"T": T, "dtype": dtype}
    if dist == "normal":
        more["sigma"] = rng.choice([2.0, 2.5, 3.0])
    if call == "rows":
        more.update(penalised=rng.random() < 0.5, with_prob=rng.random() < 0.5)
    else:
        style = rng.choices(["both", "nucleus", "top_k", "none"], [4, 3, 1, 1])[0]
        more["temperature"] = rng.choice([1.0, 1.0, 0.6, 0.7, 0.8, 1.2])
        if style in ("both", "top_k"):
            more["top_k"] = rng.choice([1, 10, 20, 40, 50, 50, 100, 200, 1000])
        if style in ("both", "nucleus"):
            more["top_p"] = rng.choice([0.3, 0.5, 0.8, 0.9, 0.9, 0.95])
    c = _case("", call, B, V, dist, **more)
    del c["name"]
    return c


def _logits(case, gen):
    B, T, V = case["B"], case["T"], case["V"]
    shape = (B, T, V) if T > 1 else (B, V)
    dist = case["dist"]
    if dist == "uniform":
        x = torch.rand(shape, generator=gen, device="cuda")
    else:
        x = torch.randn(shape, generator=gen, device="cuda")
        if dist == "normal":
            x *= case["sigma"]
        elif dist == "peaked":
            x *= 2
            ids = torch.randint(0, V, shape[:-1] + (32,), generator=gen, device="cuda")
            x.scatter_add_(-1, ids, torch.full_like(ids, 10, dtype=x.dtype))
        elif dist == "boosted":
            ids = torch.randint(0, V, shape[:-1] + (max(1, V // 100),), generator=gen, device="cuda")
            x.scatter_add_(-1, ids, torch.full_like(ids, 8, dtype=x.dtype))
    return x.to(DTYPES[case["dtype"]])


def prepare(case, seed):
    """Logits, the rows' random states, and what the call needs besides: a penalties tensor as some hundred tokens of
    context leave it, the rows' parameters, or the vocab-parallel sampler."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, V = case["B"], case["V"]
    s = {"case": case, "logits": _logits(case, gen), "states": sampler.setup_rand(seed, B)}
    if case["call"] == "penalties" or case.get("penalised"):
        seen = torch.randint(0, V, (B, 200), generator=gen, device="cuda")
        value = torch.rand((B, 200), generator=gen, device="cuda") * 0.5
        s["penalties"] = torch.zeros((B, V), device="cuda").scatter_reduce_(1, seen, value, "amax")
    if case["call"] == "rows":
        def pick(values, dtype):
            at = torch.randint(0, len(values), (B,), generator=gen, device="cuda")
            return torch.tensor(values, dtype=dtype, device="cuda")[at].contiguous()
        s["temperature"] = pick([1.0, 0.6, 0.7, 0.8, 0.9, 1.2], torch.float32)
        s["top_k"] = pick([-1, 20, 40, 50, 100], torch.int32)
        s["top_p"] = pick([1.0, 0.8, 0.9, 0.95], torch.float32)
    if case["call"] == "vocab":
        s["plan"] = VocabParallelSampler(B, V, rank=0, world=1)
    return s


def run(state):
    c, logits, states = state["case"], state["logits"], state["states"]
    call = c["call"]
    if call == "plain":
        f = sampler.batch_sampling_temperature_topk_topp if c["dtype"] == "f32" else sampler.batch_sampling_temperature_topk_topp_any
        return f(logits, states, c["temperature"], c["top_k"], c["top_p"]), states
    if call == "penalties":
        f = (sampler.batch_sampling_repetition_temperature_topk_topp if c["dtype"] == "f32"
             else sampler.batch_sampling_repetition_temperature_topk_topp_any)
        penalties = state["penalties"]
        ids = f(logits, penalties, states, c["presence"], c["repetition"], c["decay"], c["temperature"], c["top_k"], c["top_p"])
        return ids, states, penalties
    if call == "rows":
        penalties = state.get("penalties")
        got = sampler.batch_sampling_rows(logits, states, state["temperature"], state["top_k"], state["top_p"], penalties,
                                          c["presence"], c["repetition"], c["decay"], c["with_prob"])
        return got, states, penalties
    return state["plan"].sample(logits, states, c["temperature"], c["top_k"], c["top_p"]), states


def work(case):
    """The last position's logits read once, the penalties read and written once, every row's random state (64 bytes)
    read and written and its id written; with per-row parameters 12 bytes of them and, if asked for, two more results.
    Arithmetic: the scaling, the exponential and its sum per logit, the penalty's subtraction and decay."""
    B, V = case["B"], case["V"]
    penalised = case["call"] == "penalties" or case.get("penalised", False)
    size = 4 if case["dtype"] == "f32" else 2
    per_row = V * size + (8 * V if penalised else 0) + 2 * 64 + 4
    if case["call"] == "rows":
        per_row += 12 + (8 if case["with_prob"] else 0)
    return {"bytes": B * per_row, "flops": B * V * (5 if penalised else 3)}


def tolerance(case):
    """Ids and random states are whole numbers fixed by the draw and by the order in which this sampler defines its fp32
    sums, and a penalty is one fused multiply-add: all exact.  The returned probability and kept mass are fp32 values."""
    if case["call"] == "rows" and case["with_prob"]:
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0}
    return "exact"
