"""The work that users of this package have it do, as a list of cases that can be timed and compared.

A case is one pass through a public entry point:

  train      fastmax_custom forward + backward through autograd (the attention call of a training step)
  infer      fastmax_custom forward only, no gradient recorded
  boundary   FASTMultiHeadAttention_Function forward + backward: the float32 boundary the reference's model file calls
  prefill    FastmaxDecoder.prefill of a prompt: causal attention that leaves the moment state behind
  decode     FastmaxDecoder.step: one new token per (batch, head)

Shapes are those of this repository's benchmark, tests and configurations, and the range around them.  Scores are
q.k / temperature with temperature = 8 sqrt(d), or 1 where q and k are normalised (the reference's convention);
a0 = a1 = 1, a2 = 1/2.
"""
import math

import torch

from reproducing_fastmax_results_b200 import FASTMultiHeadAttention_Function, fastmax_custom
from reproducing_fastmax_results_b200.decoding import FastmaxDecoder


def _case(kind, batch, heads, n, d, dtype, order=2, causal=True, normalize=False, split=False, nk=0, scale=1.0):
    return {"kind": kind, "batch": batch, "heads": heads, "n": n, "nk": nk or n, "d": d, "dtype": dtype,
            "order": order, "causal": causal, "normalize": normalize, "split": split, "scale": scale}


def _named(name, *shape, **options):
    return {"name": name, **_case(*shape, **options)}


def listed():
    return [
        # generating text for one user: one token through eight heads, nothing but latency
        _named("decode_one_user", "decode", 1, 8, 1, 64, "bf16"),
        # serving a batch of users, one token each (the benchmark's decoding workload)
        _named("decode_batch", "decode", 32, 16, 1, 64, "bf16"),
        # reading a few prompts of no round length before decoding
        _named("prefill_ragged", "prefill", 4, 16, 1999, 64, "bf16"),
        # the smallest training call: the configuration that a CPU can run, float32, no mask
        _named("train_small_f32", "train", 2, 4, 256, 32, "f32", causal=False),
        # the attention of the reference's transformer as its model file calls it: float32, normalised, (n, b*h, d) copies
        _named("boundary_model_f32", "boundary", 16, 8, 1024, 64, "f32", normalize=True),
        # the same block under bf16 autocast: head-split views, normalised q and k, gradient through the normalisation
        _named("train_model_bf16", "train", 16, 8, 1024, 64, "bf16", normalize=True, split=True),
        # the headline benchmark: a training step of long sequences
        _named("train_headline_bf16", "train", 8, 16, 4096, 64, "bf16"),
        # an encoder over patches and a class token: no mask, odd length, contiguous heads
        _named("train_encoder_bf16", "train", 16, 12, 577, 64, "bf16", causal=False),
        # narrow heads in bf16
        _named("train_narrow_bf16", "train", 8, 16, 2048, 32, "bf16", split=True),
        # order 1, wide batch, forward only: the memory-bound configuration
        _named("infer_order1_wide", "infer", 64, 12, 1024, 64, "bf16", order=1, causal=False, scale=0.5),
        # one very long sequence in bf16 with few heads
        _named("train_long_bf16", "train", 1, 8, 131072, 64, "bf16"),
        # one very long sequence in float32 (the configuration that is split over GPUs; here all of it on one)
        _named("train_long_f32", "train", 1, 8, 131072, 32, "f32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "train", "infer", "infer", "boundary", "prefill", "decode"])
    d = rng.choice([64, 64, 64, 32, 32, 16])
    if kind == "decode":
        heads = rng.choice([4, 6, 8, 12, 16])
        return _case(kind, _log_int(rng, 1, 512 // heads), heads, 1, d, rng.choice(["bf16", "bf16", "f32"]),
                     order=rng.choice([2, 2, 2, 1]))
    dtype = "f32" if kind == "boundary" else rng.choice(["bf16", "bf16", "bf16", "f32"])
    causal = kind == "prefill" or rng.random() < 0.7
    heads = rng.choice([4, 6, 8, 12, 16, 20])
    # lengths from a short sentence to a long document; the batch is what fits beside them in a step
    n = _log_int(rng, 64, 16384)
    room = (8 * 16 * 4096 if dtype == "bf16" else 16 * 8 * 1024) // (heads * n)
    batch = _log_int(rng, 1, max(1, min(64, room)))
    nk = n if causal or rng.random() < 0.6 else _log_int(rng, 64, 4096)   # cross attention where there is no mask
    order = 1 if rng.random() < 0.2 else 2
    normalize = kind in ("train", "boundary") and rng.random() < 0.4
    return _case(kind, batch, heads, n, d, dtype, order=order, causal=causal, normalize=normalize,
                 split=kind in ("train", "infer") and rng.random() < 0.5, nk=nk)


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bf16" else torch.float32


def _temperature(case):
    return 1.0 if case["normalize"] else 8.0 * math.sqrt(case["d"])


def _tensor(case, n, gen):
    b, h, d = case["batch"], case["heads"], case["d"]
    if case["split"]:   # what a projection leaves: (b, n, h*d), seen as (b, h, n, d)
        x = torch.randn(b, n, h, d, device="cuda", generator=gen).mul_(case["scale"])
        return x.to(_dtype(case)).transpose(1, 2)
    return torch.randn(b, h, n, d, device="cuda", generator=gen).mul_(case["scale"]).to(_dtype(case))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if case["kind"] == "decode":
        # the state of a prompt that was read before; a fresh token for every step
        dec = FastmaxDecoder(case["batch"], case["heads"], case["d"], p=case["order"], temperature=_temperature(case))
        prompt = dict(case, split=False)
        q, k, v = (_tensor(prompt, 128, gen) for _ in range(3))
        dec.prefill(q, k, v)
        state["decoder"] = dec
        state["q"], state["k"], state["v"] = (_tensor(prompt, 1, gen)[:, :, 0] for _ in range(3))
        return state
    n, nk = case["n"], case["nk"]
    state["q"], state["k"], state["v"] = _tensor(case, n, gen), _tensor(case, nk, gen), _tensor(case, nk, gen)
    if case["kind"] == "prefill":
        state["decoder"] = FastmaxDecoder(case["batch"], case["heads"], case["d"], p=case["order"],
                                          temperature=_temperature(case))
    if case["kind"] in ("train", "boundary"):
        for name in ("q", "k", "v"):
            state[name].requires_grad_(True)
        state["do"] = _tensor(case, n, gen)
    if case["kind"] == "boundary":
        # what transformer/model.py hands over and the operator ignores
        state["noise"] = torch.zeros_like(state["q"])
        state["rpe"] = torch.zeros(2 * nk - 1, case["d"], device="cuda")
    return state


def run(state):
    case = state["case"]
    kind, q, k, v = case["kind"], state["q"], state["k"], state["v"]
    if kind == "decode":
        return {"o": state["decoder"].step(q, k, v), "state": state["decoder"].state}
    if kind == "prefill":
        state["decoder"].reset()
        o = state["decoder"].prefill(q, k, v)
        return {"o": o, "state": state["decoder"].state}
    options = (case["causal"], 0.0, case["normalize"], _temperature(case), 1.0, 1.0, 0.5, 1.0, case["order"])
    if kind == "infer":
        with torch.no_grad():
            return fastmax_custom(q, k, v, None, None, *options)
    if kind == "boundary":
        o = FASTMultiHeadAttention_Function.apply(q, k, v, state["noise"], state["rpe"], *options)
    else:
        o = fastmax_custom(q, k, v, None, None, *options)
    dq, dk, dv = torch.autograd.grad(o, (q, k, v), state["do"])
    return {"o": o.detach(), "dq": dq, "dk": dk, "dv": dv}


def _features(case):
    d = case["d"]
    return (d * (d + 1) // 2 if case["order"] == 2 else 0) + d + 1


def work(case):
    """Bytes: every input once, every output once.  Operations: the cheaper of the two ways to evaluate the sums, over
    pairs of tokens (4 d per visible pair forward, 10 d more backward) or over moments (feature x value products:
    build and apply forward, twice that backward)."""
    bh, n, nk, d = case["batch"] * case["heads"], case["n"], case["nk"], case["d"]
    size = 2 if case["dtype"] == "bf16" else 4
    m = _features(case)
    state = bh * m * (d + 1) * 4
    if case["kind"] == "decode":
        return {"bytes": 2 * state + 4 * bh * d * size, "flops": 4.0 * bh * m * (d + 1)}
    pairs = n * (n + 1) / 2 if case["causal"] else n * nk
    moments = 2.0 * bh * (n + nk) * m * (d + 1)
    io = bh * (2 * n + 2 * nk) * d * size
    if case["kind"] == "prefill":   # the state has to come out, so the keys' moments are built in any case
        return {"bytes": io + state, "flops": min(4.0 * d * bh * pairs, moments / 2) + moments / 2}
    flops = min(4.0 * d * bh * pairs, moments)
    if case["kind"] in ("train", "boundary"):
        io += bh * (2 * n + 2 * nk) * d * size
        flops += min(10.0 * d * bh * pairs, 2 * moments)
    return {"bytes": io, "flops": flops}


def tolerance(case):
    """bf16: operands and results are rounded to 8 bits.  float32: sums of up to 131072 terms in 32 bits, in any order.
    Single values are measured against the root mean square of their tensor, and in a causal call the gradients of the
    first few tokens are a hundred times that (their denominators have few terms), with bf16 errors to match: against
    float64, single values of dq are off by up to 0.9 of the tensor's root mean square at 131072 tokens."""
    if case["kind"] == "decode":   # the state is float32 and is added to in place
        return {"rel": 1e-2 if case["dtype"] == "bf16" else 1e-5}
    return {"rel": 1e-2, "max": 0.9} if case["dtype"] == "bf16" else {"rel": 1e-5, "max": 1e-3}
