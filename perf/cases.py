"""The work a user of this framework has it do, as timed cases over its public entry points.

``flash_attn_func`` and ``flash_attn_padded_func`` are called the way a model calls them: a forward
without gradients for inference, a forward and a backward through autograd for training.  Sizes are
the workloads of ``bench.py`` and of ``tests/`` or of the same ranges; inputs are N(0, 1) like theirs.

A case has:
  mode       "infer" (forward under no_grad) or "train" (forward, then dq, dk, dv)
  z h n d    batch, heads, query rows, head dimension; nk = keys (n unless it is cross-attention)
  dtype      "fp16" or "bf16"
  causal     the ordinary causal mask
  packed     q, k, v are views of one (z, n, 3, h, d) projection output
  padded     right-padded batch: real lengths spread evenly over [n/8, n] (see ``_lengths``)
  det        deterministic dQ (an option of ``flash_attn_padded_func``)
"""
import os
import sys

import torch

_PKG = os.path.abspath("flash-attention-v100_b200")  # of the working folder
if _PKG not in sys.path:
    sys.path.insert(1, _PKG)

from flash_attn_v100.flash_attn_interface import flash_attn_func, flash_attn_padded_func  # noqa: E402

_DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _case(mode, z, h, n, d, dtype, causal, nk=None, packed=False, padded=False, det=False):
    return {"mode": mode, "z": z, "h": h, "n": n, "nk": n if nk is None else nk, "d": d, "dtype": dtype,
            "causal": causal, "packed": packed, "padded": padded, "det": det}


def listed():
    cases = {
        # a unit-test-sized training step: nothing but launches and host work
        "train_tiny": _case("train", 2, 4, 128, 64, "fp16", False),
        # a short prompt through one layer of a model: latency of one forward
        "infer_short": _case("infer", 1, 16, 160, 128, "bf16", True, packed=True),
        # training of a small language model, one layer (bench: cfg2)
        "train_small_d64": _case("train", 4, 16, 1024, 64, "fp16", True),
        # training of an encoder on many short sequences (bench: cfg4, the whole batch)
        "train_encoder_d64": _case("train", 64, 16, 512, 64, "bf16", False),
        # the workload the headline figure is quoted on (bench: cfg3)
        "train_d128_causal": _case("train", 8, 32, 2048, 128, "fp16", True),
        # the same without a mask, bf16 (bidirectional training)
        "train_d128_full": _case("train", 8, 32, 2048, 128, "bf16", False),
        # head dimension 96 (bench: cfg3's shape at 96)
        "train_d96_causal": _case("train", 8, 32, 2048, 96, "fp16", True),
        # prefill of a batch of prompts, length not a multiple of any tile (bench: cfg3 ragged)
        "infer_ragged": _case("infer", 8, 32, 2016, 128, "bf16", True, packed=True),
        # a batch of unequal documents padded to the longest: padding has to be skipped
        "train_padded": _case("train", 8, 16, 2048, 128, "bf16", True, padded=True),
        # reproducible training
        "train_deterministic": _case("train", 2, 16, 2048, 128, "bf16", True, det=True),
        # few queries over a long context (cross-attention, a late chunk of a prompt)
        "infer_few_queries": _case("infer", 2, 32, 64, 128, "bf16", False, nk=8192),
        # long-context training on one GPU (bench: cfg5)
        "train_long": _case("train", 1, 32, 32768, 128, "fp16", True),
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _mult32(rng, lo, hi):
    """A multiple of 32 in [lo, hi], spread over the logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random() / 32.0)) * 32))


def draw(rng):
    while True:
        mode = "train" if rng.random() < 0.6 else "infer"
        d = rng.choice((64, 96, 128, 128))
        dtype = rng.choice(("fp16", "bf16"))
        h = rng.choice((1, 4, 5, 8, 12, 16, 16, 32, 32, 40))
        z = max(1, int(round(64 ** rng.random())))
        n = _mult32(rng, 32, 32768)
        causal = rng.random() < 0.6
        what = rng.random()
        if what < 0.15:  # cross-attention: few or many queries over another sequence
            c = _case(mode, z, h, n, d, dtype, False, nk=_mult32(rng, 32, 32768))
        elif what < 0.30:
            c = _case(mode, max(2, z), h, n, d, dtype, causal, padded=True)
        elif what < 0.40:
            c = _case("train", z, h, n, d, dtype, causal, det=True)
        else:
            c = _case(mode, z, h, n, d, dtype, causal, packed=rng.random() < 0.35)
        most = _case("train", 1, 32, 32768, 128, "fp16", True)
        w, m = work(c), work(most)
        # (the deterministic mode runs at a fraction of the rate)
        if w["flops"] * (4 if c["det"] else 1) <= m["flops"] and w["bytes"] <= m["bytes"]:
            return c


def _lengths(n, z):
    """Real lengths of a padded batch: even steps from n/8 to n (the longest one is the padded
    length), odd ones among them; the same set for every seed, in another order."""
    lo = max(1, n // 8)
    return [lo + (n - lo) * i // max(1, z - 1) for i in range(z)]


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    z, h, n, nk, d = case["z"], case["h"], case["n"], case["nk"], case["d"]
    opts = {"generator": g, "device": "cuda", "dtype": _DTYPES[case["dtype"]]}
    if case["packed"]:
        q, k, v = torch.randn((z, n, 3, h, d), **opts).unbind(2)
    else:
        q = torch.randn((z, n, h, d), **opts)
        k, v = torch.randn((z, nk, h, d), **opts), torch.randn((z, nk, h, d), **opts)
    state = {"causal": case["causal"], "det": case["det"], "lengths": None, "dout": None}
    if case["padded"]:
        cpu = torch.Generator()
        cpu.manual_seed(int(seed))
        order = torch.randperm(z, generator=cpu).tolist()
        lengths = _lengths(n, z)
        state["lengths"] = torch.tensor([lengths[i] for i in order], dtype=torch.int32, device="cuda")
    if case["mode"] == "train":
        q, k, v = (t.detach().requires_grad_() for t in (q, k, v))
        state["dout"] = torch.randn((z, n, h, d), **opts)
    state["qkv"] = (q, k, v)
    return state


def _attention(state):
    q, k, v = state["qkv"]
    if state["lengths"] is not None or state["det"]:
        return flash_attn_padded_func(q, k, v, state["lengths"], state["lengths"], causal=state["causal"],
                                      deterministic=state["det"])
    return flash_attn_func(q, k, v, causal=state["causal"])


def run(state):
    if state["dout"] is None:
        with torch.no_grad():
            return _attention(state)
    out = _attention(state)
    dq, dk, dv = torch.autograd.grad(out, state["qkv"], state["dout"])
    return out, dq, dk, dv


def work(case):
    """Forward: two products over every visible (query, key) pair, backward: five.  q, k, v (and
    dout) are read once, o (and dq, dk, dv) written once; of a padded batch the real rows are read
    and all rows are written."""
    z, h, n, nk, d = case["z"], case["h"], case["n"], case["nk"], case["d"]
    train = case["mode"] == "train"
    lens = _lengths(n, z) if case["padded"] else None
    pairs = sum(x * x for x in lens) if lens else z * n * nk
    flops = (14.0 if train else 4.0) * h * d * pairs * (0.5 if case["causal"] else 1.0)
    rows_q, rows_k = (sum(lens),) * 2 if lens else (z * n, z * nk)
    read = rows_q + 2 * rows_k + (rows_q if train else 0)
    written = z * n + (z * n + 2 * z * nk if train else 0)
    return {"bytes": 2.0 * h * d * (read + written), "flops": flops}


def tolerance(case):
    # P, dS and the results are rounded to the 16-bit type on the way (relative rounding 2^-12 for
    # fp16, 2^-9 for bf16 on average), sums are fp32
    return {"rel": 3e-3 if case["dtype"] == "fp16" else 1e-2}
