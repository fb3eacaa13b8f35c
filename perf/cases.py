"""The work a user of this framework has it do, as sized cases: chunked prefill (forward, no
gradients) and training (forward + backward) of the gated delta rule, through the public entry
points.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` makes what
a program holds before the call, ``run`` is one pass, ``work`` what the pass cannot do without and
``tolerance`` how far two correct implementations of the same precision may be apart.

A case is a dict of plain values:

``mode``       "prefill": forward with the final state, as a serving engine runs it;
               "train": forward, then the gradients of every differentiable input
``entry``      "op": ``chunk_gated_delta_rule``, what a model calls;
               "direct": ``chunk_gated_delta_rule_fwd`` / ``_bwd``, what a program with its own
               autograd (and the benchmark) calls
``batch``, ``tokens``  fixed-length input ``[batch, tokens]`` (``packed`` false)
``packed``     true: ``batch`` sequences behind one ``cu_seqlens``; ``tokens`` is then the total
``spread``     packed only: how uneven the lengths are, "uniform" (1 : 32) or "lognormal" (e^N(0,1))
``hq, hv``     query/key heads and value heads (hv a multiple of hq: grouped values)
``dim``        key and value dimension, 64 or 128
``dtype``      "bf16" or "fp16" (q, k, v);  ``beta``: "bf16" or "fp32"
``gate``       "logsigmoid": every head forgets within a chunk or two;
               "mixed": logsigmoid / 16, and every fourth head does not decay at all
``h0``         an initial state per sequence is passed in (a continued prompt)
``l2norm``     q and k are normalised by the operator;  ``v_first``: states as [V, K]
"""

import math
import random

import torch

from flash_qla import (
    chunk_gated_delta_rule,
    chunk_gated_delta_rule_bwd,
    chunk_gated_delta_rule_fwd,
)

_BASE = dict(mode="prefill", entry="op", batch=1, tokens=1024, packed=False, spread="uniform",
             hq=8, hv=8, dim=128, dtype="bf16", beta="bf16", gate="logsigmoid", h0=False,
             l2norm=False, v_first=False)


def _case(name, **over):
    assert set(over) <= set(_BASE)
    return dict(_BASE, name=name, **over)


def listed():
    return [
        # One short prompt, or the tail chunk of a longer one, on one tensor-parallel rank: the
        # smallest call, where latency and launches are all there is.
        _case("prefill_short", tokens=100, hq=2, hv=8, h0=True, l2norm=True),
        # A few short requests of a serving step with many grouped value heads, ragged lengths.
        _case("prefill_ragged_gva", batch=3, tokens=985, packed=True, hq=16, hv=64, h0=True,
              beta="fp32"),
        # A serving step of many short prompts, half precision inputs and the state layout some
        # engines keep.
        _case("prefill_fp16", batch=8, tokens=8192, packed=True, hq=2, hv=8, dtype="fp16",
              h0=True, l2norm=True, v_first=True),
        # A batched prefill of equal lengths: the default benchmark.
        _case("prefill_fixed", entry="direct", batch=4, tokens=8192, hq=16, hv=16),
        # Agent traffic: 64 packed prompts of very different lengths, all continued.
        _case("prefill_packed", batch=64, tokens=135161, packed=True, h0=True),
        # One long prompt on few heads, gates that partly never forget (the shape and the gates
        # of the reference benchmark's single-sequence row).
        _case("prefill_mixed_gate", tokens=32768, hq=2, hv=8, gate="mixed", h0=True,
              beta="fp32"),
        # Long context: one sequence of 262144 tokens.
        _case("prefill_long", tokens=262144),
        # The reference's CPU-sized configuration: head dimension 64, fp32 beta.
        _case("train_dim64", mode="train", tokens=512, hq=4, hv=4, dim=64, beta="fp32", h0=True),
        # A training micro-batch of one 4096-token sequence, grouped values, in-operator norm.
        _case("train_sequence", mode="train", tokens=4096, hq=2, hv=8, beta="fp32", l2norm=True),
        # A training micro-batch whose gates partly never forget, odd length.
        _case("train_mixed_gate", mode="train", batch=2, tokens=8111, hq=4, hv=8, gate="mixed"),
        # The training benchmark: 32768 tokens of packed documents, grouped values.
        _case("train_packed", mode="train", entry="direct", batch=23, tokens=32768, packed=True,
              spread="lognormal", hq=16, hv=32, h0=True),
        # Long-context training: the largest.
        _case("train_long", mode="train", tokens=262144),
    ]


_HEADS = [(1, 1), (1, 2), (2, 4), (4, 4), (2, 8), (4, 8), (8, 8), (4, 16), (16, 16), (16, 32),
          (32, 32), (16, 64)]


def draw(rng):
    """One more case of the listed ranges: 64 to 262144 tokens over their logarithm (odd totals
    as often as not), 1 to 64 value heads, every direction, data type and option."""
    c = dict(_BASE)
    c["mode"] = rng.choice(["prefill", "train"])
    c["entry"] = rng.choice(["op", "op", "direct"])
    c["dim"] = rng.choice([128, 128, 128, 64])
    c["gate"] = rng.choice(["logsigmoid", "logsigmoid", "mixed"])
    c["hq"], c["hv"] = rng.choice(_HEADS)
    # (token, value head) pairs of the largest listed case; the mixed gate and the narrow head
    # are listed (and used) at smaller sizes only
    pairs = 2_097_152
    if c["gate"] == "mixed":
        pairs //= 8
    if c["dim"] == 64:
        pairs //= 16
    most = min(262144, pairs // c["hv"])
    total = int(round(math.exp(rng.uniform(math.log(64), math.log(most)))))
    if total > 256 and rng.random() < 0.5:
        total -= total % 64
    shape = rng.choice(["one", "fixed", "packed"])
    if shape == "one":
        c["tokens"] = total
    elif shape == "fixed":
        c["batch"] = rng.randint(2, max(2, min(8, total // 64)))
        c["tokens"] = max(33, total // c["batch"])
    else:
        c["packed"] = True
        c["batch"] = rng.randint(2, max(2, min(64, total // 48)))
        c["tokens"] = max(total, 48 * c["batch"])
        c["spread"] = rng.choice(["uniform", "lognormal"])
    c["dtype"] = rng.choice(["bf16", "bf16", "bf16", "fp16"])
    c["beta"] = rng.choice(["bf16", "fp32"])
    c["h0"] = rng.random() < 0.5
    c["l2norm"] = c["entry"] == "op" and rng.random() < 0.5
    c["v_first"] = rng.random() < 0.25
    return c


def _lengths(case):
    """Sequence lengths of a packed case: a function of the case alone."""
    n, total = case["batch"], case["tokens"]
    rng = random.Random(1000003 * n + total)
    if case["spread"] == "uniform":
        share = [rng.uniform(1, 32) for _ in range(n)]
    else:
        share = [math.exp(max(-2.5, min(2.0, rng.gauss(0, 1)))) for _ in range(n)]
    whole = sum(share)
    lens = [max(1, int(total * s / whole)) for s in share]
    lens[lens.index(max(lens))] += total - sum(lens)
    return lens


def _sizes(case):
    """(rows B, rows T, number of sequences)"""
    if case["packed"]:
        return 1, case["tokens"], case["batch"]
    return case["batch"], case["tokens"], case["batch"]


def prepare(case, seed):
    B, T, N = _sizes(case)
    hq, hv, D = case["hq"], case["hv"], case["dim"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.bfloat16 if case["dtype"] == "bf16" else torch.float16

    def rn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    q, k = rn(B, T, hq, D), rn(B, T, hq, D)
    if not case["l2norm"]:
        q = torch.nn.functional.normalize(q, dim=-1)
        k = torch.nn.functional.normalize(k, dim=-1)
    s = dict(case=case, q=q.to(dtype), k=k.to(dtype), v=rn(B, T, hv, D).to(dtype))
    g = torch.nn.functional.logsigmoid(rn(B, T, hv))
    if case["gate"] == "mixed":
        g = g / 16
        g[:, :, 3::4] = 0.0
    s["g"] = g
    beta = torch.sigmoid(rn(B, T, hv))
    s["beta"] = beta if case["beta"] == "fp32" else beta.bfloat16()
    s["h0"] = 0.1 * rn(N, hv, D, D) if case["h0"] else None
    s["cu"] = None
    if case["packed"]:
        ends = [0]
        for n in _lengths(case):
            ends.append(ends[-1] + n)
        s["cu"] = torch.tensor(ends, dtype=torch.int32, device="cuda")
    if case["mode"] == "train":
        s["do"] = rn(B, T, hv, D).to(dtype)
        s["dht"] = 0.1 * rn(N, hv, D, D)
        if case["entry"] == "op":
            s["leaves"] = [s[n] for n in ("q", "k", "v", "g", "beta", "h0") if s[n] is not None]
            for t in s["leaves"]:
                t.requires_grad_(True)
    return s


def run(state):
    s, c = state, state["case"]
    if c["entry"] == "op":
        def forward():
            return chunk_gated_delta_rule(
                s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["h0"],
                output_final_state=True, use_qk_l2norm_in_kernel=c["l2norm"],
                cu_seqlens=s["cu"], state_v_first=c["v_first"])

        if c["mode"] == "prefill":
            with torch.no_grad():
                return forward()
        o, ht = forward()
        return (o.detach(), ht.detach()) + torch.autograd.grad((o, ht), s["leaves"],
                                                               (s["do"], s["dht"]))
    train = c["mode"] == "train"
    g_cum, A, o, _, ht, cache = chunk_gated_delta_rule_fwd(
        s["q"], s["k"], s["v"], s["g"], s["beta"], initial_state=s["h0"], cu_seqlens=s["cu"],
        output_final_state=True, state_v_first=c["v_first"], enable_fwd_cp_cache=train)
    if not train:
        return g_cum, A, o, ht
    grads = chunk_gated_delta_rule_bwd(
        s["q"], s["k"], s["v"], g_cum, s["beta"], A, s["do"], s["dht"], initial_state=s["h0"],
        cu_seqlens=s["cu"], state_v_first=c["v_first"], cp_cache=cache)
    return (g_cum, A, o, ht) + tuple(grads)


def work(case):
    """Every input once and every output once; the products of the chunked form (chunk 64): per
    (token, value head) four of 64 x dim and three of dim x dim forward, three times that again
    for the gradients."""
    B, T, N = _sizes(case)
    rows, hq, hv, D = B * T, case["hq"], case["hv"], case["dim"]
    gate_bytes = rows * hv * (4 + (4 if case["beta"] == "fp32" else 2))
    state_bytes = 4 * N * hv * D * D
    qk, val = 2 * rows * hq * D * 2, rows * hv * D * 2
    n_bytes = qk + val + gate_bytes + (state_bytes if case["h0"] else 0) + val + state_bytes
    flops = rows * hv * (8 * 64 * D + 6 * D * D)
    if case["entry"] == "direct":
        n_bytes += rows * hv * (4 + 2 * 64)  # the cumulative gate and A come back too
    if case["mode"] == "train":
        n_bytes += val + state_bytes  # gradients of the outputs
        n_bytes += qk + val + gate_bytes + (state_bytes if case["h0"] else 0)
        flops *= 4
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case):
    """bf16 operands and a bf16 copy of the state in every product (fp32 accumulation): two
    correct implementations, each a few 1e-3 off the exact result, differ by up to 1e-2."""
    return {"rel": 1e-2, "max": 0.4}
