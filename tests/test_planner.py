"""The native segment planner against a plain restatement of its rule (no pruning)."""

import heapq
import math
import random

import pytest


def _plan(bounds, heads, n_sm, min_chunks=8):
    chunks = [math.ceil((e - s) / 64) for s, e in zip(bounds[:-1], bounds[1:])]
    longest = max(chunks)
    if longest < 2 * min_chunks:
        return None

    def layout(limit):
        parts = [max(1, math.ceil(c / limit)) for c in chunks]
        per = [math.ceil(c / p) for c, p in zip(chunks, parts)]
        costs = [min(pc, c - i * pc) + 2 + (2 if i else 0)
                 for c, p, pc in zip(chunks, parts, per) for i in range(p) if c - i * pc > 0]
        loads = [0] * n_sm
        for c in sorted(costs, reverse=True):
            for _ in range(heads):
                heapq.heapreplace(loads, loads[0] + c)
        return parts, per, max(loads)

    limits = []
    for p in range(2, longest // min_chunks + 1):
        limit = math.ceil(longest / p)
        if limit >= min_chunks and limit not in limits:
            limits.append(limit)
    cands = [layout(limit) for limit in limits]
    if not cands or min(c[2] for c in cands) > 0.97 * layout(longest)[2]:
        return None
    parts, per, _ = next(c for c in cands if c[2] <= 1.03 * min(c[2] for c in cands))
    seg, begin = [], []
    for s, n, pc in zip(bounds[:-1], parts, per):
        begin.append(len(seg))
        seg += [s + i * pc * 64 for i in range(n)]
    return seg + [bounds[-1]], begin + [len(seg)]


@pytest.mark.parametrize("seed", range(12))
def test_native_planner_follows_its_rule(seed):
    from flashqla_b200.cp import split_sequences

    rng = random.Random(seed)
    heads = rng.choice([1, 2, 4, 8, 32])
    bounds = [0]
    for _ in range(rng.choice([1, 2, 7, 40])):
        bounds.append(bounds[-1] + rng.choice([0, 1, 63, 64, 65, rng.randint(1, 20000)]))
    assert split_sequences(bounds, heads, 148) == _plan(bounds, heads, 148)
