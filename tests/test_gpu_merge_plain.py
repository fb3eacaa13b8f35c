"""Merge chains that apply no transition matrix are copies of the local states: they come out exact, beside
pairs that do apply some, whatever the flag of the segment at the end of a chain (never read) holds."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pad", [0, 1], ids=["aligned", "odd_stride"])
@pytest.mark.parametrize("reverse", [False, True], ids=["forward", "reverse"])
@pytest.mark.parametrize("D,Hv,counts", [(128, 3, [9, 1, 0, 300]), (64, 5, [4, 0, 2]), (128, 8, [9])])
@pytest.mark.parametrize("with_raw", [True, False])
def test_pairs_without_m(D, Hv, counts, reverse, pad, with_raw):
    from flashqla_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(D + Hv)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    n_seg, n = sum(counts), Hv * D * D
    begin = [sum(counts[:i]) for i in range(len(counts) + 1)]
    rec = torch.full((n_seg, 2 * n + Hv + pad), float("nan"), device="cuda")
    local, M = rec[:, :n].unflatten(1, (Hv, D, D)), rec[:, n:2 * n].unflatten(1, (Hv, D, D))
    use = rec[:, 2 * n:2 * n + Hv].view(torch.int32)
    local.copy_(rn(n_seg, Hv, D, D))
    use.zero_()
    chained = []  # (sequence, head) pairs that apply M once, in the middle or at an edge of the chain
    for r, c in enumerate(counts):
        if c > 1:
            last = begin[r] if reverse else begin[r + 1] - 1
            use[last] = 1  # the flags of the segment that hands nothing on
            local[last].fill_(float("nan"))
            at = begin[r] + (c // 2 if c // 2 + begin[r] != last else c // 2 - 1)
            use[at, r % Hv] = 1
            M[at, r % Hv] = 0.05 * rn(D, D)
            chained.append((r, r % Hv))
    raw = rn(len(counts), Hv, D, D) if with_raw else None
    out = ops.merge_states(local, M, use, raw, torch.tensor(begin, dtype=torch.int32, device="cuda"),
                           reverse=reverse)
    for r in range(len(counts)):
        idx = list(range(begin[r], begin[r + 1]))[::-1 if reverse else 1]
        for hv in range(Hv):
            cur = raw[r, hv].double() if with_raw else torch.zeros(D, D, device="cuda", dtype=torch.float64)
            for i in idx:
                if (r, hv) in chained:
                    assert (out[i, hv].double() - cur).norm() <= 1e-5 * cur.norm(), (r, hv, i)
                else:
                    assert torch.equal(out[i, hv].double(), cur), (r, hv, i)
                cur, prev = local[i, hv].double(), cur
                if use[i, hv] and i != idx[-1]:
                    m = M[i, hv].double()
                    cur = cur + (m.T if reverse else m) @ prev
