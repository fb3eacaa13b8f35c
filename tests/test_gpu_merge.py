"""The merge chain against a float64 host chain: both head dimensions, chains of one segment up to
more than the kernel's three buffers, more (sequence, head) pairs than it has rows of CTAs, entries
at 16-byte and at 4-byte alignment, pairs with and without a chain; and states kept as [V, K].

Bound: a chain of s steps is s fp32 sums of at most 128 products with the matrices' norm below 1
here, each in any order: 128 * 2^-24 * s < 1e-4 at s = 9."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pad", [0, 1], ids=["aligned", "odd_stride"])
@pytest.mark.parametrize("reverse", [False, True], ids=["forward", "reverse"])
@pytest.mark.parametrize("D,Hv,counts", [(128, 3, [9, 1, 0, 4]), (128, 23, [2, 3]), (64, 5, [4, 0, 9]),
                                         (64, 40, [3, 1])])
@pytest.mark.parametrize("flags", ["none", "some"])
def test_chain(D, Hv, counts, reverse, pad, flags):
    from flashqla_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(D + Hv)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    n_seg, n = sum(counts), Hv * D * D
    begin = [sum(counts[:i]) for i in range(len(counts) + 1)]
    rec = torch.full((n_seg, 2 * n + Hv + pad), float("nan"), device="cuda")
    local, M = rec[:, :n].unflatten(1, (Hv, D, D)), rec[:, n:2 * n].unflatten(1, (Hv, D, D))
    local.copy_(rn(n_seg, Hv, D, D))
    M.copy_(rn(n_seg, Hv, D, D) * 0.05)
    use = rec[:, 2 * n:2 * n + Hv].view(torch.int32)
    use.copy_((rn(n_seg, Hv) > -0.5).int())
    raw = rn(len(counts), Hv, D, D)
    chained = (rn(len(counts), Hv) > 0).int() if flags == "some" else None
    out = ops.merge_states(local, M, use, raw, torch.tensor(begin, dtype=torch.int32, device="cuda"),
                           reverse=reverse, any_fallback=chained)
    for r in range(len(counts)):
        idx = list(range(begin[r], begin[r + 1]))
        cur = raw[r].double()
        for j, i in enumerate(idx[::-1] if reverse else idx):
            heads = slice(None) if chained is None or j == 0 else chained[r].bool()
            err = (out[i][heads].double() - cur[heads]).norm() / cur[heads].norm().clamp_min(1e-30)
            assert err < 1e-4, (r, i)
            m = M[i].double().transpose(-1, -2) if reverse else M[i].double()
            cur = local[i].double() + use[i].view(Hv, 1, 1) * (m @ cur)


def test_states_kept_value_first_through_a_split_sequence():
    """A gate that never forgets makes every segment take its start state from the chain."""
    from flash_qla import chunk_gated_delta_rule

    gen = torch.Generator(device="cuda").manual_seed(5)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    unit = torch.nn.functional.normalize
    q, k = (unit(rn(1, 8192 + 17, 2, 128), dim=-1).bfloat16() for _ in range(2))
    v, beta = rn(1, 8192 + 17, 4, 128).bfloat16(), torch.sigmoid(rn(1, 8192 + 17, 4))
    g = torch.nn.functional.logsigmoid(rn(1, 8192 + 17, 4)) / 16
    g[..., 1::2] = 0.0
    h0, dht = rn(1, 4, 128, 128), rn(1, 4, 128, 128)
    do = rn(*v.shape).bfloat16()
    got = []
    for v_first in (False, True):
        x = [t.clone().requires_grad_() for t in (q, k, v, g, beta)]
        s = (h0.transpose(-1, -2).contiguous() if v_first else h0.clone()).requires_grad_()
        o, ht = chunk_gated_delta_rule(*x, initial_state=s, output_final_state=True, state_v_first=v_first)
        grads = torch.autograd.grad((o, ht), x + [s], (do, dht.transpose(-1, -2) if v_first else dht))
        states = [ht, grads[-1]]
        got.append([o, *grads[:-1]] + [t.transpose(-1, -2) if v_first else t for t in states])
    for a, b in zip(*got):
        assert torch.equal(a, b)
