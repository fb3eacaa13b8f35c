"""D = 64: the sequential kernels walk 32-wide slices of the state while there are few (sequence, head)
pairs and 64-wide ones otherwise.  A column's arithmetic is the same in both, so a packed batch of
many sequences (wide) gives bit for bit what its sequences give one by one (narrow); and a split
sequence, whose transition matrices add slices, agrees with the unsplit one.

dg and dbeta are not compared bit for bit: the chunk-parallel kernel behind the sequential ones sums
them with shared-memory atomics, in any order.  Bound: some 500 fp32 additions of terms below 10,
500 * 2^-24 * 10 = 3e-4."""

import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu


def _run(x, h0, dht, cu, auto_cp=False, v_first=False):
    from flash_qla import chunk_gated_delta_rule

    leaves = [t.detach().clone().requires_grad_() for t in (*x[:5], h0)]
    o, ht = chunk_gated_delta_rule(*leaves[:5], initial_state=leaves[5], output_final_state=True,
                                   cu_seqlens=cu, auto_cp=auto_cp, state_v_first=v_first)
    return (o.detach(), ht.detach(), *torch.autograd.grad((o, ht), leaves, (x[5], dht)))


def _inputs(T, n, hq, hv, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    unit = torch.nn.functional.normalize
    q, k = (unit(rn(1, T, hq, 64), dim=-1).bfloat16() for _ in range(2))
    x = (q, k, rn(1, T, hv, 64).bfloat16(), torch.nn.functional.logsigmoid(rn(1, T, hv)),
         torch.sigmoid(rn(1, T, hv)), rn(1, T, hv, 64).bfloat16())
    return x, 0.1 * rn(n, hv, 64, 64), 0.1 * rn(n, hv, 64, 64)


@pytest.mark.parametrize("v_first", [False, True])
@pytest.mark.parametrize("hq,hv", [(2, 4), (1, 2)])
def test_wide_and_narrow_slices_agree_bit_for_bit(hq, hv, v_first):
    lens = [1, 63, 64, 65, 130] * 8  # 40 sequences: 80 or 160 pairs
    x, h0, dht = _inputs(sum(lens), len(lens), hq, hv, hv)
    ends = [sum(lens[:i]) for i in range(len(lens) + 1)]
    got = _run(x, h0, dht, torch.tensor(ends, dtype=torch.int32, device="cuda"), v_first=v_first)
    for i in range(5):
        a, b = ends[i], ends[i + 1]
        alone = _run([t[:, a:b].contiguous() for t in x], h0[i:i + 1], dht[i:i + 1], None, v_first=v_first)
        for j, (y, z) in enumerate(zip(got, alone)):
            y = y[i:i + 1] if j in (1, 7) else y[:, a:b]
            if j in (5, 6):
                assert torch.allclose(y, z, rtol=0, atol=3e-4), (i, j)
            else:
                assert torch.equal(y, z), (i, j)


def test_split_against_unsplit():
    """Bound: two correct evaluations in bf16 (the tolerance of the parity tests)."""
    x, h0, dht = _inputs(4096 + 33, 1, 1, 2, 9)
    x = (*x[:3], x[3] * torch.tensor([1.0, 0.0], device="cuda"), *x[4:])  # one head without decay
    for y, z in zip(_run(x, h0, dht, None, auto_cp=True), _run(x, h0, dht, None)):
        assert orc.rel_err(y, z) < 1e-2
