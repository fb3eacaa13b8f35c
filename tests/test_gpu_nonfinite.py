"""NaN and infinity in one row of k, beta or the gate: the inverse of ``kkt_solve`` shows them wherever
forward substitution would (row r and all rows after it, the columns before r), at and off the edges of
its 16 x 16 blocks, and nothing before that block row, in other chunks or in other heads changes."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D,Hq,Hv", [(128, 2, 2), (128, 1, 5), (64, 2, 4)])
@pytest.mark.parametrize("where,value", [("beta", "nan"), ("beta", "inf"), ("k", "nan"), ("g", "nan")])
@pytest.mark.parametrize("r", [1, 15, 16, 17, 32, 48, 63])
def test_the_inverse_shows_them(D, Hq, Hv, where, value, r):
    from flashqla_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(r)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, row = 64 * 3, 64 + r
    x = dict(k=torch.nn.functional.normalize(rn(1, T, Hq, D), dim=-1).bfloat16(),
             beta=torch.sigmoid(rn(1, T, Hv)), g=torch.nn.functional.logsigmoid(rn(1, T, Hv)))
    want = ops.kkt_solve(x["k"], x["beta"], x["g"], raw_gate=True)[1]
    x[where][0, row, 0] = float(value)
    A = ops.kkt_solve(x["k"], x["beta"], x["g"], raw_gate=True)[1]
    heads = Hv // Hq if where == "k" else 1  # that see the value
    assert not torch.isfinite(A[0, row:128, :heads, :r]).any()
    assert torch.equal(A[0, :, heads:], want[0, :, heads:])
    first = 64 + r // 16 * 16
    assert torch.equal(A[0, :first], want[0, :first]) and torch.equal(A[0, 128:], want[0, 128:])
