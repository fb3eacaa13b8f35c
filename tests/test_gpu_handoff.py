"""End states and transition matrices of the exact hand-off (K = V = 128) against the same walk in
64 bits, with bf16 roundings where the kernel's operands need them and nowhere else: the copy of the
state, W = beta (V - gamma K S) against the part of A below its diagonal, and rho Vn (A comes in as bf16).

One chunk: the two differ where fp32 sums (relative error about 1e-6) put a value on the other side of
a bf16 boundary (spacing 2^-8): a share of 5e-4 of the values moves by 2^-8, 1e-4 in the norm; bound
4e-4.  A rounding more in the walk costs 2e-3.  Later chunks inherit the differences through their own
roundings, so longer walks are compared by their error against the walk without roundings: it may be 5 %
above that of the 64-bit walk with them (the errors are norms over 16384 values per head, several heads
and sequences; another rounding of A or of w costs 9 to 17 %)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(lens, Hq, Hv, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    T = sum(lens)
    k = torch.nn.functional.normalize(rn(1, T, Hq, 128), dim=-1).bfloat16()
    v, beta = rn(1, T, Hv, 128).bfloat16(), torch.sigmoid(rn(1, T, Hv))
    g = torch.nn.functional.logsigmoid(rn(1, T, Hv)) / 16
    g[..., 1::2] = 0.0
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    return k, v, g, beta, cu


def _walk(k, v, A, g_cum, beta, s, e, start, rounded):
    """State [Hv, D, D] after rows s .. e of one sequence, in 64 bits."""
    rnd = (lambda x: x.bfloat16().double()) if rounded else (lambda x: x)
    Hv = v.shape[2]
    S = start.clone()
    for a in range(s, e, 64):
        b = min(a + 64, e)
        K = k[0, a:b].double().repeat_interleave(Hv // k.shape[2], 1).transpose(0, 1)
        V, Ac = v[0, a:b].double().transpose(0, 1), A[0, a:b, :, :b - a].double().transpose(0, 1)
        gc, bt = g_cum[0, a:b].double().T[..., None], beta[0, a:b].double().T[..., None]
        W = bt * (V - gc.exp() * (K @ rnd(S)))
        Vn = Ac @ rnd(W) + (W - rnd(W))
        S = gc[:, -1:].exp() * S + K.transpose(1, 2) @ rnd((gc[:, -1:] - gc).exp() * Vn)
    return S


def _run(lens, Hq, Hv, seed):
    from flashqla_b200 import ops

    k, v, g, beta, cu = _inputs(lens, Hq, Hv, seed)
    g_cum, A = ops.kkt_solve(k, beta, g, cu, raw_gate=True)
    out = ops.fwd_seq(None, k, v, A, g_cum, beta, 1.0, output_o=False, output_final_state=True,
                      output_m=True, cu_seqlens=cu)
    eye = torch.eye(128, device=DEV, dtype=torch.float64).expand(Hv, -1, -1)
    bounds = list(zip(cu.tolist()[:-1], cu.tolist()[1:]))
    want = {}
    for rounded in (True, False):
        walk = lambda vv, st: torch.stack([_walk(k, vv, A, g_cum, beta, s, e, st, rounded)  # noqa: E731
                                           for s, e in bounds])
        want[rounded] = walk(v, torch.zeros_like(eye)), walk(torch.zeros_like(v), eye)
    return (out["ht"].double(), out["M"].double()), want


@pytest.mark.parametrize("lens", [[1], [64], [63, 2, 17, 64]], ids=str)
@pytest.mark.parametrize("Hq,Hv", [(1, 1), (2, 4)])
def test_one_chunk_rounds_only_the_operands(lens, Hq, Hv):
    got, want = _run(lens, Hq, Hv, 3)
    for x, y, z in zip(got, want[True], want[False]):
        # M of a chunk of few rows is nearly the identity: relative to what the chunk changed
        change = (z - torch.eye(128, device=DEV, dtype=torch.float64)).norm() if y is want[True][1] else z.norm()
        assert (x - y).norm() < 4e-4 * change


@pytest.mark.parametrize("chunks", [8, 28])
def test_longer_walks_are_as_exact_as_their_operands_allow(chunks):
    n = 64 * chunks
    got, want = _run([n, n - 1, n - 63, n], 2, 4, 7)
    for x, y, z in zip(got, want[True], want[False]):
        assert (x - z).norm() < 1.05 * (y - z).norm()
