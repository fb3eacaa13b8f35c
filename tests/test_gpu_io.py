"""The one-pass kernels in front of and behind the recurrence (``fqla_prepare_inputs``,
``fqla_finish_grads``) against the same expressions in fp32, at row counts around a thread block's
edge (256 threads x 8 elements) and for every type and head dimension they take.

Bounds: a value rounded once to bf16 / fp16 is off by at most 2^-9 / 2^-12 of itself, so the
normalised error of a tensor rounded once is below 2^-9 / 2^-12; the reductions are fp32 sums of at
most 128 terms (1e-5)."""

import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUND = {torch.bfloat16: 2.0 ** -9, torch.float16: 2.0 ** -12}


def _call(name, *args):
    from flashqla_b200 import _lib

    st = getattr(_lib.load(), name)(*[a.data_ptr() if isinstance(a, torch.Tensor) else a for a in args],
                                    torch.cuda.current_stream().cuda_stream)
    assert st == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("rows,G", [(1, 1), (3, 4), (16, 1), (33, 2), (1000, 8)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("norm", [False, True], ids=["plain", "l2norm"])
def test_inputs_and_gradients_one_pass(rows, G, D, dtype, norm):
    gen = torch.Generator(device=DEV).manual_seed(rows * 8 + G)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    q, k, v = rn(rows, D).to(dtype), rn(rows, D).to(dtype), rn(rows * G, D).to(dtype)
    f16 = dtype == torch.float16
    qo, ko, vo = (torch.full_like(t, float("nan"), dtype=torch.bfloat16) for t in (q, k, v))
    rstd = torch.full((2, rows), float("nan"), device=DEV)
    _call("fqla_prepare_inputs", q, k, v, qo, ko, vo, rstd[0], rstd[1], rows, rows * G, D, int(f16),
          int(norm), 1e-6)
    for x, y, r in ((q, qo, rstd[0]), (k, ko, rstd[1])):
        want_r = torch.rsqrt(x.float().square().sum(-1) + 1e-6)
        if norm:
            assert orc.rel_err(r, want_r) < 1e-5
        want = x.float() * want_r[:, None] if norm else x.float()
        assert orc.rel_err(y.float(), want) < ROUND[torch.bfloat16]
    assert orc.rel_err(vo.float(), v.float()) < ROUND[torch.bfloat16]

    gq, gk, gv = (rn(rows * G, D).bfloat16() for _ in range(3))
    dq, dk, dv = torch.full_like(q, float("nan")), torch.full_like(k, float("nan")), torch.full_like(v, float("nan"))
    r_args = (rstd[0], rstd[1]) if norm else (None, None)
    _call("fqla_finish_grads", gq, gk, gv, q, k, *r_args, dq, dk, dv, rows, G, D, int(f16))
    for x, gr, out, r in ((q, gq, dq, rstd[0]), (k, gk, dk, rstd[1])):
        want = gr.float().view(rows, G, D).sum(1)
        if norm:
            y = x.float() * r[:, None]
            want = (want - (want * y).sum(-1, keepdim=True) * y) * r[:, None]
        assert orc.rel_err(out.float(), want) < ROUND[dtype] + 1e-5
    assert orc.rel_err(dv.float(), gv.float()) < ROUND[dtype]


def test_operator_keeps_nothing_for_a_backward_that_cannot_come():
    """Without a differentiable input, or with gradients off, the operator records nothing; with
    one it gives the same values and a gradient."""
    import flashqla_b200 as fq

    x = orc.make_inputs(1, 130, 1, 2, 128, 128, seed=3, with_h0=True)
    d = {n: (x[n].bfloat16() if n in ("q", "k", "v", "beta") else x[n]).to(DEV)
         for n in ("q", "k", "v", "g", "beta")}
    plain, _ = fq.chunk_gated_delta_rule(**d)
    assert plain.grad_fn is None
    d["v"].requires_grad_(True)
    with torch.no_grad():
        off, ht = fq.chunk_gated_delta_rule(**d, output_final_state=True)
    assert off.grad_fn is None and ht.grad_fn is None
    on, ht = fq.chunk_gated_delta_rule(**d, output_final_state=True)
    assert on.grad_fn is not None and ht.grad_fn is not None
    assert torch.equal(on, plain) and torch.equal(off, plain)
    # only the final state is used: the gradient of o is absent, not zero-filled by the caller
    (gv,) = torch.autograd.grad(ht.sum(), d["v"])
    assert gv.dtype == torch.bfloat16 and bool(gv.float().abs().sum() > 0)
