"""Where states enter and leave the sequential kernels: the row maps of a split plan, both state
layouts and float16 output, against the plain form of the same call (same arithmetic: same bits)."""

import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(T, Hq, Hv, D, cu, seed=5):
    cu_t = torch.tensor(cu, dtype=torch.int32)
    x = orc.make_inputs(1, T, Hq, Hv, D, D, seed=seed, cu_seqlens=cu_t, with_h0=True)
    d = {n: (x[n].bfloat16() if n in ("q", "k", "v", "beta", "do") else x[n]).to(DEV)
         for n in ("q", "k", "v", "g", "beta", "h0", "do", "dht")}
    return d, cu_t.to(DEV)


# a split sequence, an empty one, one shorter than a chunk, a ragged tail; both kernel families
@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("cu", [[0, 2100, 2100, 2140, 3701], [0, 1, 65]], ids=["split", "short"])
def test_state_layouts_give_the_same_bits(D, cu):
    import flashqla_b200 as fq

    d, cu_t = _inputs(cu[-1], 1, 2, D, cu)
    tr = lambda t: t.transpose(-1, -2).contiguous()  # noqa: E731
    res = []
    for vf in (False, True):
        f = tr if vf else (lambda t: t)
        g_cum, A, o, _, ht, cache = fq.chunk_gated_delta_rule_fwd(
            d["q"], d["k"], d["v"], d["g"], d["beta"], None, f(d["h0"]), cu_t, state_v_first=vf,
            enable_fwd_cp_cache=True)
        grads = fq.chunk_gated_delta_rule_bwd(
            d["q"], d["k"], d["v"], g_cum, d["beta"], A, d["do"], f(d["dht"]), None, f(d["h0"]),
            cu_t, vf, cp_cache=cache)
        res.append([o, f(ht), *grads[:5], f(grads[5])])
    # the D = 64 chunk kernel sums dg, dbeta with shared-memory atomics: equal up to fp32 rounding
    for a, b in zip(*res):
        assert torch.equal(a, b) or (D == 64 and orc.rel_err(a, b) < 1e-5)
    # an empty sequence hands its state through
    empty = [i for i in range(len(cu) - 1) if cu[i] == cu[i + 1]]
    for i in empty:
        assert torch.equal(res[0][1][i], d["h0"][i])


@pytest.mark.parametrize("T", [1, 64, 130])
def test_float16_output_is_the_rounding_of_the_same_accumulators(T):
    """o leaves the kernel as fp16 straight from the fp32 accumulators: against the bf16 output it
    may differ by bf16's rounding (2^-9 of a value) and nothing more."""
    import flashqla_b200 as fq

    d, cu_t = _inputs(T, 1, 2, 128, [0, T])
    o_bf, ht_bf = fq.chunk_gated_delta_rule(d["q"], d["k"], d["v"], d["g"], d["beta"],
                                            initial_state=d["h0"], output_final_state=True)
    h = {n: d[n].half() for n in ("q", "k", "v")}  # bf16 values of this range are exact in fp16
    o_h, ht_h = fq.chunk_gated_delta_rule(h["q"], h["k"], h["v"], d["g"], d["beta"],
                                          initial_state=d["h0"], output_final_state=True)
    assert o_h.dtype == torch.float16 and torch.equal(ht_h, ht_bf)
    assert bool(((o_h.float() - o_bf.float()).abs() <= 2.0 ** -8 * o_bf.float().abs() + 1e-6).all())
