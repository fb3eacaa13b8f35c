"""The chunk-parallel backward where its tiles have edges: chunks that end inside and at the borders of the
8-row blocks of its 64 x 64 operand tiles (the one that is kept together with its transpose among them),
alone and as the last chunk of a longer sequence, and beta that is zero, negative or above one.

Reference: the fp32 oracle.  Tolerance: what the repository states for gradients, 1e-2 of the norm (bf16
operands, each rounding 2^-9)."""

import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", ["sigmoid", "signed"])
@pytest.mark.parametrize("lens,hq,hv", [([1, 2, 7, 8, 9], 1, 2), ([15, 16, 17, 31, 33], 2, 2),
                                        ([63, 64, 65, 47], 1, 1), ([64 * 3 + 24, 64 * 2 + 40], 2, 4)])
def test_gradients_at_block_edges(lens, hq, hv, beta):
    import flashqla_b200 as fq

    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    x = orc.make_inputs(1, sum(lens), hq, hv, 128, 128, len(lens) + hv, cu_seqlens=cu)
    if beta == "signed":  # zeros, negative values and values up to 2
        x["beta"] = (4 * x["beta"].float() - 2).clamp(min=-1).where(x["beta"].float() > 0.3, 0.0)
    f = {n: (t.float() if t is not None else None) for n, t in x.items()}
    ref = orc.chunk_gdr_bwd(f["q"], f["k"], f["v"], f["g"], f["beta"], f["do"], f["dht"], None, f["h0"], cu)
    d = {n: (t.cuda() if t is not None else None) for n, t in x.items()}
    d["q"], d["k"], d["v"], d["do"] = (d[n].bfloat16() for n in ("q", "k", "v", "do"))
    g_cum, A, *_ = fq.chunk_gated_delta_rule_fwd(d["q"], d["k"], d["v"], d["g"].float(), d["beta"], None,
                                                 d["h0"], cu.cuda(), output_final_state=True)
    got = fq.chunk_gated_delta_rule_bwd(d["q"], d["k"], d["v"], g_cum, d["beta"], A, d["do"], d["dht"], None,
                                        d["h0"], cu.cuda())
    for name, a, b in zip(("dq", "dk", "dv", "db", "dg", "dh0"), got, ref):
        assert orc.rel_err(a.float(), b) <= 1e-2, name
