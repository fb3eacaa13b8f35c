"""The forward recurrence with two and with three stages of its tiles: which one a launch takes depends on the mean
length of its walks, and the same sequence comes out the same bits in both."""

import pytest
import torch

import flashqla_b200 as fq
from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("state_v_first", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("length", [768, 769, 831, 896, 959])
def test_same_bits_in_a_long_and_in_a_short_batch(length, dtype, state_v_first):
    # alone: walks of twelve chunks and more; among 24 sequences of one token: below
    short = 24
    x = orc.make_inputs(1, length + short, 2, 4, 128, 128, seed=length,
                        cu_seqlens=torch.tensor([0, length, *range(length + 1, length + short + 1)]))
    d = {n: t.cuda() for n, t in x.items()}
    q, k, v = (d[n].to(dtype) for n in ("q", "k", "v"))

    def run(rows, ends):
        cu = torch.tensor([0, *ends], dtype=torch.int32, device="cuda")
        h0 = d["h0"][:len(ends)].contiguous()
        _, _, o, _, ht, _ = fq.chunk_gated_delta_rule_fwd(
            q[:, :rows].contiguous(), k[:, :rows].contiguous(), v[:, :rows].contiguous(),
            d["g"][:, :rows].contiguous(), d["beta"][:, :rows].contiguous(), None, h0, cu,
            output_final_state=True, state_v_first=state_v_first, auto_cp=False)
        return o[:, :length], ht[:1]

    alone = run(length, [length])
    among = run(length + short, [length, *range(length + 1, length + short + 1)])
    for a, b in zip(alone, among):
        assert torch.equal(a, b)
    if dtype == torch.bfloat16 and not state_v_first:
        ref = orc.chunk_gdr_fwd(*(x[n][:, :length] for n in ("q", "k", "v", "g", "beta")), None, x["h0"][:1],
                                torch.tensor([0, length]))
        assert orc.rel_err(alone[0].float(), ref[2]) <= 5e-3
        assert orc.rel_err(alone[1], ref[4]) <= 5e-3
