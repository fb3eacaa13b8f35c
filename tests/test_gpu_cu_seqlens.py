"""``cu_seqlens`` that changes between calls: the index tables follow its values, however it was made."""

import pytest
import torch

from oracle import gdr_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"
FIRST, THEN = [0, 500, 1500, 3000], [0, 64, 2950, 3000]


def _call(args, cu):
    import flashqla_b200 as fq

    return fq.chunk_gated_delta_rule(*args, output_final_state=True, cu_seqlens=cu)


def _args():
    x = orc.make_inputs(1, 3000, 1, 2, 128, 128, seed=4)
    return [x[n].bfloat16().to(DEV) for n in ("q", "k", "v")] + [x["g"].to(DEV), x["beta"].to(DEV)]


@pytest.mark.parametrize("made_in_inference_mode", [False, True])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_changed_in_place(made_in_inference_mode, dtype):
    args = _args()
    with torch.inference_mode(made_in_inference_mode):
        cu = torch.tensor(FIRST, dtype=dtype, device=DEV)
        assert cu.is_inference() == made_in_inference_mode
    with torch.inference_mode():
        for values in (FIRST, THEN, FIRST, FIRST):
            cu.copy_(torch.tensor(values, dtype=dtype))
            got, want = _call(args, cu), _call(args, torch.tensor(values, dtype=dtype, device=DEV))
            for a, b in zip(got, want):
                assert torch.equal(a, b)


def test_inference_tensor_under_capture():
    args = _args()
    with torch.inference_mode():
        cu = torch.tensor(FIRST, dtype=torch.int32, device=DEV)
        _call(args, cu)
        cu.copy_(torch.tensor(THEN, dtype=torch.int32))
        want = _call(args, cu)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = _call(args, cu)
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(out, want):
            assert torch.equal(a, b)
