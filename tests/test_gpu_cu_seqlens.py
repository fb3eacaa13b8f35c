"""``cu_seqlens`` that changes between calls: the index tables follow its values, however it was made;
and values outside the rows, which are refused before anything is launched."""

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


@pytest.mark.parametrize("values", [[], [-1, 3000], [0, 3001], [0, 1600, 1500, 3000], [0, 2 ** 33]], ids=str)
def test_bounds_outside_the_rows_are_refused(values):
    args = _args()
    cu = torch.tensor(values, dtype=torch.int64, device=DEV)
    with pytest.raises(ValueError, match="cu_seqlens"):
        _call(args, cu)


@pytest.mark.parametrize("values", [[0], [0, 0, 2000], [64, 2500]], ids=str)
def test_bounds_inside_the_rows_are_taken(values):
    """No sequence, an empty one, rows before the first and behind the last."""
    args = _args()
    o, ht = _call(args, torch.tensor(values, dtype=torch.int64, device=DEV))
    assert ht.shape[0] == len(values) - 1
    for i, (a, b) in enumerate(zip(values[:-1], values[1:])):
        if a < b:
            alone = _call([t[:, a:b].contiguous() for t in args], None)
            assert orc.rel_err(o[:, a:b], alone[0]) < 5e-3 and orc.rel_err(ht[i], alone[1][0]) < 5e-3
