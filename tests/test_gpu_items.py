"""The chunk-parallel backward hands its (chunk, head) items to the CTAs as they go: every item must
be done once, whoever takes it.  Its results do not depend on that, so a packed batch gives bit for
bit what its sequences give one by one (a few items each), at item counts around the number of SMs
and around the size from which a launch without a counter makes its own."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(lens, hq, hv, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T = sum(lens)
    unit = torch.nn.functional.normalize
    q, k = (unit(rn(1, T, hq, 128), dim=-1).bfloat16() for _ in range(2))
    return (q, k, rn(1, T, hv, 128).bfloat16(), torch.nn.functional.logsigmoid(rn(1, T, hv)),
            torch.sigmoid(rn(1, T, hv)), rn(1, T, hv, 128).bfloat16())


def _grads(x, cu):
    from flash_qla import chunk_gated_delta_rule_bwd, chunk_gated_delta_rule_fwd

    q, k, v, g, beta, do = x
    g_cum, A, *_ = chunk_gated_delta_rule_fwd(q, k, v, g, beta, cu_seqlens=cu, auto_cp=False)
    return chunk_gated_delta_rule_bwd(q, k, v, g_cum, beta, A, do, cu_seqlens=cu, auto_cp=False)[:5]


@pytest.mark.parametrize("lens,hq,hv", [([1], 1, 1), ([64, 65], 1, 2), ([64] * 37, 2, 4),
                                        ([63, 1, 64 * 35 + 1], 2, 4), ([700, 3, 65, 641, 128] * 3, 4, 8),
                                        ([64 * 37 - 5, 1000], 8, 16)])
def test_packed_equals_each_alone(lens, hq, hv):
    x = _batch(lens, hq, hv, len(lens) * hv)
    ends = [sum(lens[:i]) for i in range(len(lens) + 1)]
    got = _grads(x, torch.tensor(ends, dtype=torch.int32, device="cuda"))
    for a, b in zip(ends[:-1], ends[1:]):
        alone = _grads([t[:, a:b].contiguous() for t in x], None)
        for name, y, z in zip(("dq", "dk", "dv", "db", "dg"), got, alone):
            assert torch.equal(y[:, a:b], z), (name, a, b)


def test_a_launch_without_a_counter():
    """The positional entry point, also replayed from a CUDA graph, against the operator."""
    from flashqla_b200 import ops

    lens = [640, 333, 64 * 20 + 7]
    q, k, v, g, beta, do = x = _batch(lens, 32, 32, 3)
    ends = [sum(lens[:i]) for i in range(len(lens) + 1)]
    cu = torch.tensor(ends, dtype=torch.int32, device="cuda")
    want = _grads(x, cu)
    tables = ops.SeqTables(1, sum(lens), cu)
    scale = 128 ** -0.5
    g_cum, A = ops.kkt_solve(k, beta, g, cu, raw_gate=True)
    fw = ops.fwd_seq(None, k, v, A, g_cum, beta, scale, None, output_o=False, output_h=True,
                     output_vnew=True, tables=tables, operand_tiles=True)
    bw = ops.bwd_dh(q, k, A, g_cum, beta, do, scale, None, tables=tables, operand_tiles=True)

    def main():
        return ops.bwd_main(q, k, v, fw["vnew"], A, g_cum, beta, do, bw["du"], fw["h"], bw["dh"], scale,
                            tables=tables, operand_tiles=True)

    for y, z in zip(main()[:4], want[:4]):
        assert torch.equal(y, z)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = main()
    for _ in range(2):
        for t in out:
            t.zero_()
        graph.replay()
        for y, z in zip(out[:4], want[:4]):
            assert torch.equal(y, z)
