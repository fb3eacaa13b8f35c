"""The chunk-parallel backward of callers without a counter (positional entry point): its blocks take the
work of those that have not started, at item counts around the number of SMs and far above, beside another
kernel too, and nothing is allocated for it."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _call(lens, hq, hv, tiles):
    """(launch of the positional entry point, what the operator's backward gives)"""
    from flash_qla import chunk_gated_delta_rule_bwd
    from flashqla_b200 import ops

    gen = torch.Generator(device=DEV).manual_seed(sum(lens) + hv)
    rn = lambda *s: torch.randn(*s, device=DEV, generator=gen)  # noqa: E731
    T = sum(lens)
    q, k = (torch.nn.functional.normalize(rn(1, T, hq, 128), dim=-1).bfloat16() for _ in range(2))
    v, do = rn(1, T, hv, 128).bfloat16(), rn(1, T, hv, 128).bfloat16()
    g, beta = torch.nn.functional.logsigmoid(rn(1, T, hv)), torch.sigmoid(rn(1, T, hv))
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
    tables, scale = ops.SeqTables(1, T, cu), 128 ** -0.5
    g_cum, A = ops.kkt_solve(k, beta, g, cu, raw_gate=True)
    fw = ops.fwd_seq(None, k, v, A, g_cum, beta, scale, None, output_o=False, output_h=True,
                     output_vnew=True, tables=tables, operand_tiles=tiles)
    bw = ops.bwd_dh(q, k, A, g_cum, beta, do, scale, None, tables=tables, operand_tiles=tiles)
    want = chunk_gated_delta_rule_bwd(q, k, v, g_cum, beta, A, do, cu_seqlens=cu, auto_cp=False)[:4]
    if hq != hv:  # the operator sums dq, dk over value heads
        want = (None, None, *want[2:])
    return lambda: ops.bwd_main(q, k, v, fw["vnew"], A, g_cum, beta, do, bw["du"], fw["h"], bw["dh"], scale,
                                tables=tables, operand_tiles=tiles), want


@pytest.mark.parametrize("tiles", [True, False])
@pytest.mark.parametrize("lens,hq,hv", [([1], 1, 1), ([64] * 37, 4, 4), ([63, 1, 64 * 35 + 1], 4, 4),
                                        ([64 * 149], 1, 1), ([700, 3, 65, 641, 128] * 3, 4, 8),
                                        ([64 * 150 + 9, 64 * 80], 16, 16)])
def test_every_item_is_done_once(lens, hq, hv, tiles):
    call, want = _call(lens, hq, hv, tiles)
    for _ in range(3):
        for x, y in zip(call(), want):
            assert y is None or torch.equal(x, y)


def test_beside_another_kernel():
    """Blocks of two launches share the SMs: each launch still does its own items."""
    a, want_a = _call([64 * 90, 333], 8, 8, True)
    b, want_b = _call([1000, 64 * 70], 8, 8, True)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    out = []
    for i in range(8):
        with torch.cuda.stream(streams[i % 2]):
            out.append((a() if i % 2 else b(), want_a if i % 2 else want_b))
    torch.cuda.synchronize()
    for got, want in out:
        for x, y in zip(got, want):
            assert torch.equal(x, y)


def test_nothing_is_allocated():
    call, _ = _call([64 * 200], 8, 8, True)  # 1600 items
    call()
    torch.cuda.synchronize()
    cuda = ctypes.CDLL("libcuda.so.1")
    pool, used = ctypes.c_void_p(), ctypes.c_uint64(0)
    assert cuda.cuDeviceGetDefaultMemPool(ctypes.byref(pool), torch.cuda.current_device()) == 0
    USED_HIGH = 8  # CU_MEMPOOL_ATTR_USED_MEM_HIGH; writing zero resets it
    assert cuda.cuMemPoolSetAttribute(pool, USED_HIGH, ctypes.byref(used)) == 0
    call()
    torch.cuda.synchronize()
    assert cuda.cuMemPoolGetAttribute(pool, USED_HIGH, ctypes.byref(used)) == 0
    assert used.value == 0
