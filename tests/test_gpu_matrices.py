"""The transition matrices that the forward keeps for the backward (attributes of its cache): the
gradients are bit for bit those of a backward that makes its own.  Segments that never forget, gates that
rise again (where the scans of the two directions decide differently, so that each side has matrices the other
lacks), ragged ends, several sequences, one of them unsplit."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gate", ["never", "rising", "mixed"])
@pytest.mark.parametrize("lens", [[64 * 70], [64 * 41 + 9, 100, 64 * 30]])
def test_kept_matrices_change_nothing(lens, gate):
    import flashqla_b200 as fq

    gen = torch.Generator(device="cuda").manual_seed(len(lens))
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    T, hq, hv = sum(lens), 2, 4
    unit = torch.nn.functional.normalize
    q, k = (unit(rn(1, T, hq, 128), dim=-1).bfloat16() for _ in range(2))
    v, do = rn(1, T, hv, 128).bfloat16(), rn(1, T, hv, 128).bfloat16()
    g = torch.nn.functional.logsigmoid(rn(1, T, hv)) / 16
    if gate == "never":
        g[:] = 0.0
    elif gate == "rising":  # a fall of 12 over one chunk in every six, slowly made up for by the others
        chunk = torch.arange(T, device="cuda") // 64 % 6
        g[:] = torch.where(chunk == 2, -12.0 / 64, 2.3 / 64)[None, :, None]
    else:
        g[..., 3::4] = 0.0
    beta = torch.sigmoid(rn(1, T, hv))
    h0, dht = 0.1 * rn(len(lens), hv, 128, 128), 0.1 * rn(len(lens), hv, 128, 128)
    cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device="cuda")
    g_cum, A, *_, cache = fq.chunk_gated_delta_rule_fwd(q, k, v, g, beta, None, h0, cu, output_final_state=True,
                                                        enable_fwd_cp_cache=True)
    assert len(cache) == 4 and cache.seg_m is not None
    args = (q, k, v, g_cum, beta, A, do, dht, None, h0, cu)
    own = fq.chunk_gated_delta_rule_bwd(*args, cp_cache=tuple(cache))
    for _ in range(2):
        for a, b in zip(fq.chunk_gated_delta_rule_bwd(*args, cp_cache=cache), own):
            assert torch.equal(a, b)
