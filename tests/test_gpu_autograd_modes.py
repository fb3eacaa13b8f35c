"""The operator under the modes of PyTorch that see more than a call's values: traces, functorch
transforms, forward-mode tangents, saved-tensor hooks and non-reentrant checkpoints.  The native
autograd node must do there what ``ChunkGatedDeltaRuleFunction`` does, and refuse what it refuses."""

import pytest
import torch
from torch.utils.checkpoint import checkpoint

pytestmark = pytest.mark.gpu


def _inputs(seed, grad=False):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    unit = torch.nn.functional.normalize
    q, k = (unit(rn(1, 100, 2, 128), dim=-1).bfloat16() for _ in range(2))
    out = [q, k, rn(1, 100, 4, 128).bfloat16(), torch.nn.functional.logsigmoid(rn(1, 100, 4)),
           torch.sigmoid(rn(1, 100, 4))]
    return [t.requires_grad_(grad) for t in out]


def _op(*args):
    from flash_qla import chunk_gated_delta_rule

    return chunk_gated_delta_rule(*args, output_final_state=True)


def test_a_trace_records_the_call():
    traced = torch.jit.trace(_op, tuple(_inputs(0)), check_trace=False)
    other = _inputs(1)
    for got, want in zip(traced(*other), _op(*other)):
        assert torch.equal(got, want)


def test_a_forward_mode_tangent_is_refused():
    import torch.autograd.forward_ad as fwAD

    args = _inputs(0)
    with fwAD.dual_level():
        args[2] = fwAD.make_dual(args[2], torch.ones_like(args[2]))
        with pytest.raises((NotImplementedError, RuntimeError), match="jvp|forward"):
            _op(*args)


@pytest.mark.parametrize("transform", ["vmap", "grad"])
def test_functorch_transforms_are_refused(transform):
    args = _inputs(0)
    with pytest.raises(RuntimeError, match="autograd.Function"):
        if transform == "vmap":
            torch.func.vmap(lambda v: _op(args[0], args[1], v, *args[3:])[0])(args[2][None])
        else:
            torch.func.grad(lambda g: _op(*args[:3], g, args[4])[0].float().sum())(args[3])


@pytest.mark.parametrize("l2norm", [False, True])
def test_checkpoint_gives_the_same_gradients(l2norm):
    """Its recomputation is ended by an exception thrown in a saved-tensor hook."""
    from flash_qla import chunk_gated_delta_rule

    grads = []
    for wrap in (False, True):
        args = _inputs(3, grad=True)

        def f(*a):
            return chunk_gated_delta_rule(*a, use_qk_l2norm_in_kernel=l2norm)[0]

        o = checkpoint(f, *args, use_reentrant=False) if wrap else f(*args)
        o.float().square().sum().backward()
        grads.append([a.grad for a in args])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


def test_an_exception_in_a_saved_tensor_hook_arrives_as_it_is():
    class Stop(Exception):
        pass

    def pack(t):
        raise Stop("from the hook")

    with pytest.raises(Stop, match="from the hook"):
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
            _op(*_inputs(0, grad=True))
    _op(*_inputs(0, grad=True))[0].sum().backward()  # and the operator works on


def test_a_wrong_number_of_dimensions_is_an_index_error():
    args = _inputs(0)
    args[1] = args[1][0, 0]
    with pytest.raises(IndexError):
        _op(*args)
