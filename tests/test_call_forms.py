"""Forms of a call that need no GPU: modes around the operators and types of arguments."""
import numpy as np
import pytest
import torch
import torch.autograd.forward_ad as forward_ad

from cute_triadic_gdn_b200 import (chunk_gdn_joint, chunk_gdn_joint_segment, conv_split_act_call, conv_split_norm_call, gdn_joint_call,
                                   gdn_joint_decode)


@pytest.fixture
def cpu_operators():
    """The forward operators on the CPU, as far as a call around them goes: outputs of the right shapes."""
    lib = torch.library.Library("tgdn_b200", "IMPL", "CPU")

    def norm(x, w, heads, slices, eps, cu=None):
        B, T, _ = x.shape
        return (*[x.new_zeros(B, T, heads, 128) for _ in range(3)], *[torch.zeros(B, T, heads, slices) for _ in range(2)])

    lib.impl("joint_fwd", lambda q, k, v, *rest: [v + 1] + [torch.zeros(1) for _ in range(6)])
    lib.impl("conv_split_act_fwd", lambda x, w, act, cu=None: x + 1)
    lib.impl("conv_split_norm_fwd", norm)
    yield
    lib._destroy()


def _calls():
    q = torch.ones(1, 64, 2, 128, dtype=torch.bfloat16)
    k2 = torch.ones(1, 64, 2, 4)
    x, w = torch.ones(1, 8, 784, dtype=torch.bfloat16), torch.ones(784, 4, dtype=torch.bfloat16)
    return {"core": (gdn_joint_call, (q, q, q, k2, k2, k2, k2[..., 0].contiguous())),
            "conv": (lambda x, w: conv_split_act_call(x, w, 8), (x, w)),
            "glue": (lambda x, w: conv_split_norm_call(x, w, 2, 4)[0], (x, w))}


@pytest.mark.parametrize("name", ["core", "conv", "glue"])
def test_inputs_with_tangents_and_nothing_to_differentiate(cpu_operators, name):
    """The operators have no forward-mode derivative: values are computed, tangents end there."""
    call, args = _calls()[name]
    ref = call(*args)
    with forward_ad.dual_level():
        out = forward_ad.unpack_dual(call(*[forward_ad.make_dual(t, torch.ones_like(t)) for t in args]))
    assert torch.equal(out.primal, ref) and out.tangent is None
    out, tangent = torch.func.jvp(call, args, args)
    assert torch.equal(out, ref) and not tangent.any()


@pytest.mark.parametrize("name", ["core", "conv", "glue"])
def test_leaves_are_tracked_only_under_grad_mode(cpu_operators, name):
    call, args = _calls()[name]
    leaves = [t.clone().requires_grad_(True) for t in args]
    assert call(*leaves).requires_grad and not call(*args).requires_grad
    with torch.no_grad():
        assert not call(*leaves).requires_grad
    with torch.inference_mode():
        assert not call(*args).requires_grad


@pytest.mark.parametrize("scale", [0.5, 1, "0.5", np.float32(0.5), torch.tensor(0.5)])
@pytest.mark.parametrize("tokens", [64, 64.0, "64", np.int64(64), torch.tensor(64)])
def test_whatever_converts_to_a_number_is_one(scale, tokens):
    """Numbers may be of any type that float() and int() take: these calls come as far as the checks of the inputs (which want a GPU)."""
    q = torch.ones(1, 64, 2, 128, dtype=torch.bfloat16)
    k2 = torch.ones(1, 64, 2, 4)
    args = (q, q, q, k2, k2, k2, k2[..., 0].contiguous())
    with pytest.raises(AssertionError, match="CUDA device"):
        chunk_gdn_joint(*args, scale=scale, checkpoint_tokens=tokens)
    with pytest.raises(AssertionError, match="CUDA device"):
        chunk_gdn_joint_segment(*args, scale=scale)
    with pytest.raises(ValueError, match="CUDA device"):
        gdn_joint_decode(*[t[:, :1] for t in args], torch.zeros(1, 2, 4, 128, 128), scale=scale)
    with pytest.raises(NotImplementedError, match="CPU"):
        gdn_joint_call(*args, scale=scale)
