"""Forms of a call that a program may use: strides, sizes, argument types, threads and modes around it."""
import ctypes
import threading

import pytest
import torch

from cute_triadic_gdn_b200 import (_lib, chunk_gdn_joint, chunk_gdn_joint_segment, conv_split_act_call, conv_split_norm_call,
                                   gdn_joint_call, gdn_joint_decode)
from oracle import triadic_oracle as orc

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def conv_step(x, w, act, dy):
    x, w = x.detach().requires_grad_(True), w.detach().requires_grad_(True)
    y = conv_split_act_call(x, w, act)
    return (y.detach(), *torch.autograd.grad(y, (x, w), dy))


@pytest.mark.parametrize("B,T,C", [(2, 1, 77), (3, 1, 80), (2, 1, 1), (1, 1, 1), (1, 5, 1), (2, 6, 1), (1, 7, 48)])
def test_convolution_of_axes_of_size_one(B, T, C):
    """An axis of size one has whatever stride the tensor was made with, in x and in the gradient (an expanded scalar: zeros)."""
    g = torch.Generator().manual_seed(C)
    x, w = torch.randn(B, T, C, generator=g).to(BF16).cuda(), torch.randn(C, 4, generator=g).to(BF16).cuda()
    ref = conv_step(x, w, C // 2, torch.ones_like(x))
    views = [x.transpose(1, 2).contiguous().transpose(1, 2), x.permute(2, 1, 0).contiguous().permute(2, 1, 0),
             torch.cat([x, x], -1)[..., :C], torch.cat([x, x], 1)[:, :T],
             x.contiguous().as_strided((B, T, C), (x.stride(0) if B > 1 else 3, x.stride(1) if T > 1 else 5, 1 if C > 1 else 7))]
    for v in views:
        for dy in (torch.ones_like(x), torch.ones((), dtype=BF16, device="cuda").expand(B, T, C)):
            for a, b in zip(conv_step(v, w, C // 2, dy), ref):
                assert torch.equal(a, b)
    assert _lib.device_status() == 0


def test_glue_of_one_token_with_any_stride():
    H, E = 2, 4
    C = H * (3 * 128 + 2 * E)
    g = torch.Generator().manual_seed(3)
    x, w = torch.randn(2, 1, C, generator=g).to(BF16).cuda(), torch.randn(C, 4, generator=g).to(BF16).cuda()
    view = x.transpose(1, 2).contiguous().transpose(1, 2)
    for a, b in zip(conv_split_norm_call(view, w, H, E), conv_split_norm_call(x, w, H, E)):
        assert torch.equal(a, b)


def test_convolution_of_more_tokens_than_a_grid_has_rows():
    """65535 runs of 2048 tokens and five more: two bytes a token."""
    T = 65535 * 2048 + 5
    x = torch.ones(1, T, 1, dtype=BF16, device="cuda")
    x[0, -1] = 3.0
    w = torch.tensor([[1.0, 2.0, 4.0, 8.0]], dtype=BF16, device="cuda")
    y = conv_split_act_call(x, w, 0)
    dx, dw = torch.ops.tgdn_b200.conv_split_act_bwd(x, x, w, 0, None)
    assert _lib.device_status() == 0
    assert y[0, :4, 0].tolist() == [8, 12, 14, 15] and y[0, -2:, 0].tolist() == [15, 31] and bool((y[0, 3:-1] == 15).all())
    assert dx[0, -5:, 0].tolist() == [15, 17, 18, 20, 24] and bool((dx[0, :-4] == 15).all())
    # dw[j] = sum of x[t] x[t - 3 + j]: T in f32 partials, rounded to bf16 (2^-9) at the end
    assert torch.allclose(dw.float(), torch.full_like(dw, T).float(), rtol=2 ** -8)


def test_thread_whose_context_was_taken_away():
    """Another library in the process may leave a thread without a current context after the thread's first call."""
    ins = [t.cuda() for t in orc.make_inputs(1, 64, 2, 2, seed=5)]
    ref, got = gdn_joint_call(*ins), []

    def work():
        try:
            got.append(gdn_joint_call(*ins))
            assert ctypes.CDLL("libcuda.so.1").cuCtxSetCurrent(None) == 0
            got.append(gdn_joint_call(*ins))
            torch.cuda.synchronize()
        except Exception as e:                               # noqa: BLE001 (shown by the comparison below)
            got.append(e)

    thread = threading.Thread(target=work)
    thread.start()
    thread.join()
    assert len(got) == 2 and all(torch.equal(o, ref) for o in got), got


@pytest.mark.parametrize("E", [2, 8, 16])
def test_operator_with_a_chunk_map_that_misses_tokens(E):
    """Rows of o and dV that no document holds are zero, whatever the allocator hands out."""
    T, H, cu = 256, 2, torch.tensor([0, 60, 130], dtype=torch.int32).cuda()
    ins = [t.cuda() for t in orc.make_inputs(1, T, H, E, seed=E)]
    do = orc.make_grad_output((1, T, H, 128), 1).cuda()
    offsets, chunk_map, valid = torch.ops.tgdn_b200.joint_metadata(cu, T)
    assert not bool(valid)

    def litter():                                            # freed blocks of every size full of NaN
        blocks = [torch.full((1 << n,), float("nan"), device="cuda") for n in range(8, 22) for _ in range(4)]
        del blocks

    litter()
    leaves = [t.clone().requires_grad_(True) for t in ins]
    litter()
    o = torch.ops.tgdn_b200.joint_fwd(*leaves, 0.1, offsets, chunk_map)[0]
    litter()
    dv, = torch.autograd.grad(o, leaves[2], do)
    assert _lib.device_status() == 0
    part = [t[:, :130].contiguous().requires_grad_(True) for t in ins]
    o_part = gdn_joint_call(*part, scale=0.1, cu_seqlens=cu)
    dv_part, = torch.autograd.grad(o_part, part[2], do[:, :130].contiguous())
    for whole, head in ((o, o_part), (dv, dv_part)):
        assert torch.equal(whole[:, :130], head) and bool((whole[:, 130:] == 0).all())


@pytest.mark.parametrize("call", [gdn_joint_call, chunk_gdn_joint, lambda *a: chunk_gdn_joint(*a, checkpoint_tokens=64),
                                  lambda *a: chunk_gdn_joint_segment(*a)[0]], ids=["call", "chunk", "checkpointed", "segment"])
def test_error_of_the_library_in_a_backward(call):
    """Its class is the same as in a forward: a gradient at an address that is no multiple of 16 bytes is refused."""
    leaves = [t.cuda().requires_grad_(True) for t in orc.make_inputs(1, 128, 2, 2, seed=5)]
    do = torch.empty(128 * 2 * 128 + 1, dtype=BF16, device="cuda")[1:].view(1, 128, 2, 128)
    o = call(*leaves)
    with pytest.raises(_lib.TgdnError, match="16-byte aligned"):
        o.backward(do)
    o = call(*leaves)                                        # and the next one is fine
    o.backward(torch.ones_like(o))
    assert _lib.device_status() == 0


def test_decode_takes_the_first_token_of_longer_operands():
    ins = [t.cuda() for t in orc.make_inputs(2, 64, 3, 4, seed=8)]
    first = [t[:, :1].contiguous() for t in ins]
    state = torch.randn(2, 3, 4, 128, 128, device="cuda")
    ref_state = state.clone()
    ref = gdn_joint_decode(*first, ref_state)
    for longer in range(1, 7):
        s = state.clone()
        assert torch.equal(gdn_joint_decode(*[ins[i][:, :5] if i == longer else t for i, t in enumerate(first)], s), ref)
        assert torch.equal(s, ref_state)
    with pytest.raises(ValueError, match="T must be 1"):
        gdn_joint_decode(*[t[:, :2] for t in ins], state)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T,H", [(2, 64, 0), (0, 64, 2), (1, 64, 0)])
def test_core_without_elements_is_refused(B, T, H):
    """(A division by the number of heads on the host would end the process.)"""
    q, k2 = torch.empty(B, T, H, 128, dtype=BF16, device="cuda"), torch.empty(B, T, H, 2, device="cuda")
    ins = [q, q, q, k2, k2, k2, torch.empty(B, T, H, device="cuda")]
    for call in (gdn_joint_call, chunk_gdn_joint, lambda *a: chunk_gdn_joint_segment(*a),
                 lambda *a: chunk_gdn_joint(*[t.clone().requires_grad_(True) for t in a], checkpoint_tokens=64)):
        with pytest.raises(_lib.TgdnError):
            call(*ins)


@pytest.mark.parametrize("B,T,C", [(0, 8, 16), (2, 0, 16), (2, 8, 0), (0, 8, 784), (1, 0, 784)])
def test_convolution_without_elements_is_refused(B, T, C):
    x, w = torch.empty(B, T, C, dtype=BF16, device="cuda"), torch.ones(C, 4, dtype=BF16, device="cuda")
    with pytest.raises(_lib.TgdnError):
        conv_split_act_call(x, w, 0)
    with pytest.raises(_lib.TgdnError):
        torch.ops.tgdn_b200.conv_split_act_bwd(x, x, w, 0, None)
    if C == 784:
        qkv, gates = torch.empty(B, T, 2, 128, dtype=BF16, device="cuda"), torch.empty(B, T, 2, 4, device="cuda")
        with pytest.raises(_lib.TgdnError):
            conv_split_norm_call(x, w, 2, 4)
        with pytest.raises(_lib.TgdnError):
            torch.ops.tgdn_b200.conv_split_norm_bwd(x, w, qkv, qkv, qkv, gates, gates, 2, 4, 1e-6, None)
