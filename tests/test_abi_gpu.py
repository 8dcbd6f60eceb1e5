"""The C ABI on a GPU: the stages called one by one, as include/tgdn.h declares them, give the bits of the package's calls (which reach
the same kernels by another way), and the glue's backward that only the ABI has is checked against the oracle."""
import pytest
import torch

from cute_triadic_gdn_b200 import _lib, chunk_gdn_joint_segment, conv_split_norm_call, gdn_joint_call
from cute_triadic_gdn_b200.gdn_joint import gate_item_floats
from cute_triadic_gdn_b200.joint_packing import chunk_capacity
from oracle import triadic_oracle as orc
from helpers import GRADS

pytestmark = pytest.mark.gpu
BF16, F32 = torch.bfloat16, torch.float32


def call(name, *args):
    """Tensors and None as pointers, everything else as it is, on the current stream."""
    args = [_lib.ptr(a) if a is None or torch.is_tensor(a) else a for a in args]
    _lib.check(getattr(_lib.lib, name)(*args, _lib.stream_of(torch.empty(0, device="cuda"))), name)


def empty(*shape, dtype=BF16):
    return torch.empty(*shape, dtype=dtype, device="cuda").fill_(float("nan"))


def core(ins, do, scale, cu=None, states=None):
    """o and the seven gradients, stage by stage.  `states`: (state_in, grad of the final state) -> the _state entries, and the
    final state and the gradient of the initial one at the end of the result."""
    q, k, v, k2, q2, g, beta = ins
    (B, T, H, _), E = q.shape, k2.shape[-1]
    offsets = cmap = None
    n_docs, NC = 0, T // 64
    if cu is not None:
        n_docs, NC = cu.numel() - 1, chunk_capacity(T, cu.numel() - 1)
        offsets = torch.empty(n_docs + 1, dtype=torch.int32, device="cuda")
        cmap, valid = torch.empty(3, NC, dtype=torch.int32, device="cuda"), torch.empty(1, dtype=torch.bool, device="cuda")
        call("tgdn_metadata", cu, 0, n_docs, T, offsets, cmap, NC, valid)
        assert bool(valid)
    size, items = (B, T, H, E, NC), (B, NC, H)
    NV = 4 if E <= 8 else 8
    gc, AP, Pm = empty(*items, gate_item_floats(E), dtype=F32), empty(*items, 128 * 64), empty(*items, 64 * 64)
    call("tgdn_masks", q, k, k2, q2, g, beta, scale, cmap, *size, gc, AP, Pm)
    o, W, U, h = empty(B, T, H, 128), empty(*items, 64, 128), empty(*items, 64, 128), empty(*items, E, 16, 128, 8)
    fwd = (q, k, v, k2, q2, beta, gc, AP, scale, offsets, cmap, n_docs, *size, o, W, U, h)
    dv, dU, ds = empty(B, T, H, 128), empty(*items, 64, 128), empty(*items, E, 16, 128, 8)
    dkg, dr = empty(*items, NV, 8, 128, 8), empty(*items, NV, 64, E, dtype=F32)
    rec = (q, k, do, k2, q2, beta, gc, AP, Pm, U, scale, offsets, cmap, n_docs, *size, dv, dU, ds, dkg, dr)
    handed = []
    if states is None:
        call("tgdn_fwd", *fwd)
        call("tgdn_bwd_recurrent", *rec)
    else:
        handed = [empty(B, H, E, 128, 128, dtype=F32) for _ in range(2)]
        call("tgdn_fwd_state", *fwd, states[0], handed[0])
        call("tgdn_bwd_recurrent_state", *rec, states[1], handed[1])
    dkq, dd = empty(*items, 16, 128, 8), empty(*items, E, dtype=F32)
    da, dc = empty(*items, 64, E, dtype=F32), empty(*items, 64, E, dtype=F32)
    call("tgdn_bwd_state_grads", q, k, do, dv, h, ds, dkg, k2, q2, gc, scale, cmap, *size, dkq, da, dc, dd)
    dq, dk = empty(B, T, H, 128), empty(B, T, H, 128)
    dk2, dq2, dg = (empty(B, T, H, E, dtype=F32) for _ in range(3))
    dbeta = empty(B, T, H, dtype=F32)
    call("tgdn_bwd_matrix", q, k, do, dU, W, U, AP, k2, q2, beta, gc, dkq, da, dc, dd, dr, scale, cmap, *size, dq, dk, dk2, dq2, dg, dbeta)
    assert _lib.device_status() == 0
    return [o, dq, dk, dv, dk2, dq2, dg, dbeta, *handed]


def same(got, ref, names):
    for name, a, b in zip(names, got, ref):
        assert torch.equal(a, b), name


@pytest.mark.parametrize("B,T,H,E,docs", [(2, 192, 3, E, None) for E in (1, 2, 4, 8, 12, 16)] +      # one wave of narrow blocks
                         [(4, 128, 16, E, None) for E in (1, 2, 4)] +                                 # wide ones
                         [(1, 300, 4, E, [0, 1, 65, 193, 300]) for E in (1, 2, 4, 8, 12, 16)] + [(1, 500, 16, 2, [0, 64, 100, 164, 400, 500])])
def test_core_stages(B, T, H, E, docs):
    ins = [t.cuda() for t in orc.make_inputs(B, T, H, E, seed=60 + E, dist="mild")]
    do = orc.make_grad_output((B, T, H, 128), 7).cuda()
    cu = torch.tensor(docs, dtype=torch.int32).cuda() if docs else None
    leaves = [t.clone().requires_grad_(True) for t in ins]
    o = gdn_joint_call(*leaves, cu_seqlens=cu)
    grads = torch.autograd.grad(o, leaves, do)
    same(core(ins, do, 128 ** -0.5, cu), [o.detach(), *grads], ["o", *GRADS])


@pytest.mark.parametrize("B,H,E", [(1, 2, 1), (1, 2, 4), (1, 2, 8), (1, 2, 12), (1, 2, 16), (4, 16, 1), (4, 16, 2), (4, 16, 4)])
def test_core_stages_with_states_handed_over(B, H, E):
    T = 128
    ins = [t.cuda() for t in orc.make_inputs(B, T, H, E, seed=80 + E, dist="mild")]
    do = orc.make_grad_output((B, T, H, 128), 8).cuda()
    gen = torch.Generator(device="cuda").manual_seed(E)
    state, grad = (0.1 * torch.randn(B, H, E, 128, 128, device="cuda", generator=gen) for _ in range(2))
    leaves = [t.clone().requires_grad_(True) for t in (*ins, state)]
    o, last = chunk_gdn_joint_segment(*leaves[:7], state_in=leaves[7])
    grads = torch.autograd.grad([o, last], leaves, [do, grad])
    same(core(ins, do, 128 ** -0.5, None, (state, grad)), [o.detach(), *grads[:7], last.detach(), grads[7]], ["o", *GRADS, "state", "first"])


@pytest.mark.parametrize("B,T,H,E,docs", [(2, 37, 2, 4, None), (3, 129, 4, 1, None), (1, 200, 3, 12, [0, 1, 5, 70, 133, 200]),
                                          (1, 131, 1, 4, [0, 64, 131]), (1, 333, 2, 16, [0, 7, 8, 9, 333])])
def test_glue_backward_in_two_steps(B, T, H, E, docs):
    """tgdn_glue_bwd_norm, then tgdn_conv_bwd.  Between them the gradient of the convolution's output is rounded to bf16, and the
    convolution takes SiLU' at the rounded pre-activation: twice the tolerances of the plain convolution's backward.  (The package's
    own backward does neither.)"""
    gen = torch.Generator().manual_seed(E + T)
    C = H * (3 * 128 + 2 * E)
    x, w = torch.randn(B, T, C, generator=gen).to(BF16), (0.5 * torch.randn(C, 4, generator=gen)).to(BF16)
    grads = [torch.randn(B, T, H, 128, generator=gen).to(BF16) for _ in range(3)] + [torch.randn(B, T, H, E, generator=gen) for _ in range(2)]
    cu = torch.tensor(docs, dtype=torch.int32) if docs else None
    n_docs = len(docs) - 1 if docs else 0
    xd, wd, gd, cud = x.cuda(), w.cuda(), [g.cuda() for g in grads], None if cu is None else cu.cuda()
    dy, dx, dw = empty(B, T, C), empty(B, T, C), empty(C, 4)
    call("tgdn_glue_bwd_norm", xd, wd, cud, n_docs, B, T, C, T * C, C, H, E, 1e-6, *gd, dy)
    nbytes = _lib.lib.tgdn_conv_bwd_scratch_bytes(B, T, C)
    scratch = empty(nbytes // 4, dtype=F32)
    call("tgdn_conv_bwd", xd, wd, dy, dx, dw, cud, n_docs, B, T, C, T * C, C, T * C, C, 3 * H * 128, scratch, nbytes)
    assert _lib.device_status() == 0
    xr, wr = x.float().requires_grad_(True), w.float().requires_grad_(True)
    torch.autograd.backward(orc.glue_reference(xr, wr, H, E, cu), [g.float() for g in grads])
    assert orc.rel_l2(dx.float().cpu(), xr.grad) < 8e-3
    assert orc.rel_l2(dw.float().cpu(), wr.grad) < 1.6e-2
    xl, wl = xd.clone().requires_grad_(True), wd.clone().requires_grad_(True)
    one = torch.autograd.grad(conv_split_norm_call(xl, wl, H, E, cud), (xl, wl), gd)
    assert orc.rel_l2(dx.float(), one[0].float()) < 8e-3 and orc.rel_l2(dw.float(), one[1].float()) < 1.6e-2
