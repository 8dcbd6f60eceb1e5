"""Both sides of the size rules by which the library picks a kernel variant, at the sizes where they can go wrong."""
import pytest
import torch

from cute_triadic_gdn_b200 import _lib, chunk_gdn_joint, chunk_gdn_joint_segment, conv_split_act_call, gdn_joint_call
from oracle import triadic_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("E", [1, 2, 4])
@pytest.mark.parametrize("docs", [None, [0, 1, 64, 129, 200, 263, 384]])
def test_wide_value_blocks_of_the_forward(E, docs):
    """Enough sequences for more than one wave of narrow value blocks: the 64-column variants run, dense and with chunks cut
    short by document ends, the forward also with the state handed in and out."""
    B, T, H = (1, 384, 16) if docs else (6, 128, 16)
    ins = [t.cuda() for t in orc.make_inputs(B, T, H, E, seed=70 + E, dist="mild")]
    do = orc.make_grad_output((B, T, H, 128), 5)
    cu = torch.tensor(docs, dtype=torch.int32) if docs else None
    leaves = [t.clone().requires_grad_(True) for t in ins]
    o = gdn_joint_call(*leaves, cu_seqlens=None if cu is None else cu.cuda())
    o.backward(do.cuda())
    o_ref, g_ref = orc.reference_with_grads(orc.chunk_reference, [t.cpu() for t in ins], do, cu_seqlens=cu, dtype=torch.float32)
    assert _lib.device_status() == 0
    assert orc.rel_l2(o.detach().float().cpu(), o_ref) < 1e-2
    for name, leaf, ref in zip("q k v k2 q2 g beta".split(), leaves, g_ref):
        assert orc.rel_l2(leaf.grad.float().cpu(), ref) < 2e-2, name
    if docs is None:                                   # the two halves of the row, chained by the state, are the whole row
        with torch.no_grad():
            _, s_all = chunk_gdn_joint(*ins, output_final_state=True)
            o1, s1 = chunk_gdn_joint(*[t[:, :64].contiguous() for t in ins], output_final_state=True)
            o2, s2 = chunk_gdn_joint(*[t[:, 64:].contiguous() for t in ins], initial_state=s1, output_final_state=True)
        assert torch.equal(torch.cat([o1, o2], 1), o.detach()) and torch.equal(s2, s_all)


@pytest.mark.parametrize("E", [1, 2, 4, 8, 12, 16])
@pytest.mark.parametrize("H", [3, 4, 16])                  # beta rows by loads, as tiles of four heads, wide blocks up to four slices
def test_saved_and_unsaved_forward_and_ragged_chunks(E, H):
    """The forward with and without saved tensors (other splits of the block up to eight slices) agree bitwise; whole chunks leave the
    recurrences as tiles, chunks cut short by a document end row by row."""
    docs = [0, 1, 64, 128, 191, 256]
    ins = [t.cuda() for t in orc.make_inputs(1, 256, H, E, seed=90 + E, dist="mild")]
    do = orc.make_grad_output((1, 256, H, 128), 6)
    cu = torch.tensor(docs, dtype=torch.int32)
    with torch.no_grad():                              # nothing is saved here; gdn_joint_call always saves
        plain = chunk_gdn_joint(*ins, cu_seqlens=cu.cuda())
        stated, _ = chunk_gdn_joint(*ins, cu_seqlens=cu.cuda(), output_final_state=True)
    leaves = [t.clone().requires_grad_(True) for t in ins]
    o = gdn_joint_call(*leaves, cu_seqlens=cu.cuda())
    o.backward(do.cuda())
    assert _lib.device_status() == 0 and torch.equal(plain, o.detach()) and torch.equal(stated, plain)
    o_ref, g_ref = orc.reference_with_grads(orc.chunk_reference, [t.cpu() for t in ins], do, cu_seqlens=cu, dtype=torch.float32)
    assert orc.rel_l2(o.detach().float().cpu(), o_ref) < 1e-2
    for name, leaf, ref in zip("q k v k2 q2 g beta".split(), leaves, g_ref):
        assert orc.rel_l2(leaf.grad.float().cpu(), ref) < 2e-2, name


@pytest.mark.parametrize("E", [1, 2, 4])
def test_wide_value_blocks_with_states_handed_over(E):
    """64 sequences and heads: recomputation in segments (read and written in place, the last one shorter) and segments chained by
    hand, both with the state and its gradient handed from one to the next, are the plain call."""
    B, T, H = 4, 320, 16
    ins = [t.cuda() for t in orc.make_inputs(B, T, H, E, seed=110 + E, dist="mild")]
    do = orc.make_grad_output((B, T, H, 128), 7).cuda()

    def step(call):
        leaves = [t.clone().requires_grad_(True) for t in ins]
        o = call(*leaves)
        return [o.detach(), *torch.autograd.grad(o, leaves, do)]

    def chained(*leaves):
        state, outs = None, []
        for lo, hi in ((0, 64), (64, 256), (256, T)):
            o, state = chunk_gdn_joint_segment(*[t[:, lo:hi].contiguous() for t in leaves], state_in=state)
            outs.append(o)
        return torch.cat(outs, 1)

    ref = step(gdn_joint_call)
    for call in (lambda *a: chunk_gdn_joint(*a, checkpoint_tokens=64), lambda *a: chunk_gdn_joint(*a, checkpoint_tokens=192), chained):
        for name, a, b in zip("o q k v k2 q2 g beta".split(), step(call), ref):
            assert torch.equal(a, b), name
    assert _lib.device_status() == 0


@pytest.mark.parametrize("B,T,C,act,docs", [
    (2, 37, 1930, 1920, None),                         # 4-byte rows
    (1, 150, 77, 40, [0, 1, 3, 64, 65, 150]),          # 2-byte rows, SiLU ends inside a warp's channels
    (1, 130, 516, 516, [0, 127, 128, 130]),            # 8-byte rows
    (1, 3, 130, 0, None),
    (1, 777, 264, 100, [0, 2, 48, 49, 95, 96, 97, 700, 777]),   # whole 16-byte pieces, documents that start at the edges of runs
    (3, 97, 128, 128, None),
])
def test_convolution_rows_of_every_alignment(B, T, C, act, docs):
    g = torch.Generator().manual_seed(T + C)
    x = torch.randn(B, T, C, generator=g).to(torch.bfloat16)
    w = (0.5 * torch.randn(C, 4, generator=g)).to(torch.bfloat16)
    dy = torch.randn(B, T, C, generator=g).to(torch.bfloat16)
    cu = torch.tensor(docs, dtype=torch.int32) if docs else None
    y_ref = orc.conv_reference(x, w, act, cu)
    dx_ref, dw_ref = orc.conv_reference_backward(x, w, act, dy, cu)
    wide = torch.zeros(B, T, C + 3, dtype=torch.bfloat16, device="cuda")
    wide[..., 1:C + 1] = x.cuda()
    outs = []
    for xg in (x.cuda(), wide[..., 1:C + 1]):          # contiguous, and rows of a wider tensor at an odd address
        xg, wg = xg.detach().requires_grad_(True), w.cuda().requires_grad_(True)
        y = conv_split_act_call(xg, wg, act, None if cu is None else cu.cuda())
        outs.append((y.detach(), *torch.autograd.grad(y, (xg, wg), dy.cuda())))
        assert _lib.device_status() == 0
        assert orc.rel_l2(outs[-1][0].float().cpu(), y_ref.float()) < 2e-3
        assert orc.rel_l2(outs[-1][1].float().cpu(), dx_ref.float()) < 4e-3
        assert orc.rel_l2(outs[-1][2].float().cpu(), dw_ref.float()) < 8e-3
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
