"""The fused gradient kernel against the two stages it joins (state gradients, then matrix gradients), bit by bit, where its roles have to
agree on the course of an item: which slices take a trace (none, all, the first, the last, every other), chunks cut short by a document
end, unused entries of the chunk map, fewer and more items than SMs, and the direct decay path (steep gates, gates above zero)."""
import pytest
import torch

from cute_triadic_gdn_b200 import _lib, gdn_joint_call
from cute_triadic_gdn_b200 import gdn_joint as gj
from cute_triadic_gdn_b200.joint_packing import chunk_capacity, prepare_documents
from oracle import triadic_oracle as orc

pytestmark = pytest.mark.gpu

TRACES = {"none": lambda e, E: False, "all": lambda e, E: True, "first": lambda e, E: e == 0, "last": lambda e, E: e == E - 1,
          "other": lambda e, E: e % 2 == 1}


def repeated(tensors, heads):
    """The same heads again and again, as many as asked for."""
    return [t.cuda().repeat([1, 1, heads // t.shape[2]] + [1] * (t.dim() - 3)) for t in tensors]


def both(ins, do, docs=None, drawn=None):
    q, k, v, k2, q2, g, beta = [t.cuda() for t in ins]
    do, E, scale = do.cuda(), k2.shape[-1], 128 ** -0.5
    cs = tm = None
    if docs is not None:
        cs, tm = prepare_documents((q, k, v, k2, q2, g, beta), torch.tensor(docs, dtype=torch.int32).cuda())
    gc, AP, Pm = gj._run_masks(q, k, k2, q2, g, beta, scale, tm)
    _, h, W, U = gj._run_forward(q, k, v, k2, q2, beta, gc, AP, scale, True, cs, tm)
    dV, dU, ds, dkg, dr = gj._run_reverse(q, k, do, k2, q2, beta, gc, AP, Pm, U, scale, cs, tm)
    one = gj._run_grads(q, k, do, dV, dU, ds, dkg, dr, h, W, U, AP, k2, q2, beta, gc, scale, tm, drawn)
    dkq, da, dc, dd = gj._run_state_grads(q, k, do, dV, h, ds, dkg, k2, q2, gc, scale, tm)
    two = gj._run_matrix(q, k, do, dU, W, U, AP, k2, q2, beta, gc, dkq, da, dc, dd, dr, scale, tm)
    assert _lib.device_status() == 0
    for name, a, b in zip("dq dk dk2 dq2 dg dbeta".split(), one, two):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b), name


@pytest.mark.parametrize("E", [1, 2, 4, 8, 12, 16])
@pytest.mark.parametrize("traces", list(TRACES))
@pytest.mark.parametrize("B,T,H,docs", [(2, 64, 1, None), (2, 640, 16, None), (1, 777, 5, [0, 1, 64, 129, 200, 777])])
def test_one_kernel_is_the_two_stages(E, traces, B, T, H, docs):
    ins = list(orc.make_inputs(B, T, H, E, seed=40 + E, dist="mild"))
    taken = torch.tensor([TRACES[traces](e, E) for e in range(E)])
    ins[5] = torch.where(taken, 0.02, 1.0) * ins[5].abs().neg().clamp(-1.0, -0.4)       # chunk decays above / below 2^-24, none steep
    both(ins, orc.make_grad_output((B, T, H, 128), 9), docs)


@pytest.mark.parametrize("E", [1, 2, 4, 8, 12, 16])
def test_fourteen_items_a_block(E):
    """Items enough for every slot of the blocks' item records to be used several times, every other slice with a trace."""
    ins = list(orc.make_inputs(2, 1024, 8, E, seed=40 + E, dist="mild"))
    ins[5] = torch.where(torch.arange(E) % 2 == 1, 0.02, 1.0) * ins[5].abs().neg().clamp(-1.0, -0.4)
    both(repeated(ins, 64), repeated([orc.make_grad_output((2, 1024, 8, 128), 9)], 64)[0])


@pytest.mark.parametrize("E", [1, 2, 4, 8, 12, 16])
@pytest.mark.parametrize("kind", ["steep", "rising"])
def test_direct_decay_path(E, kind):
    B, T, H = 1, 192, 3
    ins = list(orc.make_inputs(B, T, H, E, seed=50 + E, dist="mild"))
    gen = torch.Generator().manual_seed(E)
    if kind == "steep":
        ins[5] = torch.where(torch.rand(B, T, H, E, generator=gen) < 0.1, torch.full_like(ins[5], -90.0), ins[5])
    else:
        ins[5] = 0.02 * torch.randn(B, T, H, E, generator=gen)
    both(ins, orc.make_grad_output((B, T, H, 128), 10), None)


@pytest.mark.parametrize("E", [2, 4, 8, 12, 16])
@pytest.mark.parametrize("rows", [3, 21, 47, 62])
def test_roundings_behind_a_documents_end_change_nothing(E, rows):
    """The cumulative gate of the rows behind a document's end may rise by a rounding.  That is no reason for the direct decay path, whose
    sums differ in their last bits: a rise there, in a slice without weight, leaves every bit of the gradients as it is."""
    n, H, scale = 9, 16, 128 ** -0.5
    q, k, v, k2, q2, g, beta = [t.cuda() for t in orc.make_inputs(1, n * rows, H, E, seed=60 + E, dist="mild")]
    k2[..., 0] = q2[..., 0] = 0.0
    g = (g * 256).round().clamp(max=-1) / 256                # sums without roundings: gc does not rise by itself
    do = orc.make_grad_output((1, n * rows, H, 128), 11).cuda()
    cs, tm = prepare_documents((q, k, v, k2, q2, g, beta), torch.arange(0, n * rows + 1, rows, dtype=torch.int32, device="cuda"))
    gc, AP, Pm = gj._run_masks(q, k, k2, q2, g, beta, scale, tm)
    _, h, W, U = gj._run_forward(q, k, v, k2, q2, beta, gc, AP, scale, True, cs, tm)
    dV, dU, ds, dkg, dr = gj._run_reverse(q, k, do, k2, q2, beta, gc, AP, Pm, U, scale, cs, tm)
    risen = gc.clone()
    gj.chunk_gates(risen, E)[..., rows, 0] *= 1 - 2.0 ** -20
    assert (gj.chunk_gates(risen, E)[0, :n, :, rows, 0] > gj.chunk_gates(gc, E)[0, :n, :, rows - 1, 0]).all()
    one, other = (gj._run_grads(q, k, do, dV, dU, ds, dkg, dr, h, W, U, AP, k2, q2, beta, c, scale, tm) for c in (gc, risen))
    dkq, da, dc, dd = gj._run_state_grads(q, k, do, dV, h, ds, dkg, k2, q2, risen, scale, tm)
    two = gj._run_matrix(q, k, do, dU, W, U, AP, k2, q2, beta, risen, dkq, da, dc, dd, dr, scale, tm)
    for name, a, b, c in zip("dq dk dk2 dq2 dg dbeta".split(), one, other, two):
        assert torch.isfinite(a.float()).all() and torch.equal(a, b) and torch.equal(a, c), name
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E", [1, 8])
@pytest.mark.parametrize("n,H", [(40, 3), (128, 16)])
def test_unused_tail_of_the_chunk_map_is_not_drawn(E, n, H):
    """Half of the map is unused with documents of one chunk each: the blocks draw the items of the other half, and stop."""
    ins, do = orc.make_inputs(1, 64 * n, H, E, seed=70 + E, dist="mild"), orc.make_grad_output((1, 64 * n, H, 128), 12)
    drawn = torch.zeros(1, dtype=torch.int32, device="cuda")
    both(ins, do, list(range(0, 64 * n + 1, 64)), drawn)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks = min(sms, chunk_capacity(64 * n, n) * H)
    assert drawn.item() == n * H - min(n * H, blocks) + blocks   # (a block's first item is not drawn; each finds the end once)


@pytest.mark.parametrize("E", [1, 2, 4])
@pytest.mark.parametrize("H,more", [(16, 1), (16, 10)])
@pytest.mark.parametrize("T,docs", [(511, [0, 1, 64, 129, 200, 263, 384, 448, 511]), (64, [0, 1, 64]), (512, None)])
def test_short_items_again_and_again(E, T, docs, H, more):
    """With few slices an item is over before a slow warp has looked at its barriers: the same call must give the same bits each time, and
    the same for the same head.  `more`: at least as many items for each of a B200's 148 persistent blocks."""
    ins, do = orc.make_inputs(1, T, H, E, seed=20 + E, dist="mild"), orc.make_grad_output((1, T, H, 128), 4)
    chunks = -(-T // 64) if docs is None else sum(-(-(b - a) // 64) for a, b in zip(docs, docs[1:]))
    heads = H if more == 1 else H * -(-148 * more // (H * chunks))
    *ins, do = repeated([*ins, do], heads)
    cu = None if docs is None else torch.tensor(docs, dtype=torch.int32).cuda()
    first = None
    for _ in range(40):
        leaves = [t.clone().requires_grad_(True) for t in ins]
        grads = torch.autograd.grad(gdn_joint_call(*leaves, cu_seqlens=cu), leaves, do)
        first = first or grads
        assert all(torch.equal(a, b) for a, b in zip(first, grads))
    assert all(torch.equal(a, b) for a, b in zip(first, repeated([t[:, :, :H] for t in first], heads)))
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E", [1, 8])
def test_two_streams_and_a_replayed_graph(E):
    """The counter that items are drawn from belongs to the call: two backwards at a time, and a captured one replayed, give the bits of one."""
    def step(leaves, do):
        return torch.autograd.grad(gdn_joint_call(*leaves), leaves, do)

    calls = []
    for seed in (1, 2):
        ins = repeated(orc.make_inputs(1, 256, 16, E, seed=seed, dist="mild"), 96)
        calls.append(([t.requires_grad_(True) for t in ins], repeated([orc.make_grad_output((1, 256, 16, 128), seed)], 96)[0]))
    alone = [step(*c) for c in calls]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(10):
        got = []
        for s, c in zip(streams, calls):
            with torch.cuda.stream(s):
                got.append(step(*c))
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for x, y in zip(alone, got) for a, b in zip(x, y))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(*calls[0])
    for _ in range(3):
        for t in out:
            t.zero_()
        graph.replay()
        assert all(torch.equal(a, b) for a, b in zip(alone[0], out))
    assert _lib.device_status() == 0
