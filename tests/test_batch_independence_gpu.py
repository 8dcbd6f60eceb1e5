"""What a sequence gets does not depend on what runs beside it: up to four slices the recurrences pick the width of their value blocks by
the number of sequences and heads of the call, and both sides of that switch give the same bits.

Eight rows of sixteen heads are wide (four waves of narrow blocks on 148 SMs, two of wide ones), one row of them or two of their heads
are narrow."""
import pytest
import torch

from cute_triadic_gdn_b200 import HostPipeline, _lib, gdn_joint_call
from oracle import triadic_oracle as orc
from helpers import GRADS

pytestmark = pytest.mark.gpu


def step(ins, do, cu=None):
    leaves = [t.detach().contiguous().requires_grad_(True) for t in ins]
    o = gdn_joint_call(*leaves, cu_seqlens=cu)
    o.backward(do)
    return [o.detach()] + [t.grad for t in leaves]


def same(whole, part, cut):
    for name, a, b in zip(["o"] + list(GRADS), whole, part):
        assert torch.equal(cut(a), b), name


@pytest.mark.parametrize("dist", ["baseline", "mild"])
@pytest.mark.parametrize("E", [1, 2, 4])
def test_rows_and_heads_of_a_wide_batch(E, dist):
    B, T, H = 8, 192, 16
    ins = [t.cuda() for t in orc.make_inputs(B, T, H, E, seed=E, dist=dist)]
    do = orc.make_grad_output((B, T, H, 128), 3).cuda()
    whole = step(ins, do)
    for cut in (lambda t: t[5:6], lambda t: t[:, :, 6:8], lambda t: t[2:4, :, 15:]):
        same(whole, step([cut(t) for t in ins], cut(do).contiguous()), cut)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E", [1, 2, 4])
def test_documents_of_a_wide_packed_row(E):
    docs = [0, 1, 64, 129, 200, 263, 384, 448, 511]
    T, H = docs[-1], 16
    ins = [t.cuda() for t in orc.make_inputs(1, T, H, E, seed=20 + E, dist="mild")]
    do = orc.make_grad_output((1, T, H, 128), 4).cuda()
    whole = step(ins, do, torch.tensor(docs, dtype=torch.int32).cuda())
    for lo, hi in ((0, 2), (2, 3), (5, 8)):
        cut = lambda t: t[:, docs[lo]:docs[hi]]
        cu = torch.tensor([d - docs[lo] for d in docs[lo:hi + 1]], dtype=torch.int32).cuda()
        same(whole, step([cut(t) for t in ins], cut(do).contiguous(), cu), cut)
    assert _lib.device_status() == 0


@pytest.mark.parametrize("E", [2, 4])
def test_host_pipeline_of_a_wide_batch(E):
    B, T, H = 8, 128, 16
    ins = [t.pin_memory() for t in orc.make_inputs(B, T, H, E, seed=40 + E)]
    do = orc.make_grad_output((B, T, H, 128), 5).pin_memory()
    whole = step([t.cuda() for t in ins], do.cuda())
    pipe = HostPipeline(ins, do, slices=B)
    o, grads = pipe.run(ins, do)
    pipe.wait()
    same([t.cpu() for t in whole], [o] + grads, lambda t: t)
    assert _lib.device_status() == 0
