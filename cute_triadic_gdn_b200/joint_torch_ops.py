"""Triadic GDN behind torch.library operators, so that torch.compile records one opaque node per call.

Mirrors cute_triadic_gdn/ops/joint_torch_ops.py:8-95 of the reference: one forward op that returns the output and the
tensors the backward needs, one backward op, fake (meta) implementations, autograd registration with a single read of
the saved tensors and without materialising zero gradients for the auxiliary outputs, and `gdn_joint_call`.
The operators live in the namespace `tgdn_b200` so that both packages can be imported into one process.  They and their
autograd are registered natively (csrc/tgdn_torch.cpp); the fake implementations are here.
"""
from __future__ import annotations

import torch

from . import _lib
from .gdn_joint import CHUNK, gate_item_floats
from .joint_packing import prepare_documents


@torch.library.register_fake("tgdn_b200::joint_fwd")
def _joint_fwd_fake(q, k, v, k2, q2, g, beta, scale, chunk_starts=None, token_map=None, covered=False):
    B, T, H, D = q.shape
    E = k2.shape[-1]
    NC = token_map.shape[1] if token_map is not None else T // CHUNK
    return [torch.empty_like(v), g.new_empty(B, NC, H, gate_item_floats(E)), q.new_empty(B, NC, H, 128 * 64),
            q.new_empty(B, NC, H, 64 * 64), q.new_empty(B, NC, H, E, 16, 128, 8), v.new_empty(B, NC, H, CHUNK, 128),
            v.new_empty(B, NC, H, CHUNK, 128)]


@torch.library.register_fake("tgdn_b200::joint_bwd")
def _joint_bwd_fake(saved, do, scale, chunk_starts=None, token_map=None, covered=False):
    q, k, k2, q2, g, beta = saved[:6]
    return [torch.empty_like(q), torch.empty_like(k), torch.empty_like(do), torch.empty_like(k2), torch.empty_like(q2),
            torch.empty_like(g), torch.empty_like(beta)]


def gdn_joint_call(q, k, v, k2, q2, g, beta, scale=None, cu_seqlens=None):
    """Triadic GDN for training, as ONE operator node (so that torch.compile does not look inside): same arguments and
    packed-row rules as `chunk_gdn_joint`.  Unlike that function this one accepts non-contiguous inputs (it makes them
    contiguous), like the reference's entry of the same name (ops/joint_torch_ops.py:83-95).  sm_100 only,
    E in {1, 2, 4, 8, 12, 16}, head dimension 128."""
    if not torch.compiler.is_compiling():              # the same steps natively
        return _lib.host.joint_call(q, k, v, k2, q2, g, beta, None if scale is None else float(scale), cu_seqlens)
    seven = [t.contiguous() for t in (q, k, v, k2, q2, g, beta)]
    if scale is None:
        scale = seven[0].shape[-1] ** -0.5
    chunk_starts = token_map = None
    if cu_seqlens is not None:
        chunk_starts, token_map = prepare_documents(seven, cu_seqlens)
    return torch.ops.tgdn_b200.joint_fwd(*seven, float(scale), chunk_starts, token_map, True)[0]
