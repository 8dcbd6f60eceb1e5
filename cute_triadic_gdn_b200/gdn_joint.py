"""Triadic Gated DeltaNet: `chunk_gdn_joint`, the plain autograd entry, and the kernel pipeline behind it.

Mirrors the operator layer of the reference, cute_triadic_gdn/ops/gdn_joint.py: `_check` (:235-249), the forward
pipeline `_cute_forward` (:144-164), the autograd function `_JointCute` (:201-232), the GJ_SAVE_MASKS switch
(:167-198) and `chunk_gdn_joint` (:252-278).  The device work is the C ABI of libtgdn_b200 (include/tgdn.h); checks,
autograd and launches are in csrc/tgdn_torch.cpp, so that a call costs the host little more than its kernel launches.

    S_e <- exp(g_te) S_e ;  S <- S + beta_t kappa_t (v_t - S^T kappa_t)^T ;  o_t = S^T (q2_t (x) q_t) * scale

Inputs (contiguous, one CUDA device): q, k, v (B,T,H,128) bf16; k2, q2, g (B,T,H,E) f32; beta (B,T,H) f32;
E in {1,2,4,8,12,16}.  Without cu_seqlens T % 64 == 0; with cu_seqlens B = 1 and the state restarts at every document.
"""
from __future__ import annotations

from . import _lib

CHUNK = 64


def gate_item_floats(E):
    """Floats per (batch row, chunk, head) of the gate tensor: gc, a, r, c as 64 x E blocks, then d padded to 16 (include/tgdn.h)."""
    return 4 * CHUNK * E + 16


def chunk_gates(gc, E):
    """The cumulative log gate (B, NC, H, 64, E) as a view of the gate tensor that tgdn_masks writes."""
    return gc[..., :CHUNK * E].unflatten(-1, (CHUNK, E))


# The stages one by one (csrc/tgdn_torch.cpp), for the tests and the benchmark; the calls below run them natively in one go.
def _run_masks(q, k, k2, q2, g, beta, scale, token_map):
    """(gc, AP, Pm) of every chunk.  gc holds the cumulative log gate and the gate factors, AP = [A; Pm A] operand image,
    Pm image; see include/tgdn.h."""
    return _lib.host.run_masks(q, k, k2, q2, g, beta, float(scale), token_map)


def _run_forward(q, k, v, k2, q2, beta, gc, AP, scale, save, chunk_starts=None, token_map=None, state_in=None,
                 state_out=None):
    """Forward recurrence: (o, h, W, U); h, W, U are None unless save.  state_in / state_out: optional f32
    (sequences, H, E, 128, 128) tensors holding the recurrent state before the first and after the last token."""
    return _lib.host.run_forward(q, k, v, k2, q2, beta, gc, AP, float(scale), save, chunk_starts, token_map, state_in, state_out)


def _kernel_forward(q, k, v, k2, q2, g, beta, scale, save, chunk_starts=None, token_map=None):
    """masks -> forward recurrence.  Returns (o, gc, AP, Pm, h, W, U); h, W, U are None unless save."""
    gc, AP, Pm = _run_masks(q, k, k2, q2, g, beta, scale, token_map)
    o, h, W, U = _run_forward(q, k, v, k2, q2, beta, gc, AP, scale, save, chunk_starts, token_map)
    return o, gc, AP, Pm, h, W, U


def _run_reverse(q, k, do, k2, q2, beta, gc, AP, Pm, U, scale, chunk_starts=None, token_map=None, grad_state_in=None,
                 grad_state_out=None):
    """Reverse recurrence: (dV, dU, ds, dkg, dr).  ds is written only for slices whose chunk decay matters to dg.
    grad_state_in / grad_state_out: optional f32 (sequences, H, E, 128, 128) tensors, dL/dS after the last and before the
    first token (the hand-off between segments of one sequence)."""
    return _lib.host.run_reverse(q, k, do, k2, q2, beta, gc, AP, Pm, U, float(scale), chunk_starts, token_map, grad_state_in,
                                 grad_state_out)


def _run_state_grads(q, k, do, dV, h, ds, dkg, k2, q2, gc, scale, token_map=None):
    """State gradients: (dkq, da, dc, dd)."""
    return _lib.host.run_state_grads(q, k, do, dV, h, ds, dkg, k2, q2, gc, float(scale), token_map)


def _run_matrix(q, k, do, dU, W, U, AP, k2, q2, beta, gc, dkq, da, dc, dd, dr, scale, token_map=None):
    """Matrix gradients, mask gradients and final assembly: (dq, dk, dk2, dq2, dg, dbeta)."""
    return _lib.host.run_matrix(q, k, do, dU, W, U, AP, k2, q2, beta, gc, dkq, da, dc, dd, dr, float(scale), token_map)


def _run_grads(q, k, do, dV, dU, ds, dkg, dr, h, W, U, AP, k2, q2, beta, gc, scale, token_map=None, next_item=None):
    """State and matrix gradients in one kernel, as the backward runs them: (dq, dk, dk2, dq2, dg, dbeta), bitwise those of the two
    stages above.  next_item: optional int32 zero that the kernel counts the items drawn in."""
    return _lib.host.run_grads(q, k, do, dV, dU, ds, dkg, dr, h, W, U, AP, k2, q2, beta, gc, float(scale), token_map, next_item)


def chunk_gdn_joint_segment(q, k, v, k2, q2, g, beta, state_in=None, scale=None):
    """One segment of longer sequences, differentiable through the state: returns (o, state_out).  `state_in` (None:
    zero) and `state_out` are f32 (B, H, E, 128, 128), S_e as [key row][value column]; gradients flow into `state_in`
    and out of `state_out`, so that segments chained by their states (on one GPU or, with the states sent between
    ranks, on several: `context_parallel.py`) give the outputs and gradients of the unsplit sequences.  T must be a
    multiple of 64; dense rows only."""
    return _lib.host.joint_segment(q, k, v, k2, q2, g, beta, state_in, None if scale is None else float(scale))


def chunk_gdn_joint(q, k, v, k2, q2, g, beta, scale=None, cu_seqlens=None, reference=False, *, initial_state=None,
                    output_final_state=False, checkpoint_tokens=None):
    """Triadic GDN with autograd for all seven tensor inputs, on the sm_100a kernels.

    Inference that continues a sequence (no counterpart in the reference, whose forward always starts from zero):
    `initial_state` is an f32 (sequences, H, E, 128, 128) tensor, sequences = batch rows or documents, holding S_e as
    [key row][value column]; with `output_final_state=True` the call returns (o, final_state) in the same form.  Both are
    forward-only: they are rejected when a gradient is required.

    With cu_seqlens the inputs are one packed row (1, T, ...): contiguous int32/int64 CUDA offsets that start at 0,
    end at T and strictly increase; document lengths are arbitrary and the state resets at every document start.
    `checkpoint_tokens=S` (training, dense rows): backward state recomputation.  Only the inputs and the f32 state every
    S tokens are kept; the backward recomputes each segment's forward before differentiating it (bitwise the same results,
    one more forward pass, the per-chunk saved tensors of one segment at a time instead of the whole sequence).
    `reference=True` asked the reference package for its torch pipeline; this package ships kernels only (its CPU
    restatement of that pipeline lives with the tests), so the flag is rejected instead of silently running something else.
    """
    if reference:
        raise NotImplementedError("reference=True: this package has no torch fallback; the CPU oracle used by the "
                                  "tests is oracle/triadic_oracle.py")
    o, final = _lib.host.chunk_joint(q, k, v, k2, q2, g, beta, None if scale is None else float(scale), cu_seqlens, initial_state,
                                     bool(output_final_state), None if checkpoint_tokens is None else int(checkpoint_tokens))
    return (o, final) if output_final_state else o


def gdn_joint_decode(q, k, v, k2, q2, g, beta, state, scale=None):
    """One token per sequence on a resident state (decode).  No counterpart in the reference.

    q, k, v: bf16 (B, 1, H, 128) or (B, H, 128); k2, q2, g: f32 (B, 1, H, E) or (B, H, E); beta: f32 (B, 1, H) or (B, H);
    `state`: contiguous f32 (B, H, E, 128, 128), the form `chunk_gdn_joint(..., output_final_state=True)` returns; it is
    updated IN PLACE.  Returns o in the shape of v.  Forward only."""
    return _lib.host.decode(q, k, v, k2, q2, g, beta, state, None if scale is None else float(scale))
