"""Performance cases of the Triadic Gated DeltaNet package: what is timed, on which inputs, through which entry points.

    listed()            the named cases
    draw(rng)           one more case of the same ranges
    prepare(case, seed) inputs on the GPU, made from the seed
    run(state)          one pass through the public entry points
    work(case)          bytes and FLOPs of one pass that no implementation can do without
    tolerance(case)     how far another correct implementation at the same precision may be off

A case is a dict of plain values.  `kind` selects the path:

    train      gdn_joint_call forward and backward for all seven inputs (one step of a layer's core)
    recompute  chunk_gdn_joint(checkpoint_tokens=S) forward and backward (training where memory is short)
    prefill    chunk_gdn_joint without gradients; `state`: the final state is handed out for the decode that follows
    decode     gdn_joint_decode, one token per sequence on a resident f32 state
    conv       conv_split_act_call forward and backward (the pre-pass by itself)
    layer      conv_split_norm_call into gdn_joint_call, forward and backward (pre-pass and core of one layer)

`docs` cuts the one row of a packed case into documents: "equal:N", or "lognormal:M" (lengths from a lognormal with
median M and sigma 1, the last one truncated).  `gates`: "strong" is g = -softplus(N(0,1)); "mild" is the slow decay of
trained layers, g = -softplus(N(0,1) + 3) times a rate of its own per head and slice in [0, 0.2].
"""
import math
import os

import numpy as np
import torch

from cute_triadic_gdn_b200 import (chunk_gdn_joint, conv_split_act_call, conv_split_norm_call, gdn_joint_call,
                                   gdn_joint_decode)

SLICES = (1, 2, 4, 8, 12, 16)


def _case(kind, B, T, H, E, docs="", gates="strong", **more):
    return dict({"kind": kind, "B": B, "T": T, "H": H, "E": E, "docs": docs, "gates": gates}, **more)


def listed():
    cases = {
        # the smallest configuration: plain gated DeltaNet (one slice), where launches and host work are what counts
        "train_small": _case("train", 2, 256, 4, 1),
        # inference forward of a mid-size model, dense batch, nothing saved
        "prefill_dense": _case("prefill", 4, 4096, 16, 4, state=False),
        # prompts of unequal length packed into one row, their states kept for decoding; lengths are not whole chunks
        "prefill_ragged": _case("prefill", 1, 5003, 16, 12, docs="lognormal:600", gates="mild", state=True),
        # the headline training step
        "train_large": _case("train", 8, 8192, 32, 8),
        # one rank's share of it when the heads are spread over eight GPUs, with the slow decays of a trained layer
        "train_shard": _case("train", 8, 8192, 4, 8, gates="mild"),
        # documents of lognormal length packed into one long row, sixteen slices
        "train_packed": _case("train", 1, 131072, 16, 16, docs="lognormal:2048"),
        # pre-pass and core of one layer on a packed row of eight documents
        "layer_packed": _case("layer", 1, 32768, 32, 12, docs="equal:8"),
        # training with the chunk states recomputed in the backward
        "train_recompute": _case("recompute", 4, 4096, 16, 2, gates="mild", checkpoint=1024),
        # the convolution pre-pass by itself at the channel count of that layer
        "conv_large": _case("conv", 1, 32768, 32, 12, docs="equal:8"),
        # a short batch whose channel count is not a multiple of eight (five heads, one slice)
        "conv_odd": _case("conv", 3, 1000, 5, 1),
        # decode: one user, and a full batch of them
        "decode_one": _case("decode", 1, 1, 32, 8, gates="mild"),
        "decode_batch": _case("decode", 32, 1, 32, 8, gates="mild"),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "prefill", "prefill", "layer", "recompute", "conv", "decode"])
    E = rng.choice(SLICES)
    H = _log_int(rng, 1, 32)
    gates = rng.choice(["strong", "mild"])
    if kind == "decode":
        return _case(kind, _log_int(rng, 1, max(1, min(128, 8192 // (H * E)))), 1, H, E, gates=gates)
    if kind == "layer" and H * E % 4:                    # the fused pre-pass takes channel counts that are multiples of eight
        H *= 4 // math.gcd(H * E, 4)
    most = {"train": 1 << 24, "prefill": 1 << 24, "layer": 1 << 23, "recompute": 1 << 23, "conv": 1 << 23}[kind]
    tokens = _log_int(rng, 64, max(64, min(131072, most // (H * max(E, 4)))))
    if kind != "recompute" and rng.random() < 0.5:
        docs = rng.choice(["equal:%d" % max(1, min(tokens, _log_int(rng, 1, 64))), "lognormal:%d" % _log_int(rng, 100, 4000)])
        B, T = 1, tokens
    else:
        docs = ""
        B = _log_int(rng, 1, 16)
        T = max(1, tokens // B) if kind in ("conv", "layer") else 64 * max(1, tokens // (64 * B))
        if kind == "layer":
            T = 64 * max(1, T // 64)
    more = {}
    if kind == "train":
        more["save_masks"] = rng.random() < 0.75
    if kind == "recompute":
        more["checkpoint"] = 64 * max(1, T // (64 * _log_int(rng, 2, 16)))
    if kind == "prefill":
        more["state"] = rng.random() < 0.5
    return _case(kind, B, T, H, E, docs, gates, **more)


def _offsets(case):
    T = case["T"]
    how, n = case["docs"].split(":")
    if how == "equal":
        n = int(n)
        return [i * T // n for i in range(n + 1)]
    rng, cu = np.random.default_rng(31), [0]
    while cu[-1] < T:
        cu.append(min(T, cu[-1] + max(1, int(round(float(rng.lognormal(math.log(int(n)), 1.0)))))))
    return cu


def _channels(case):
    return case["H"] * (3 * 128 + 2 * case["E"])


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case = case
    kind, B, T, H, E = (case[n] for n in ("kind", "B", "T", "H", "E"))
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev).manual_seed(int(seed))
    randn = lambda *shape: torch.randn(*shape, generator=gen, device=dev)
    rand = lambda *shape: torch.rand(*shape, generator=gen, device=dev)
    norm = lambda t: t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6)
    bf16 = torch.bfloat16
    s.cu = None
    if case["docs"]:
        s.cu = torch.tensor(_offsets(case), dtype=torch.int32, device=dev)

    def core():
        q, k = norm(randn(B, T, H, 128)).to(bf16), norm(randn(B, T, H, 128)).to(bf16)
        if case["gates"] == "mild":
            v = (0.5 * randn(B, T, H, 128)).to(bf16)
            k2, q2 = (norm(torch.nn.functional.softplus(randn(B, T, H, E))) for _ in range(2))
        else:
            v = randn(B, T, H, 128).to(bf16)
            k2, q2 = norm(randn(B, T, H, E)), norm(randn(B, T, H, E))
        return q, k, v, k2, q2

    def gates():
        if case["gates"] == "mild":
            g = -torch.nn.functional.softplus(randn(B, T, H, E) + 3.0) * rand(H, E) * 0.2
        else:
            g = -torch.nn.functional.softplus(randn(B, T, H, E))
        return g, torch.sigmoid(randn(B, T, H))

    if kind in ("conv", "layer"):
        C = _channels(case)
        s.x = randn(B, T, C).to(bf16).requires_grad_()
        s.w = (0.5 * randn(C, 4)).to(bf16).requires_grad_()
        if kind == "conv":
            s.dy = randn(B, T, C).to(bf16)
        else:
            s.g, s.beta = (t.requires_grad_() for t in gates())
            s.do = randn(B, T, H, 128).to(bf16)
    else:
        s.inputs = [*core(), *gates()]
        if kind in ("train", "recompute"):
            s.inputs = [t.requires_grad_() for t in s.inputs]
            s.do = randn(B, T, H, 128).to(bf16)
        if kind == "decode":
            s.resident = 0.1 * randn(B, H, E, 128, 128)
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "decode":
        with torch.no_grad():
            o = gdn_joint_decode(*s.inputs, s.resident)
        return o, s.resident
    if kind == "prefill":
        with torch.no_grad():
            return chunk_gdn_joint(*s.inputs, cu_seqlens=s.cu, output_final_state=case["state"])
    if kind == "conv":
        y = conv_split_act_call(s.x, s.w, 3 * case["H"] * 128, s.cu)
        return (y.detach(), *torch.autograd.grad(y, (s.x, s.w), s.dy))
    if kind == "layer":
        qkv = conv_split_norm_call(s.x, s.w, case["H"], case["E"], s.cu)
        o = gdn_joint_call(*qkv, s.g, s.beta, cu_seqlens=s.cu)
        return (o.detach(), *torch.autograd.grad(o, (s.x, s.w, s.g, s.beta), s.do))
    if kind == "recompute":
        o = chunk_gdn_joint(*s.inputs, checkpoint_tokens=case["checkpoint"])
    else:
        # the switch that a user sets in the environment: keep the chunk operators for the backward, or form them again
        os.environ["GJ_SAVE_MASKS"] = "1" if case.get("save_masks", True) else "0"
        o = gdn_joint_call(*s.inputs, cu_seqlens=s.cu)
    return (o.detach(), *torch.autograd.grad(o, s.inputs, s.do))


def work(case):
    kind, B, T, H, E = (case[n] for n in ("kind", "B", "T", "H", "E"))
    rows = B * T * H                                    # (token, head) pairs
    tile, gate, unit = 256, 4 * E, 16384                # bytes of a bf16 row of 128, of an f32 row of E; FLOPs of a 64-row product per row
    state = E * 128 * 128
    if kind == "decode":
        return {"bytes": B * H * (8 * state + 4 * tile + 3 * gate + 4), "flops": B * H * 8 * state}
    if kind == "prefill":
        sequences = len(_offsets(case)) - 1 if case["docs"] else B
        return {"bytes": rows * (4 * tile + 3 * gate + 4) + (4 * state * H * sequences if case["state"] else 0),
                "flops": rows * (4 + 6 * E) * unit}
    pre_pass = {"bytes": 10 * B * T * _channels(case), "flops": 50 * B * T * _channels(case)}
    if kind == "conv":
        return pre_pass
    core = {"bytes": rows * (8 * tile + 6 * gate + 8), "flops": rows * (15 + 18 * E) * unit}
    if kind == "layer":
        # x is read and dx written; q, k, v, k2, q2 and their gradients need not leave the chip
        return {"bytes": 4 * B * T * _channels(case) + rows * (2 * tile + 2 * gate + 8), "flops": core["flops"] + pre_pass["flops"]}
    return core


def tolerance(case):
    # bf16 operands of chained products with f32 sums: each rounding is 2^-9, a result collects several of them
    if case["kind"] in ("decode", "conv"):
        return {"rel": 4e-3, "max": 3e-2}               # f32 arithmetic, one rounding to bf16
    return {"rel": 1e-2, "max": 0.3}
