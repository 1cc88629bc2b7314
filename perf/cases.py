"""Performance cases of the library: what programs do with it, through its public entry points.

A case names one pass:

* ``step``   ``fwd``       ``attention(q, k, v)`` without gradients (inference)
             ``fwd_bwd``   ``attention`` and the gradients of O with respect to q, k, v (ordinary training)
             ``jvp``       ``JVPAttn.fwd_dual`` alone: primal and tangent output (sampling, forward-mode probes)
             ``jvp_bwd_t`` ``fwd_dual`` and the gradients through the tangent output (a loss on the JVP)
             ``jvp_bwd``   ``fwd_dual`` and the gradients through both outputs
             ``hvp``       ``fwd_dual``, and a Hessian-vector product by differentiating ``attention`` twice
* ``api``    how the tangents travel: ``func`` = ``torch.func.jvp``, ``fwad`` = ``torch.autograd.forward_ad`` dual tensors
* ``mask``   ``none``, ``causal``, ``keys`` (key padding, lengths in [L/2, L]), ``bool`` (a random nine tenths of the entries
             False), ``window`` (the L/8 keys on either side of a query, as a boolean mask), ``add`` ({0, -100} at the density
             of ``bool``), ``bias`` (N(0, 1) clipped to [-5, 5])
* ``layout`` ``bhld`` contiguous tensors, ``blhd`` the (B, H, L, D) views of (B, L, H, D) projections

The cotangents are inputs: in a model they arrive from the layers above.
"""
from __future__ import annotations

import torch
import torch.autograd.forward_ad as fwAD

from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention

MASK_CONST = -100.0
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
# products of 2*D flops for each attended (query, key) pair
PRODUCTS = {"fwd": 2, "fwd_bwd": 2 + 5, "jvp": 6, "jvp_bwd_t": 6 + 10, "jvp_bwd": 6 + 12,
            # primal and tangent; O; dq of O (scores, dP, dq); tO along q alone (scores, tS, O, tO); its gradient with
            # respect to q (scores, tS, E, two products)
            "hvp": 6 + 2 + 3 + 4 + 5}


def _case(name, step, dtype, B, H, L, D, mask="none", api="func", layout="bhld", tangent_std=0.1):
    return {"name": name, "step": step, "dtype": dtype, "B": B, "H": H, "L": L, "D": D, "mask": mask, "api": api,
            "layout": layout, "tangent_std": tangent_std}


def listed():
    return [
        # one short sequence batch at inference: the time of a call, not of its arithmetic
        _case("tiny_fwd", "fwd", "bf16", 2, 12, 32, 64),
        # the small fp32 configuration (unit tests, prototyping on small models): launches and host work
        _case("fp32_small", "jvp_bwd", "fp32", 2, 4, 256, 64, tangent_std=1.0),
        # the harness's short sequences: tangents without a gradient, dual tensors
        _case("short_jvp", "jvp", "bf16", 2, 12, 256, 64, api="fwad", tangent_std=1.0),
        # small heads and a length that no tile divides
        _case("d32_ragged", "jvp_bwd", "bf16", 4, 8, 1000, 32, tangent_std=0.1),
        # ordinary training of an encoder-decoder layer: projections' views, causal, ragged length, no tangents
        _case("train_views", "fwd_bwd", "fp16", 3, 12, 1330, 64, mask="causal", layout="blhd"),
        # the key-padding configuration: a batch of sentences, loss on both outputs
        _case("keys_both", "jvp_bwd", "fp16", 8, 12, 1024, 64, mask="keys", tangent_std=1.0),
        # the harness's additive masks, loss on both outputs
        _case("add_both", "jvp_bwd", "bf16", 2, 12, 1024, 64, mask="add", api="fwad", tangent_std=1.0),
        # the harness's boolean masks at its largest length, loss on the tangent
        _case("bool_tangent", "jvp_bwd_t", "bf16", 2, 12, 2048, 64, mask="bool", api="fwad", tangent_std=1.0),
        # the headline configuration: a JVP-consistency training step
        _case("causal_step", "jvp_bwd_t", "bf16", 4, 16, 2048, 64, mask="causal"),
        # local attention over a long sequence, written as a boolean mask
        _case("window_long", "jvp_bwd", "bf16", 1, 8, 4096, 128, mask="window"),
        # the fp32 bias configuration: primal and tangent, and a Hessian-vector product
        _case("fp32_bias_hvp", "hvp", "fp32", 2, 8, 1024, 128, mask="bias", tangent_std=0.5),
        # one GPU's part of the long-sequence configuration
        _case("long_both", "jvp_bwd", "bf16", 1, 16, 8192, 128),
    ]


def _pairs(case):
    B, H, L = case["B"], case["H"], case["L"]
    if case["mask"] == "causal":
        return B * H * L * (L + 1) // 2
    if case["mask"] == "keys":
        return B * H * L * (3 * L // 4)
    if case["mask"] == "window":
        w = L // 8
        return B * H * (L * (2 * w + 1) - w * (w + 1))
    return B * H * L * L  # a random mask leaves no tile of keys out


def _mask_bytes(case):
    per = {"bool": 1, "window": 1, "add": 2, "bias": 2}.get(case["mask"], 0)
    if case["dtype"] == "fp32" and case["mask"] in ("add", "bias"):
        per = 4
    heads = 1 if case["mask"] == "window" else case["B"] * case["H"]
    return per * heads * case["L"] ** 2 + (case["B"] * case["L"] if case["mask"] == "keys" else 0)


def work(case):
    flops = 2 * case["D"] * _pairs(case) * PRODUCTS[case["step"]]
    one = case["B"] * case["H"] * case["L"] * case["D"] * (4 if case["dtype"] == "fp32" else 2)
    # q, k, v, O; with gradients a cotangent and dq, dk, dv; tangents and tO; a second cotangent
    tensors = {"fwd": 4, "fwd_bwd": 8, "jvp": 8, "jvp_bwd_t": 12, "jvp_bwd": 13, "hvp": 8 + 2 + 2}[case["step"]]
    return {"bytes": one * tensors + _mask_bytes(case), "flops": flops}


def draw(rng):
    """One more case: sequence lengths from 32 to 8192 (any even number), every head dimension, data type, mask, step and
    layout of the listed ones, at no more arithmetic than the largest of them."""
    while True:
        L = 2 * round(2 ** rng.uniform(4, 12))
        if rng.random() < 0.5 and L >= 64:
            L -= L % 64  # half of the lengths are the round ones that programs pad to
        case = _case("", rng.choice(["fwd", "fwd_bwd", "jvp", "jvp_bwd_t", "jvp_bwd", "hvp"]),
                     rng.choice(["bf16", "bf16", "fp16", "fp32"]), rng.randint(1, 8), rng.randint(1, 16), L,
                     rng.choice([32, 64, 64, 128, 128]),
                     rng.choice(["none", "none", "causal", "causal", "keys", "bool", "window", "add", "bias"]),
                     rng.choice(["func", "fwad"]), rng.choice(["bhld", "bhld", "blhd"]), rng.choice([0.1, 0.5, 1.0]))
        del case["name"]
        # fp32 products are split into several, and small heads spend more than their products: less arithmetic for these
        most = 8e10 if case["dtype"] == "fp32" else 4e11 if case["D"] == 32 else 2e12
        if work(case)["flops"] <= most and _mask_bytes(case) <= 1 << 28:
            return case


def _make_mask(case, g):
    B, H, L, dev, kind = case["B"], case["H"], case["L"], "cuda", case["mask"]
    if kind in ("none", "causal"):
        return None
    if kind == "keys":
        lens = torch.randint(L // 2, L + 1, (B,), generator=g, device=dev)
        return (torch.arange(L, device=dev)[None, :] < lens[:, None])[:, None, None, :]
    if kind == "window":
        i = torch.arange(L, device=dev)
        return ((i[:, None] - i[None, :]).abs() <= L // 8)[None, None]
    if kind == "bias":
        return torch.randn(B, H, L, L, generator=g, device=dev).clamp_(-5, 5).to(DTYPES[case["dtype"]])
    keep = torch.rand(B, H, L, L, generator=g, device=dev) > 0.9
    keep |= torch.eye(L, dtype=torch.bool, device=dev)  # no row without a key
    return keep if kind == "bool" else torch.where(keep, 0.0, MASK_CONST).to(DTYPES[case["dtype"]])


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, L, D, dtype = case["B"], case["H"], case["L"], case["D"], DTYPES[case["dtype"]]

    def tensor(std=1.0):
        shape = (B, L, H, D) if case["layout"] == "blhd" else (B, H, L, D)
        x = (torch.randn(shape, generator=g, device="cuda") * std).to(dtype)
        return x.transpose(1, 2) if case["layout"] == "blhd" else x

    state = {"step": case["step"], "api": case["api"], "causal": case["mask"] == "causal"}
    state["primals"] = tuple(tensor() for _ in range(3))
    state["tangents"] = tuple(tensor(case["tangent_std"]) for _ in range(3))
    state["cotangents"] = tuple(tensor().contiguous() for _ in range(2))
    state["direction"] = tensor()
    state["mask"] = _make_mask(case, g)
    if case["step"] in ("fwd_bwd", "jvp_bwd_t", "jvp_bwd"):
        for x in state["primals"]:
            x.requires_grad_()
    return state


def _dual(state):
    mask, causal = state["mask"], state["causal"]
    if state["api"] == "func":
        return torch.func.jvp(lambda q, k, v: JVPAttn.fwd_dual(q, k, v, attn_mask=mask, causal=causal), state["primals"],
                              state["tangents"])
    with fwAD.dual_level():
        out = JVPAttn.fwd_dual(*(fwAD.make_dual(p, t) for p, t in zip(state["primals"], state["tangents"])), attn_mask=mask,
                               causal=causal)
        return tuple(fwAD.unpack_dual(out))


def run(state):
    step = state["step"]
    go, gto = state["cotangents"]
    if step == "fwd":
        with torch.no_grad():
            return attention(*state["primals"], attn_mask=state["mask"], causal=state["causal"])
    if step == "fwd_bwd":
        o = attention(*state["primals"], attn_mask=state["mask"], causal=state["causal"])
        return (o.detach(), *torch.autograd.grad(o, state["primals"], go))
    o, to = _dual(state)
    if step == "jvp":
        return o, to
    if step == "jvp_bwd_t":
        return (o.detach(), to.detach(), *torch.autograd.grad(to, state["primals"], gto))
    if step == "jvp_bwd":
        return (o.detach(), to.detach(), *torch.autograd.grad((o, to), state["primals"], (go, gto)))
    q = state["primals"][0].detach().requires_grad_()
    o1 = attention(q, *state["primals"][1:], attn_mask=state["mask"], causal=state["causal"])
    (dq,) = torch.autograd.grad(o1, q, go, create_graph=True)
    (hq,) = torch.autograd.grad(dq, q, state["direction"])
    return o, to, dq.detach(), hq


def tolerance(case):
    # fp32: three TF32 products of a high and a low part each; 16 bits: outputs and the probabilities between the two
    # products are rounded to the data type (8 and 11 significant bits)
    return {"rel": {"fp32": 1e-5, "bf16": 1e-2, "fp16": 2e-3}[case["dtype"]]}
