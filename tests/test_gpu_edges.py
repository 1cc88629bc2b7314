"""GPU tests at the edges of the dispatch: head dimension 32 on the D = 64 tensor-core kernels, masks whose rows do not
fill 16-byte pieces, the forms of the register-tiled kernels, the range of fp32, gradients that nobody asked for, and what a
call takes of memory and of the interpreter."""
import ctypes
import pathlib
import subprocess
import sys
import threading
import time

import pytest
import torch

import jvp_flash_attention_b200.jvp_attention as ja
from jvp_flash_attention_b200 import _lib
from oracle import jvp_attention_oracle as orc
from tests import _oracle_launchers as stand_in

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DT = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _inputs(B, H, L, D, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    ts = [torch.randn(B, H, L, D, generator=g) for _ in range(8)]
    for i in (3, 4, 5):  # small tangents: |tO| stays where the spacing of bfloat16 is below the tolerance
        ts[i] = ts[i] * 0.1
    return [t.to(dtype) for t in ts]


def _mask(kind, B, H, L, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    if kind == "keys":
        lens = torch.randint(1, L + 1, (B,), generator=g)
        return (torch.arange(L)[None, :] < lens[:, None])[:, None, None, :]
    if kind == "bool":
        return (torch.rand(B, 1, L, L, generator=g) > 0.7) | torch.eye(L, dtype=torch.bool)
    if kind == "window":
        i = torch.arange(L)
        return ((i[:, None] - i[None, :]).abs() <= 40)[None, None]
    if kind == "bias":
        return torch.randn(B, H, L, L, generator=g).clamp(-5, 5).to(dtype)
    return None


def _check(B, H, L, D, dt, kind, cot, seed=0, fp32_bound=1e-5):
    """O, tO and the gradients through the asked-for outputs against the float64 oracle: 1e-5 of the largest entry for
    fp32 (every product as three, on TF32 pairs), 2e-2 (scaled with the gradients' magnitude) for 16 bits, as in the parity tests."""
    dtype = DT[dt]
    q, k, v, tq, tk, tv, go, gt = _inputs(B, H, L, D, dtype, seed + L + D)
    mask, causal = _mask(kind, B, H, L, dtype, seed + 1), kind == "causal"
    go, gt = (go if cot != "t" else None), (gt if cot != "o" else None)
    ref = orc.grads_through_both(q, k, v, tq, tk, tv, go, gt, attn_mask=mask, causal=causal)
    cu = lambda x: None if x is None else x.to(DEV)  # noqa: E731
    a = [cu(x).requires_grad_() for x in (q, k, v)]
    m = cu(mask)
    o, to = torch.func.jvp(lambda x, y, z: ja.JVPAttn.fwd_dual(x, y, z, attn_mask=m, causal=causal), tuple(a),
                           tuple(cu(x) for x in (tq, tk, tv)))
    outs = [(x, cu(w)) for x, w in ((o, go), (to, gt)) if w is not None]
    got = (o, to, *torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs]))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    for name, x, r in zip(("O", "tO", "dq", "dk", "dv"), got, ref):
        top = r.abs().max().item()
        e = orc.max_abs_err(x, r)
        assert e <= (fp32_bound * top if dt == "fp32" else 2e-2 * max(1.0, top)), (name, e, top)


@pytest.mark.parametrize("dt,B,H,L,kind,cot", [
    ("bf16", 1, 2, 66, "none", "both"), ("bf16", 2, 3, 128, "causal", "t"), ("fp16", 2, 2, 200, "keys", "both"),
    ("bf16", 1, 3, 258, "none", "o"), ("fp16", 2, 1, 320, "window", "both"), ("bf16", 1, 2, 130, "bias", "t"),
    ("bf16", 3, 8, 1000, "none", "both"),
])
def test_head_dimension_32_on_the_tensor_core_kernels(dt, B, H, L, kind, cot):
    _check(B, H, L, 32, dt, kind, cot)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dt,L,kind,cot", [
    ("bf16", 66, "bool", "both"), ("fp16", 130, "bias", "both"), ("bf16", 250, "bias", "o"), ("bf16", 334, "window", "t"),
    ("fp16", 506, "bool", "t"),
])
def test_masks_whose_rows_do_not_fill_16_byte_pieces(D, dt, L, kind, cot):
    _check(2, 2, L, D, dt, kind, cot)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,L,kind,cot", [
    (1, 1, 34, "none", "both"), (1, 3, 100, "causal", "t"), (2, 8, 320, "keys", "both"), (4, 10, 250, "bool", "o"),
    (2, 12, 450, "bias", "both"),
])
def test_row_and_key_splits_of_the_register_tiled_kernels(D, B, H, L, kind, cot):
    """16-row tiles below 296 of them run as 1 x 8 warps, below 592 as 2 x 4, above as 4 x 2 (through O alone: one warp each)."""
    _check(B, H, L, D, "fp32", kind, cot)


@pytest.mark.parametrize("dt,D", [("fp32", 64), ("fp32", 128), ("bf16", 64), ("bf16", 128), ("fp16", 32)])
@pytest.mark.parametrize("want", ["q", "kv"])
def test_gradients_nobody_asked_for_are_left_out(dt, D, want):
    """The gradients that are asked for are those of the full call (bit for bit where the same kernel forms them; dQ of
    the single pass is summed in another order than by the own-queries launch: the 16-bit tolerance)."""
    q, k, v, tq, tk, tv, go, gt = (x.to(DEV) for x in _inputs(2, 3, 200, D, DT[dt], 5))

    def run(names):
        a = {n: x.clone().requires_grad_(n in names) for n, x in (("q", q), ("k", k), ("v", v))}
        o, to = torch.func.jvp(lambda x, y, z: ja.JVPAttn.fwd_dual(x, y, z, causal=True), tuple(a.values()), (tq, tk, tv))
        return torch.autograd.grad((o, to), [a[n] for n in names], (go, gt))

    full = dict(zip("qkv", run("qkv")))
    for n, x in zip(want, run(want)):
        if dt == "fp32" or D == 128 or want == "kv":
            assert torch.equal(x, full[n]), n
        else:
            assert (x.float() - full[n].float()).abs().max().item() <= 2e-2 * max(1.0, full[n].abs().max().item())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("kind,L,D", [("bool", 128, 64), ("bool", 250, 64), ("bool", 192, 128), ("bias", 250, 64), ("bias", 250, 128)])
@pytest.mark.parametrize("how", ["data", "graph"])
def test_a_mask_written_behind_the_version_counter_is_read_as_it_is(kind, L, D, how):
    """Neither a write through ``.data`` nor one between two replays of a graph moves the counter that the mask's
    verification is remembered by; what the kernels read has to be the new entries all the same.  (Dense masks and bias:
    which tiles are stepped over, and key lengths, are those of the verification.)"""
    q, k, v, tq, tk, tv, _, _ = (x.to(DEV) for x in _inputs(2, 3, L, D, torch.bfloat16, 6))
    first, second = (_mask(kind, 2, 3, L, torch.bfloat16, s).to(DEV) for s in (1, 2))
    a = [x.clone().requires_grad_() for x in (q, k, v)]

    def run(m):
        o, to = torch.func.jvp(lambda x, y, z: ja.JVPAttn.fwd_dual(x, y, z, attn_mask=m), tuple(a), (tq, tk, tv))
        return (o, to, *torch.autograd.grad((o, to), a, (q, v)))

    want = [x.detach().clone() for x in run(second.clone())]
    mask = first.clone()
    if how == "data":
        run(mask)
        mask.data.copy_(second)
        got = run(mask)
    else:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            run(mask)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run(mask)
        mask.copy_(second)
        graph.replay()
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    for x, y in zip(got[:2], want[:2]):
        assert torch.equal(x, y)
    for x, y in zip(got[2:], want[2:]):  # dQ may be summed by reductions: the order of two runs differs
        assert (x.float() - y.float()).abs().max().item() <= 2e-2 * max(1.0, y.abs().max().item())


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,L", [(1, 2, 34), (2, 10, 250), (2, 12, 450)])
def test_fp32_rows_of_very_different_magnitude(B, H, L, D):
    """Rows of V and its tangent up to a factor of 2^40 apart, and masked-out keys that hold 1e15, must cost no precision.
    Every product is within 2^-21 of its operands' magnitudes; a gradient passes three in a row and sums a few hundred
    terms: 1e-5 of P |V| for O, of the head's largest V for tO, of the head's largest entry for a gradient."""
    q, k, v, tq, tk, tv, go, gt = _inputs(B, H, L, D, torch.float32, L + D)
    g = torch.Generator().manual_seed(L)
    vscale = torch.exp2(torch.randint(-20, 21, (B, H, L, 1), generator=g).float())
    v, tv = v * vscale, tv * vscale
    dead = torch.rand(B, 1, L, 1, generator=g) > 0.8
    dead[:, :, 0] = False
    mask = (torch.rand(B, 1, L, L, generator=g) > 0.3) & ~dead.transpose(2, 3)
    mask[..., 0] = True
    clean = [x.masked_fill(dead, 0.0) for x in (k, v, tk, tv)]
    ref = orc.grads_through_both(q, clean[0], clean[1], tq, clean[2], clean[3], go, gt, attn_mask=mask)
    k, v, tk, tv = (x.masked_fill(dead, 1e15) for x in (k, v, tk, tv))
    a = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    m = mask.to(DEV)
    o, to = torch.func.jvp(lambda x, y, z: ja.JVPAttn.fwd_dual(x, y, z, attn_mask=m), tuple(a), tuple(x.to(DEV) for x in (tq, tk, tv)))
    got = (o, to, *torch.autograd.grad((o, to), a, (go.to(DEV), gt.to(DEV))))
    head = lambda x: x.double().abs().amax(dim=(2, 3), keepdim=True)  # noqa: E731
    scores = (q.double() @ clean[0].double().transpose(-1, -2) * D**-0.5).masked_fill(~mask, float("-inf"))
    weight = torch.softmax(scores, -1) @ clean[1].double().abs()
    for name, x, r in zip(("O", "tO", "dq", "dk", "dv"), got, ref):
        x = x.detach().cpu().double()
        assert torch.isfinite(x).all(), name
        top = weight if name == "O" else head(clean[1]) if name == "tO" else head(r)
        off = ((x - r.double()).abs() / top.clamp(min=1e-30)).max().item()
        assert off <= 1e-5, (name, off)


def _grads_fp32(a, tangents, go, gt):
    a = [x.to(DEV).requires_grad_() for x in a]
    o, to = torch.func.jvp(ja.JVPAttn.fwd_dual, tuple(a), tuple(x.to(DEV) for x in tangents))
    return (o, to, *torch.autograd.grad((o, to), a, (go.to(DEV), gt.to(DEV))))


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,L", [(1, 2, 34), (2, 10, 250), (2, 12, 450)])
@pytest.mark.parametrize("big", [1e8, 1e15, 1e36, float("inf"), float("nan")])
def test_fp32_a_large_entry_costs_the_others_nothing(D, B, H, L, big):
    """One entry of V (of gO for dV) that is very large, Inf or NaN: the other columns are what they are without it.  Every
    product is within 2^-21 of its own operands and a column sums a few hundred: 1e-5 of P |V| (of P^T |gO|) there."""
    q, k, v, tq, tk, tv, go, gt = _inputs(B, H, L, D, torch.float32, L + D)
    v[:, :, L // 2, 5] = big
    o, to, *_ = _grads_fp32((q, k, v), (tq, tk, tv), go, gt)
    rest = [c for c in range(D) if c != 5]
    p = torch.softmax(q.double() @ k.double().transpose(-1, -2) * D**-0.5, -1)
    ts = (tq.double() @ k.double().transpose(-1, -2) + q.double() @ tk.double().transpose(-1, -2)) * D**-0.5
    w = p * (ts - (p * ts).sum(-1, keepdim=True))
    vd, tvd = v.double()[..., rest], tv.double()[..., rest]
    for x, r, top in ((o, p @ vd, p @ vd.abs()), (to, w @ vd + p @ tvd, (p * ts.abs().amax(-1, keepdim=True)) @ vd.abs() + p @ tvd.abs())):
        assert ((x.detach().cpu().double()[..., rest] - r).abs() / top).max().item() <= 1e-5
        assert big < 1e30 or not torch.isfinite(x[..., 5]).any() or big == 1e36
    v[:, :, L // 2, 5] = 1.0
    go[:, :, L // 3, 5] = big
    dv = _grads_fp32((q, k, v), (tq, tk, tv), go, torch.zeros_like(gt))[4].cpu().double()[..., rest]
    pt, god = p.transpose(-1, -2), go.double()[..., rest]
    assert ((dv - pt @ god).abs() / (pt @ god.abs())).max().item() <= 1e-5


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,L", [(1, 2, 34), (2, 10, 250), (2, 12, 450)])
def test_fp32_channels_of_very_different_magnitude(D, B, H, L):
    """One channel of q and its tangent scaled by 1e6 and of k by 1e-6, another the other way round: the scores are those of
    the unscaled tensors, and so are the results but for the scales.  1e-5 of the largest entry, as in the rest of this file."""
    q, k, v, tq, tk, tv, go, gt = _inputs(B, H, L, D, torch.float32, L + D)
    s = torch.ones(D)
    s[1], s[2] = 1e6, 1e-6
    ref = orc.grads_through_both(q * s, k / s, v, tq * s, tk / s, tv, go, gt)
    got = _grads_fp32((q * s, k / s, v), (tq * s, tk / s, tv), go, gt)
    for name, x, r, scale in zip(("O", "tO", "dq", "dk", "dv"), got, ref, (1.0, 1.0, s, 1 / s, 1.0)):
        x, r = x.detach().cpu().double() * scale, r.double() * scale
        assert ((x - r).abs().max() / r.abs().max()).item() <= 1e-5, name


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("B,H,L,kind", [(1, 2, 34, "none"), (2, 10, 250, "bias"), (2, 12, 450, "causal")])
def test_fp32_second_differentiation_along_q_alone(B, H, L, D, kind):
    """With K and V held fixed their zero tangents are left out (both routes form the same products otherwise): against the
    general route, which a zero direction for K and V takes.  1e-5 of the largest entry, the fp32 bound of this file."""
    q, k, v, u, _, _, go, _ = (x.to(DEV) for x in _inputs(B, H, L, D, torch.float32, L + D))
    mask = _mask(kind, B, H, L, torch.float32, 1)
    mask = None if mask is None else mask.to(DEV)

    def second(leaves):
        a = [x.clone().requires_grad_(n in leaves) for n, x in (("q", q), ("k", k), ("v", v))]
        w = go.clone().requires_grad_()
        o = ja.attention(*a, attn_mask=mask, causal=kind == "causal")
        first = torch.autograd.grad(o, [x for x in a if x.requires_grad], w, create_graph=True)
        z = [u] + [torch.zeros_like(k) for _ in first[1:]]
        return torch.autograd.grad(first, [a[0], w], z)

    for x, y in zip(second("q"), second("qkv")):
        assert (x - y).abs().max().item() <= 1e-5 * y.abs().max().item()


@pytest.mark.parametrize("dt", ["bf16", "fp16"])
@pytest.mark.parametrize("D,L,kind", [(32, 250, "none"), (32, 256, "bias"), (64, 250, "bool"), (64, 250, "bias"), (128, 250, "bool"),
                                      (128, 250, "bias")])
def test_the_largest_probability_of_a_row_is_held_exactly(dt, D, L, kind):
    """Head dimension 32 and masks with ragged rows: the running maximum is the reference, as on the register-tiled kernels,
    so a row's largest probability is 1 and not rounded.  Here it outweighs the rest (2^-5.6 at most) and lies in a later tile
    than a runner-up within the 2^8 that lazy rescaling would leave: all that is left of O's error is its own rounding to 16
    bits, plus 2^-5.6 of a probability's."""
    B, H, dtype = 2, 2, DT[dt]
    g = torch.Generator().manual_seed(D + L)
    q, k = torch.zeros(B, H, L, D), torch.zeros(B, H, L, D)
    q[..., 0], q[..., 1] = 1.0, torch.rand(B, H, L, generator=g)
    unit = D**0.5 * 0.6931471805599453  # one of the softmax's powers of two
    k[..., 0] = -40 * unit
    k[:, :, 3, 0], k[:, :, 200, 0], k[:, :, 200, 1] = unit, 7 * unit, unit
    q, k = q.to(dtype), k.to(dtype)
    v = torch.randn(B, H, L, D, generator=g).to(dtype)
    mask = torch.ones(B, 1, L, L, dtype=torch.bool) if kind == "bool" else torch.zeros(B, H, L, L, dtype=dtype)
    if kind == "bool":
        mask[:, :, ::2, 5] = False
    m = None if kind == "none" else mask.to(DEV)
    o = ja.attention(q.to(DEV), k.to(DEV), v.to(DEV), attn_mask=m).cpu().double()
    ref = torch.softmax(q.double() @ k.double().transpose(-1, -2) * D**-0.5, -1) @ v.double()
    assert (o - ref).norm() <= 1.1 * (ref.to(dtype).double() - ref).norm()


@pytest.mark.parametrize("D,L,kind,cot", [(32, 1000, "none", "both"), (32, 514, "causal", "t"), (32, 512, "bias", "o"),
                                          (64, 506, "bool", "both"), (64, 1000, "bias", "o"), (64, 506, "bias", "o")])
def test_gradients_summed_in_a_fixed_order(D, L, kind, cot):
    """Head dimension 32, and masks whose rows are not whole 16-byte pieces: bit for bit the same from run to run."""
    B, H = 3, 6
    q, k, v, tq, tk, tv, go, gt = (x.to(DEV) for x in _inputs(B, H, L, D, torch.bfloat16, L))
    mask = _mask(kind, B, H, L, torch.bfloat16, 1)
    mask = None if mask is None else mask.to(DEV)
    a = [x.clone().requires_grad_() for x in (q, k, v)]

    def run():
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=mask, causal=kind == "causal"), tuple(a), (tq, tk, tv))
        outs = [(o, go)] * (cot != "t") + [(to, gt)] * (cot != "o")
        return torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs])

    first = run()
    for _ in range(10):
        for x, y in zip(run(), first):
            assert torch.equal(x, y)


@pytest.mark.parametrize("D,L", [(32, 500), (64, 1024), (128, 500), (128, 1410)])
@pytest.mark.parametrize("std", [0.1, 1.0])
def test_fp32_gradients_through_both_outputs_are_as_exact_as_through_one(D, L, std):
    """Each score product has an accumulator of its own.  A tensor core adds with truncation: 3 D / 8 adds, each losing half a
    unit (0.72 x 2^-24 on average) of a partial sum that is two thirds of the result, come to 0.18 D 2^-24.  A gradient passes
    two such products, independent of one another: 0.25 D 2^-24; a third more is allowed.  With two products in one
    accumulator it was 0.35."""
    B, H = 2, 4
    x = [t.float() for t in _inputs(B, H, L, D, torch.float32, L + D)]
    for i in (3, 4, 5):
        x[i] = x[i] * (10 * std)
    ref = orc.grads_through_both(*x, causal=True)
    a = [t.to(DEV).requires_grad_() for t in x[:3]]
    o, to = torch.func.jvp(lambda *t: ja.JVPAttn.fwd_dual(*t, causal=True), tuple(a), tuple(t.to(DEV) for t in x[3:6]))
    got = torch.autograd.grad((o, to), a, (x[6].to(DEV), x[7].to(DEV)))
    for name, y, r in zip(("dq", "dk", "dv"), got, ref[2:]):
        assert ((y.cpu().double() - r).norm() / r.norm()).item() <= D / 3 * 2**-24, name


@pytest.mark.parametrize("kind", ["none", "bias"])
def test_a_trace_is_refused_rather_than_recorded_as_a_constant(kind):
    """Under torch.jit.trace sizes are tensors, which the argument checks refuse.  A call that went past them left the output
    of the traced input in the trace."""
    q, k, v, *_ = (x.to(DEV) for x in _inputs(1, 2, 64, 64, torch.bfloat16, 1))
    mask = None if kind == "none" else _mask(kind, 1, 2, 64, torch.bfloat16, 1).to(DEV)
    ja.attention(q, k, v, attn_mask=mask)
    with pytest.raises(AssertionError, match="HEAD_DIM"):
        torch.jit.trace(lambda x: ja.attention(x, k, v, attn_mask=mask), (q,), check_trace=False)


def _peak(run):
    """Outputs of a call, its peak of allocated bytes, and what it leaves allocated, both over what was there before."""
    out = run()  # the mask's verification, kernels' first use
    del out
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    out = run()
    return out, torch.cuda.max_memory_allocated() - before, torch.cuda.memory_allocated() - before


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dims", [(1, 1), (8, 1), (1, 16)])
def test_a_ragged_bias_that_broadcasts_is_not_written_out(D, dims):
    """Rows of 250 elements are padded to 256 for the tensor-core kernels: what the copy takes is the bias's own extents, a
    view that expands costs no more than the tensor it is a view of (and what the allocator's blocks are larger, up to 1 MiB).
    Written out it would be 16 MB."""
    B, H, L = 8, 16, 250
    q, k, v, *_ = (x.to(DEV) for x in _inputs(B, H, L, D, torch.bfloat16, D))
    own = _mask("bias", *dims, L, torch.bfloat16, 1).to(DEV)
    view = own.expand(B, H, L, L)
    assert 0 in view.stride()
    with torch.no_grad():
        got, peak, _ = _peak(lambda: ja.attention(q, k, v, attn_mask=view))
        _, plain, _ = _peak(lambda: ja.attention(q, k, v))
        want = ja.attention(q, k, v, attn_mask=view.contiguous())
    assert torch.equal(got, want)
    assert peak - plain <= dims[0] * dims[1] * L * 256 * 2 + (1 << 20)


def test_the_copy_of_a_ragged_bias_does_not_wait_for_the_backward():
    B, H, L, D = 4, 8, 506, 64
    q, k, v, _, _, _, go, _ = (x.to(DEV) for x in _inputs(B, H, L, D, torch.bfloat16, 3))
    bias = _mask("bias", B, H, L, torch.bfloat16, 1).to(DEV)
    a = [x.clone().requires_grad_() for x in (q, k, v)]
    o, _, held = _peak(lambda: ja.attention(*a, attn_mask=bias))
    _, _, plain = _peak(lambda: ja.attention(*a))
    assert held <= plain + (1 << 20)  # blocks may be that much larger than what is asked for; the copy takes 16.6 MB
    ref = orc.grads_through_both(*(x.cpu() for x in (q, k, v)), *(torch.zeros(B, H, L, D) for _ in range(3)), go.cpu(), None, attn_mask=bias.cpu())
    for x, r in zip(torch.autograd.grad(o, a, go), ref[2:]):
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item())


@pytest.mark.parametrize("kind", ["bias", "bool"])
def test_a_mask_whose_copy_does_not_fit_is_read_in_place(kind):
    """With room for the results but not for another form of the mask, the call runs as it did without one."""
    B, H, L, D = 2, 24, 2050, 64
    q, k, v, *_ = (x.to(DEV) for x in _inputs(B, H, L, D, torch.bfloat16, 4))
    mask = _mask("bias", B, H, L, torch.bfloat16, 1).to(DEV) if kind == "bias" else (torch.rand(B, H, L, L, device=DEV) > 0.5)
    torch.cuda.empty_cache()  # the results get memory of their own, not a part of what the mask was made in
    with torch.no_grad():
        want = ja.attention(q, k, v, attn_mask=mask)
        torch.cuda.empty_cache()
        room = torch.cuda.memory_reserved() + (20 << 20)  # O and its row statistics take 13 MB, the bits of `bool` 26 MB
        try:
            torch.cuda.set_per_process_memory_fraction(room / torch.cuda.get_device_properties(0).total_memory)
            got = ja.attention(q, k, v, attn_mask=mask)
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
    assert (got.float() - want.float()).abs().max().item() <= 2e-2 * max(1.0, want.abs().max().item())
    assert _lib.device_status() == 0


@pytest.mark.parametrize("kind", ["none", "bool"])
def test_other_threads_run_while_the_launch_queue_is_full(kind):
    """Launches behind half a second of device time: more than the queue holds, so the launching thread waits.  Another
    thread's largest pause stays far below that wait."""
    q, *_ = (x.to(DEV) for x in _inputs(1, 2, 66, 64, torch.bfloat16, 5))
    mask = None if kind == "none" else _mask(kind, 1, 2, 66, torch.bfloat16, 1).to(DEV)
    pauses, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            pauses.append(now - last)
            last = now

    with torch.no_grad():
        ja.attention(q, q, q, attn_mask=mask)
        torch.cuda.synchronize()
        other = threading.Thread(target=tick)
        other.start()
        torch.cuda._sleep(1_000_000_000)  # clock cycles
        begin = time.perf_counter()
        for _ in range(4000):
            ja.attention(q, q, q, attn_mask=mask)
        waited = time.perf_counter() - begin
        torch.cuda.synchronize()
        stop.set()
        other.join()
    assert waited > 0.2 and max(pauses) < waited / 4, (waited, max(pauses))


@pytest.mark.parametrize("dt", ["bfloat16", "float32"])
def test_first_calls_of_several_threads(dt):
    """In a process of its own: threads that have made no CUDA call before, and whose buffers come from torch's cache, call the library
    at once.  (The tensor maps are encoded by the driver, which refuses a thread that has no current context.)"""
    code = f"""
import threading, torch
import jvp_flash_attention_b200.jvp_attention as ja
from jvp_flash_attention_b200 import _lib
x = torch.randn(2, 16, 256, 64, device="cuda", dtype=torch.{dt})
cached = [torch.empty_like(x) for _ in range(64)] + [torch.empty(1 << 24, dtype=torch.uint8, device="cuda") for _ in range(16)]
del cached
_lib.load(), _lib.native(), torch.cuda.synchronize()
start, out = threading.Barrier(8), [None] * 8
def call(n):
    start.wait()
    try:
        out[n] = ja.attention(x, x, x)
    except Exception as e:
        out[n] = e
threads = [threading.Thread(target=call, args=(n,)) for n in range(8)]
[t.start() for t in threads], [t.join() for t in threads]
assert all(isinstance(o, torch.Tensor) for o in out), out
torch.cuda.synchronize()
assert all(torch.equal(o, out[0]) for o in out) and _lib.device_status() == 0
"""
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, cwd=pathlib.Path(__file__).parent.parent)


@pytest.mark.parametrize("L", [34, 130, 1000, 4200])
@pytest.mark.parametrize("layout", ["rows", "keys", "one row", "expanded"])
def test_tile_bitmaps_are_those_of_the_host_stand_in(L, layout):
    """jvpfa_mask_tiles against the eager reductions that stand in for it in the CPU tests, ragged and in other strides."""
    g = torch.Generator().manual_seed(L)
    m = torch.rand(2, 1 if L > 1000 else 3, 1 if layout == "one row" else L, L, generator=g) > 1 - 2 / (128 * 64)
    m[:, :, 0, L // 3] = True
    if layout == "keys":
        m = m.transpose(2, 3)
    if layout == "expanded":
        m = m[:1].expand(2, -1, -1, -1)

    def spec(t):
        return _lib.MaskSpec(_lib.MASK_BOOL, t.view(torch.uint8), tuple(0 if n == 1 else s for n, s in zip(t.shape, t.stride())))

    dev = torch.empty_strided(m.shape, m.stride(), dtype=torch.bool, device=DEV).copy_(m) if layout != "expanded" else m[:1].to(DEV).expand(2, -1, -1, -1)
    for x, y in zip(_lib.mask_tiles(spec(dev), L), stand_in.mask_tiles(spec(m), L)):
        assert torch.equal(x.cpu(), y.to(x.dtype))


@pytest.mark.parametrize("L", [33, 66, 130, 257, 520])
@pytest.mark.parametrize("layout", ["rows", "offset", "padded", "keys", "one row", "expanded"])
def test_packed_bits_are_the_mask(L, layout):
    """Bits by rows and transposed, of rows that begin at any address: whole pieces, words that straddle them, and the mask's ends."""
    g = torch.Generator().manual_seed(L)
    heads, n_rows = (2, 3), 1 if layout == "one row" else L
    m = torch.rand(*heads, n_rows, L, generator=g) > 0.5
    dev = m.to(DEV)
    if layout == "offset":  # the first entry one byte behind a 16-byte boundary, the last one at the end of its storage
        dev = torch.cat([torch.ones(1, dtype=torch.bool, device=DEV), dev.flatten()])[1:].view(m.shape)
    elif layout == "padded":
        dev = torch.nn.functional.pad(dev, (3, 4), value=True)[..., 3:-4]
    elif layout == "keys":
        dev = dev.transpose(2, 3).contiguous().transpose(2, 3)
    elif layout == "expanded":
        m, dev = m[:, :1], dev[:, :1].contiguous().expand(2, 3, L, L)
    n_h, w, wt = m.shape[1], (L + 63) // 64 * 2, (n_rows + 63) // 64 * 2 if n_rows > 1 else 1
    a = _lib.MaskTilesArgs(struct_size=ctypes.sizeof(_lib.MaskTilesArgs), n_b=2, n_h=n_h, n_rows=n_rows, L=L)
    a.mask = _lib.MaskSpec(_lib.MASK_BOOL, dev.view(torch.uint8), tuple(0 if n == 1 else s for n, s in zip(m.shape, dev.stride()))).to_c()
    a.mask.stride[3] = dev.stride(3)
    bits = torch.zeros(2 * n_h, n_rows, w, dtype=torch.int32, device=DEV)
    bits_t = torch.zeros(2 * n_h, L, wt, dtype=torch.int32, device=DEV)
    a.bits, a.bits_t = bits.data_ptr(), bits_t.data_ptr()
    _lib.check(_lib.load().jvpfa_mask_tiles(ctypes.byref(a), torch.cuda.current_stream().cuda_stream), "jvpfa_mask_tiles")
    one = torch.arange(32, dtype=torch.int32)

    def unpack(x, n):
        return (x.cpu()[..., None] >> one & 1).flatten(-2).bool()[..., :n]

    m = m.reshape(-1, n_rows, L)
    assert torch.equal(unpack(bits, L), m)
    assert torch.equal(unpack(bits_t, n_rows), m.transpose(1, 2))


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("how,kind,cot", [("fp32", "none", "o"), ("fp32", "bias", "o"), ("tf32", "causal", "both"), ("tf32", "bool", "o"),
                                          ("bf16", "keys", "both"), ("fp16", "bias", "t"), ("bf16", "causal", "o")])
def test_register_tiled_kernels_with_one_warp_for_16_rows(monkeypatch, D, how, kind, cot):
    """From 592 (backward) or 1184 (forward) 16-row tiles on; here 1200 of them, of a length that no tile divides.  Single TF32
    products: 5e-3 of the largest entry, as in the parity tests."""
    if how == "tf32":
        monkeypatch.setattr(_lib, "FP32_PRECISION", "tf32")
    elif how != "fp32":
        monkeypatch.setattr(ja, "KERNEL_IMPL", _lib.IMPL_GENERIC)
    _check(4, 10, 474, D, "fp32" if how == "tf32" else how, kind, cot, fp32_bound=5e-3 if how == "tf32" else 1e-5)


@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("want", ["q", "kv"])
@pytest.mark.parametrize("impl", [_lib.IMPL_GENERIC, _lib.IMPL_AUTO], ids=["one warp", "tcgen05"])
def test_one_warp_for_16_rows_leaves_out_what_nobody_asked_for(monkeypatch, D, want, impl):
    """Of the register-tiled kernels with one warp for 16 rows, and of the fp32 tcgen05 kernels, which serve such a call otherwise."""
    monkeypatch.setattr(ja, "KERNEL_IMPL", impl)
    q, k, v, _, _, _, go, _ = (x.to(DEV) for x in _inputs(4, 10, 474, D, torch.float32, 5))

    def run(names):
        a = {n: x.clone().requires_grad_(n in names) for n, x in (("q", q), ("k", k), ("v", v))}
        return torch.autograd.grad(ja.attention(*a.values(), causal=True), [a[n] for n in names], go)

    full = dict(zip("qkv", run("qkv")))
    for n, x in zip(want, run(want)):
        assert torch.equal(x, full[n]), n
