"""fp32 on the tcgen05 kernels (three bf16 parts of every entry): at the edges of their tiles, in every form of mask and layout
that the register-tiled kernels take, against the float64 oracle and against those kernels; and where the dispatch begins."""
import ctypes
import math

import pytest
import torch

from jvp_flash_attention_b200 import _lib
from oracle import jvp_attention_oracle as orc

DEV = "cuda:0"


def _fwd_args(ts, tangents, mask, out, impl, strides=None):
    """jvpfa_fwd_args on tensors (or, for the host logic alone, on addresses that nothing follows)."""
    at = lambda x: None if x is None else x if isinstance(x, int) else x.data_ptr()  # noqa: E731
    B, H, L, D = ts[0].shape
    a = _lib.FwdArgs(struct_size=ctypes.sizeof(_lib.FwdArgs), dtype=_lib.FP32, B=B, H=H, L=L, D=D, impl=impl, sm_scale=D**-0.5)
    a.q, a.k, a.v = (at(x) for x in ts)
    a.tq, a.tk, a.tv = (at(x) for x in (*tangents, None, None, None)[:3])
    a.o, a.to, a.lse, a.mu = (at(x) for x in out)
    a.flags = 8 if len(tangents) == 1 else 0  # JVPFA_ZERO_TKV
    a.mask = mask
    if strides:
        a.in_stride[0], a.in_stride[1], a.in_stride[2] = strides
    return a


def _mask(kind, B, H, L, g):
    """(kernel-side description, what keeps it alive, the oracle's mask, causal)"""
    m = _lib.Mask(kind=_lib.MASK_NONE)
    if kind == "none":
        return m, None, None, False
    if kind == "causal":
        m.kind = _lib.MASK_CAUSAL
        return m, None, None, True
    if kind == "keys":
        lens = torch.randint(0, L + 1, (B,), generator=g)
        lens[0] = L  # (and one sequence may be empty)
        t = lens.to(DEV, torch.int32)
        m.kind, m.kv_len = _lib.MASK_KVLEN, t.data_ptr()
        return m, t, (torch.arange(L)[None] < lens[:, None])[:, None, None], False
    if kind.startswith("bool"):
        x = torch.rand(B, 1 if kind == "bool_shared" else H, L, L, generator=g) > 0.5
        x[:, :, L // 2] = False  # a row without a key
        t = x.to(DEV)
        if kind == "bool_transposed":  # keys are not the contiguous dimension
            t = t.transpose(2, 3).contiguous().transpose(2, 3)
        m.kind = _lib.MASK_BOOL
    else:
        dt = {"bias": torch.float32, "bias_bf16": torch.bfloat16, "bias_odd": torch.float32, "bias_row": torch.float16}[kind]
        x = torch.randn(B, H, 1 if kind == "bias_row" else L, L, generator=g).to(dt)
        t = x.to(DEV)
        if kind == "bias_odd":  # rows that begin 4 bytes off a 16-byte boundary
            t = torch.nn.functional.pad(t, (1, 0))[..., 1:]
        m.kind, m.bias_dtype = _lib.MASK_BIAS, _lib.DTYPE_ENUM[dt]
    m.ptr = t.data_ptr()
    for d in range(4):
        m.stride[d] = t.stride(d) if t.size(d) > 1 else 0
    if t.size(3) == 1:
        m.stride[3] = 1
    return m, t, x, False


def _run_fwd(ts, tangents, mask, impl, strides=None):
    B, H, L, D = ts[0].shape
    nan = lambda *s: torch.full(s, math.nan, device=DEV)  # noqa: E731
    out = [nan(B, H, L, D), nan(B, H, L, D) if tangents else None, nan(B, H, L), nan(B, H, L) if tangents else None]
    a = _fwd_args(ts, tangents, mask, out, impl, strides)
    lib = _lib.load()
    if impl == _lib.IMPL_TCGEN05:
        ws = torch.full((lib.jvpfa_fwd_workspace(ctypes.byref(a)),), 0x7F, dtype=torch.uint8, device=DEV)
        assert ws.numel() > 0
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    _lib.check(lib.jvpfa_fwd(ctypes.byref(a), torch.cuda.current_stream().cuda_stream), "jvpfa_fwd")
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    return out


def _rel(x, r):
    return ((x.cpu().double() - r).norm() / r.norm().clamp(min=1e-30)).item()


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("L,kind,n_tangents", [
    (1, "none", 3), (34, "causal", 3), (63, "bias", 0), (65, "bool", 1), (128, "none", 0), (129, "causal", 1), (130, "bias_odd", 3),
    (192, "bool_transposed", 3), (200, "keys", 3), (257, "bias_bf16", 1), (300, "bool_shared", 0), (384, "keys", 1), (500, "bias", 3),
    (333, "bias_row", 3),
])
def test_forward_on_three_bf16_parts(D, L, kind, n_tangents):
    """A product is exact to 2^-24 of its operands and an accumulator takes up to 48 instructions a key tile, each truncated at 2^-24
    of what is there by then: 1e-5 of the largest entry, the fp32 bound of the parity tests, and no further from 64 bits than
    the register-tiled kernels (1.2 times, for the luck of a few rows)."""
    B, H = 2, 3
    g = torch.Generator().manual_seed(L + D)
    ts = [torch.randn(B, H, L, D, generator=g) for _ in range(3)]
    tg = [torch.randn(B, H, L, D, generator=g) for _ in range(n_tangents)]
    mask, alive, attn_mask, causal = _mask(kind, B, H, L, g)
    zero = torch.zeros(B, H, L, D)
    if attn_mask is not None and attn_mask.dtype == torch.bool:
        attn_mask = attn_mask.expand(B, H, L, L)
    elif attn_mask is not None:
        attn_mask = attn_mask.double()
    ref = orc.sdpa_jvp(*ts, *(*tg, zero, zero, zero)[:3], attn_mask, causal)
    # the (B, H, L, D) view of (B, L, H, D) tensors, read in place
    dev = [x.transpose(1, 2).contiguous().to(DEV).transpose(1, 2) for x in (*ts, *tg)]
    runs = {}
    for impl in (_lib.IMPL_GENERIC, _lib.IMPL_TCGEN05):
        runs[impl] = _run_fwd(dev[:3], dev[3:], mask, impl, (L * H * D, D, H * D))
    old, new = runs[_lib.IMPL_GENERIC], runs[_lib.IMPL_TCGEN05]
    for n, r in enumerate(ref if n_tangents else ref[:1]):
        assert orc.max_abs_err(new[n], r) <= 1e-5 * max(r.abs().max().item(), 1e-30), n
        assert _rel(new[n], r) <= max(1.2 * _rel(old[n], r), 2**-22), n
    for n in (2, 3):  # lse (+inf where no key attends) and mu
        if new[n] is not None:
            same = torch.isfinite(old[n])
            assert torch.equal(same, torch.isfinite(new[n])) and torch.equal(old[n][~same], new[n][~same])
            if same.any():
                assert (new[n] - old[n])[same].abs().max().item() <= 1e-5 * max(1.0, old[n][same].abs().max().item())
    dense = _run_fwd([x.contiguous() for x in dev[:3]], [x.contiguous() for x in dev[3:]], mask, _lib.IMPL_TCGEN05)
    for x, y in zip(dense, new):
        assert x is None or torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("through", ["o", "t"])
@pytest.mark.parametrize("L,kind", [
    (1, "none"), (34, "causal"), (63, "bias"), (65, "bool"), (128, "none"), (129, "causal"), (130, "bias_odd"),
    (192, "bool_transposed"), (200, "keys"), (257, "bias_bf16"), (300, "bool_shared"), (500, "bias"), (333, "bias_row"),
])
def test_backward_on_three_bf16_parts(D, through, L, kind):
    """Through O, and dQ through tO with no tangents of K and V, from the lse and mu of the forward on the same kernels: 1e-5 of
    the largest entry, and no further from 64 bits than the register-tiled pair (1.2 times).  dQ alone is dQ of the full call."""
    B, H = 2, 3
    g = torch.Generator().manual_seed(L + D)
    q, k, v, tq, cot = (torch.randn(B, H, L, D, generator=g) for _ in range(5))
    mask, alive, attn_mask, causal = _mask(kind, B, H, L, g)
    zero = torch.zeros(B, H, L, D)
    if attn_mask is not None:
        attn_mask = attn_mask.expand(B, H, L, L) if attn_mask.dtype == torch.bool else attn_mask.double()
    ref = orc.grads_through_both(q, k, v, tq, zero, zero, cot if through == "o" else None, cot if through == "t" else None, attn_mask, causal)[2:]
    strides = (L * H * D, D, H * D)
    dq_, dk_, dv_, dtq_ = (x.transpose(1, 2).contiguous().to(DEV).transpose(1, 2) for x in (q, k, v, tq))
    cot = cot.to(DEV)
    lib, got = _lib.load(), {}
    full = 0 if through == "o" else 2  # JVPFA_SKIP_DKDV
    for impl, skip in ((_lib.IMPL_GENERIC, full), (_lib.IMPL_TCGEN05, 2), (_lib.IMPL_TCGEN05, full)):
        o, to, lse, mu = _run_fwd([dq_, dk_, dv_], [dtq_] if through == "t" else [], mask, impl, strides)
        stats = torch.empty(3, B, H, L, device=DEV)
        _lib.bwd_preprocess(o, to, *((cot, None) if through == "o" else (None, cot)), mu, *stats)
        grads = [torch.full((B, H, L, D), math.nan, device=DEV) for _ in range(3)]
        a = _lib.BwdArgs(struct_size=ctypes.sizeof(_lib.BwdArgs), dtype=_lib.FP32, B=B, H=H, L=L, D=D, impl=impl, sm_scale=D**-0.5)
        a.q, a.k, a.v = dq_.data_ptr(), dk_.data_ptr(), dv_.data_ptr()
        a.lse, a.delta, a.eps, a.cterm = lse.data_ptr(), *(x.data_ptr() for x in stats)
        a.dq, a.flags, a.mask = grads[0].data_ptr(), skip, mask
        if not skip:
            a.dk, a.dv = (x.data_ptr() for x in grads[1:])
        if through == "t":
            a.tq, a.gto, a.mu, a.flags = dtq_.data_ptr(), cot.data_ptr(), mu.data_ptr(), 2 | 8
        else:
            a.go = cot.data_ptr()
        a.in_stride[0], a.in_stride[1], a.in_stride[2] = strides
        if impl == _lib.IMPL_TCGEN05:
            ws = torch.full((lib.jvpfa_bwd_workspace(ctypes.byref(a)),), 0x7F, dtype=torch.uint8, device=DEV)
            a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        _lib.check(lib.jvpfa_bwd(ctypes.byref(a), torch.cuda.current_stream().cuda_stream), "jvpfa_bwd")
        torch.cuda.synchronize()
        assert _lib.device_status() == 0
        got.setdefault(impl, []).append(grads)
    (old,), (alone, new) = got[_lib.IMPL_GENERIC], got[_lib.IMPL_TCGEN05]
    assert torch.equal(alone[0], new[0])
    for n, r in enumerate(ref if through == "o" else ref[:1]):
        if L == 1 and n < 2:  # (one key: no gradient of q and k)
            assert new[n].abs().max().item() <= 1e-5
            continue
        assert orc.max_abs_err(new[n], r) <= 1e-5 * r.abs().max().item(), n
        assert _rel(new[n], r) <= max(1.2 * _rel(old[n], r), 2**-22), n


@pytest.mark.gpu
@pytest.mark.parametrize("D,L,kind", [(64, 514, "bool"), (128, 500, "bias"), (128, 334, "bool"), (32, 1410, "causal"), (64, 1024, "none")])
def test_what_is_asked_of_a_call_decides_the_kernels(D, L, kind):
    """A Hessian-vector product along q runs on the tcgen05 kernels; one that k and v take part in differentiates through tO with
    tangents of all three, which the register-tiled kernels do.  All against the float64 oracle."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    B, H = 2, 6
    g = torch.Generator().manual_seed(L)
    q, k, v, w, u = (torch.randn(B, H, L, D, generator=g) for _ in range(5))
    mask = None
    if kind == "bool":
        mask = (torch.rand(B, 1, L, L, generator=g) > 0.7) | torch.eye(L, dtype=torch.bool)
    elif kind == "bias":
        mask = torch.randn(B, H, L, L, generator=g)
    causal = kind == "causal"
    m = None if mask is None else mask.to(DEV)
    ref = orc.hvp_q(q, k, v, w, u, mask, causal)
    errors = {}
    for leaves in ("q", "qkv"):
        a = [x.to(DEV).requires_grad_(n in leaves) for n, x in zip("qkv", (q, k, v))]
        o = ja.attention(*a, attn_mask=m, causal=causal)
        (dq,) = torch.autograd.grad(o, a[0], w.to(DEV), create_graph=True)
        hq = torch.autograd.grad(dq, [x for x in a if x.requires_grad], u.to(DEV))[0]
        for name, x, r in zip(("O", "dq", "hq"), (o, dq, hq), ref):
            assert orc.max_abs_err(x, r) <= 1e-5 * r.abs().max().item(), (leaves, name)
            errors[leaves, name] = _rel(x.detach(), r)
    for name in ("O", "dq", "hq"):
        assert errors["q", name] <= max(1.2 * errors["qkv", name], 2**-22), (name, errors)
    assert _lib.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("rest", [math.nan, math.inf])
def test_what_padded_keys_hold_does_not_matter(D, rest):
    """Lengths that end inside a 64-key tile; K, V and their tangents hold NaN or Inf from there on: all results are what they are
    with zeros there."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    B, H, L = 4, 16, 512
    lens = torch.tensor([512, 96, 161, 352])
    live = torch.arange(L)[None] < lens[:, None]
    m = live[:, None, None].to(DEV)
    g = torch.Generator().manual_seed(D)
    q, k, v, tq, tk, tv, go = (torch.randn(B, H, L, D, generator=g).to(DEV) for _ in range(7))
    u = torch.randn(B, H, L, D, generator=g).to(DEV)
    keys = live[:, None, :, None].to(DEV)

    def run(fill):
        kk, vv, tkk, tvv = (x.masked_fill(~keys, fill) for x in (k, v, tk, tv))
        a = [x.clone().requires_grad_() for x in (q, kk, vv)]
        o = ja.attention(*a, attn_mask=m)
        o_grads = torch.autograd.grad(o, a, go, create_graph=False)
        dual = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), (q, kk, vv), (tq, tkk, tvv))
        along_q = q.clone().requires_grad_()
        (dq,) = torch.autograd.grad(ja.attention(along_q, kk, vv, attn_mask=m), along_q, go, create_graph=True)
        return o, *o_grads, *dual, dq, torch.autograd.grad(dq, along_q, u)[0]

    for n, (x, y) in enumerate(zip(run(rest), run(0.0))):
        assert torch.isfinite(x).all() and torch.equal(x, y), n


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
def test_forward_up_to_the_end_of_the_range(D):
    """All of V, and of its tangent, 3e36, and a key of the second tile 2^7.8 times as probable as the others: sums of a tile's P V
    stay below 64 * 3e36 < FLT_MAX with probabilities of at most 1.  O and tO are 3e36, to 2^-20 for 512 terms."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    q, k = torch.zeros(2, 32, 512, D, device=DEV), torch.zeros(2, 32, 512, D, device=DEV)
    v = torch.full((2, 32, 512, D), 3e36, device=DEV)
    q[..., 0], k[:, :, 100, 0] = 1.0, 5.4 * D**0.5
    o, to = torch.func.jvp(ja.JVPAttn.fwd_dual, (q, k, v), (torch.zeros_like(q), torch.zeros_like(k), v))
    for x in (o, to, ja.attention(q, k, v)):
        assert ((x.double() - 3e36).abs().max() / 3e36).item() <= 2**-20


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("L,width,std", [(513, 0, 3.0), (512, 0, 1.0), (320, 1, 3.0), (450, None, 3.0)])
def test_the_launch_that_owns_keys_forms_the_scores_of_the_forward(monkeypatch, D, L, width, std):
    """A row with one live key has a probability of 1 and dV is gO, to 2^-23, if S has the bits that lse was made of.  With more keys,
    or all: dV no further from 64 bits than the register-tiled kernels' (1.2 times, for the luck of a few rows)."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    monkeypatch.setattr(ja, "STRICT_SEQUENCE_LENGTH", False)
    B, H = 2, 32 if D == 32 else 16
    g = torch.Generator().manual_seed(L + D)
    q, k, v, go = (torch.randn(B, H, L, D, generator=g).to(DEV) for _ in range(4))
    q, k = q * std, k * std
    i = torch.arange(L, device=DEV)
    mask = None if width is None else ((i[:, None] - i[None]).abs() <= width)[None, None].expand(B, 1, L, L).contiguous()
    s = (q.double() @ k.double().transpose(-1, -2)) * D**-0.5
    p = torch.softmax(s if mask is None else s.masked_fill(~mask, -math.inf), -1)
    ref = p.transpose(-1, -2) @ go.double()
    errors = {}
    for impl in (_lib.IMPL_GENERIC, _lib.IMPL_AUTO):
        monkeypatch.setattr(ja, "KERNEL_IMPL", impl)
        a = [x.clone().requires_grad_() for x in (q, k, v)]
        (dv,) = torch.autograd.grad(ja.attention(*a, attn_mask=mask), a[2], go)
        errors[impl] = ((dv.double() - ref).norm() / ref.norm()).item()
        if width == 0 and impl == _lib.IMPL_AUTO:
            assert (dv - go).abs().max().item() <= 2**-23 * go.abs().max().item()
    assert errors[_lib.IMPL_AUTO] <= max(1.2 * errors[_lib.IMPL_GENERIC], 2**-23), errors


@pytest.mark.gpu
def test_a_replayed_call_is_computed_behind_a_16_bit_launch_that_gave_up():
    """The failure is made on the host, which sets the status word as a thread of a 16-bit kernel would."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    g = torch.Generator().manual_seed(2)
    q, k, v, go = (torch.randn(2, 16, 512, 64, generator=g).to(DEV) for _ in range(4))
    a = [x.requires_grad_() for x in (q, k, v)]

    def step():
        o = ja.attention(*a)
        return [x.detach() for x in (o, *torch.autograd.grad(o, a, go))]

    side = torch.cuda.Stream()  # (the legacy stream's graph nodes cannot be captured)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ref = step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    for code in (5, 0):
        if code:
            _lib.device_status_inject(code)
        try:
            for x in got:
                x.zero_()
            graph.replay()
            torch.cuda.synchronize()
            for x, y in zip(got, ref):
                assert torch.equal(x, y)
        finally:
            assert _lib.device_status(clear=True) == code


@pytest.mark.gpu
def test_a_forward_without_memory_for_its_workspace_decides_for_the_backward(monkeypatch):
    """Both run on the register-tiled kernels then, whose lse and scores belong together, also where the backward finds memory."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    g = torch.Generator().manual_seed(4)
    q, k, v, go = (torch.randn(2, 16, 2048, 64, generator=g).to(DEV) for _ in range(4))
    a = [x.requires_grad_() for x in (q, k, v)]

    def grads(o):
        return [x.detach() for x in (o, *torch.autograd.grad(o, a, go))]

    monkeypatch.setattr(ja, "KERNEL_IMPL", _lib.IMPL_GENERIC)
    want = grads(ja.attention(*a))
    monkeypatch.setattr(ja, "KERNEL_IMPL", _lib.IMPL_AUTO)
    assert not torch.equal(want[0], ja.attention(*a).detach())
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (48 << 20)) / total)  # O needs 17 MB, the workspace 75
    try:
        o = ja.attention(*a)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for x, y in zip(grads(o), want):
        assert torch.equal(x, y)


def _all_results(q, k, v, tq, tk, tv, go, mask=None, **kw):
    """O and its gradients, and O and tO of a call without gradients: the calls that the tcgen05 kernels serve as a whole."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    dev = [x.to(DEV) for x in (q, k, v, tq, tk, tv)]
    m = None if mask is None else mask.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, **kw), tuple(dev[:3]), tuple(dev[3:]))
    a = [x.requires_grad_() for x in dev[:3]]
    o2 = ja.attention(*a, attn_mask=m, **kw)
    assert torch.allclose(o, o2, 0.0, 0.0, equal_nan=True)
    return [x.detach().cpu().double() for x in (o, to, *torch.autograd.grad(o2, a, go.to(DEV)))]


def _range_inputs(D):
    """Rows enough for the tcgen05 kernels at every head dimension, with or without a mask."""
    B, H, L = 2, 24 if D == 32 else 14, 450
    assert _workspace(B, H, L, D)[0] > 0
    g = torch.Generator().manual_seed(D)
    return (B, H, L), g, [torch.randn(B, H, L, D, generator=g) * (0.1 if n in (3, 4, 5) else 1.0) for n in range(7)]


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("big", [1e8, 1e15, 1e36, 3.4e38, math.inf, math.nan])
def test_a_large_entry_costs_the_others_nothing(D, big):
    """One entry of V (of gO for dV) that is very large (3.4e38: above bf16's largest number), Inf or NaN: the other columns are what
    they are without it, to 2^-20 of P |V| (P^T |gO|): products are exact to 2^-24 and a column sums a few hundred.  That column is
    P V, or not finite where V is not."""
    (B, H, L), g, (q, k, v, tq, tk, tv, go) = _range_inputs(D)
    rest = [c for c in range(D) if c != 5]
    p = torch.softmax(q.double() @ k.double().transpose(-1, -2) * D**-0.5, -1)
    ts = (tq.double() @ k.double().transpose(-1, -2) + q.double() @ tk.double().transpose(-1, -2)) * D**-0.5
    w = p * (ts - (p * ts).sum(-1, keepdim=True))
    v[:, :, L // 2, 5] = big
    o, to, *_ = _all_results(q, k, v, tq, tk, tv, go)
    vd, tvd = v.double()[..., rest], tv.double()[..., rest]
    for x, r, top in ((o, p @ vd, p @ vd.abs()), (to, w @ vd + p @ tvd, (p * ts.abs().amax(-1, keepdim=True)) @ vd.abs() + p @ tvd.abs())):
        assert ((x[..., rest] - r).abs() / top).max().item() <= 2**-20
    if math.isfinite(big):
        assert (o[..., 5] - (p @ v.double()[..., 5:6])[..., 0]).abs().max().item() <= 2**-20 * big
    else:
        assert not torch.isfinite(o[..., 5]).any()
    v[:, :, L // 2, 5] = 1.0
    go[:, :, L // 3, 5] = big
    dv = _all_results(q, k, v, tq, tk, tv, go)[4][..., rest]
    pt, god = p.transpose(-1, -2), go.double()[..., rest]
    assert ((dv - pt @ god).abs() / (pt @ god.abs())).max().item() <= 2**-20


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("bad", [math.nan, -math.inf])
@pytest.mark.parametrize("what,first", [("tail", 352), ("tail", 65), ("v", 130), ("tv", 447), ("k", 300), ("strided", 201)])
def test_rows_before_a_key_that_is_not_finite(D, bad, what, first):
    """Causal: rows that end before the key are what they are without it, also in its own tile, and the rows that attend it are not
    finite where its value belongs: in its column, or in all of them."""
    from jvp_flash_attention_b200 import jvp_attention as ja

    (B, H, L), g, ts = _range_inputs(D)
    q, k, v, tq, tk, tv, go = (x.to(DEV) for x in ts)
    if what == "strided":
        q, k, v, tq, tk, tv = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (q, k, v, tq, tk, tv))

    def run(*leaves):
        q_, k_, v_, tq_, tk_, tv_ = leaves
        dual = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, causal=True), (q_, k_, v_), (tq_, tk_, tv_))
        along_q = q_.clone().requires_grad_()
        o = ja.attention(along_q, k_, v_, causal=True)
        (dq,) = torch.autograd.grad(o, along_q, go, create_graph=True)
        return *dual, o.detach(), dq.detach(), torch.autograd.grad(dq, along_q, tq_)[0]

    clean = run(q, k, v, tq, tk, tv)
    if what in ("tail", "strided"):
        for x in (k, v, tk, tv):
            x[:, :, first:] = bad
    else:
        dict(v=v, tv=tv, k=k)[what][:, :, first, 5] = bad
    got = run(q, k, v, tq, tk, tv)
    for n, (x, y) in enumerate(zip(got, clean)):
        assert torch.equal(x[:, :, :first], y[:, :, :first]), n
        if what == "tv" and n != 1:  # only tO has anything to do with it
            assert torch.equal(x, y), n
        elif what in ("v", "tv") and n < 3:
            assert not torch.isfinite(x[:, :, first:, 5]).any(), n
            assert torch.equal(x[..., :5], y[..., :5]) and torch.equal(x[..., 6:], y[..., 6:]), n
        else:
            assert not torch.isfinite(x[:, :, first:]).any(), n


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("bad", [math.nan, math.inf])
@pytest.mark.parametrize("where", ["q", "k", "v", "tq", "tk", "tv", "go"])
def test_what_is_not_finite_reaches_what_it_reached(monkeypatch, D, bad, where):
    """One entry that is not a number, or Inf: the results that are finite are those of the register-tiled kernels, with and without
    rows that have no key.  (Of the gradients under a mask some more: a masked pair has none here, where those kernels have 0 * NaN.)"""
    from jvp_flash_attention_b200 import jvp_attention as ja

    (B, H, L), g, ts = _range_inputs(D)
    q, k, v, tq, tk, tv, go = (x.to(DEV) for x in ts)
    dict(q=q, k=k, v=v, tq=tq, tk=tk, tv=tv, go=go)[where][:, ::2, L // 3, 7] = bad
    mask = torch.rand(B, 1, L, L, generator=g).to(DEV) > 0.3
    mask[:, :, 5] = False
    for m in (None, mask):
        finite = {}
        for impl in (_lib.IMPL_GENERIC, _lib.IMPL_AUTO):
            monkeypatch.setattr(ja, "KERNEL_IMPL", impl)
            dual = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), (q, k, v), (tq, tk, tv))
            a = [x.clone().requires_grad_() for x in (q, k, v)]
            o = ja.attention(*a, attn_mask=m)
            finite[impl] = [torch.isfinite(x.detach()) for x in (*dual, o, *torch.autograd.grad(o, a, go))]
        for n, (x, y) in enumerate(zip(finite[_lib.IMPL_GENERIC], finite[_lib.IMPL_AUTO])):
            assert torch.equal(x, y if m is None or n < 3 else x & y), (n, m is not None, x.float().mean().item(), y.float().mean().item())


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
def test_rows_and_channels_of_very_different_magnitude(D):
    """Rows of V and its tangent up to a factor of 2^40 apart, masked-out keys that hold 1e15, and a channel of q a million times
    larger where k is that much smaller: 1e-5 of P |V| for O, of the head's largest V for tO, of a gradient's largest entry."""
    (B, H, L), g, (q, k, v, tq, tk, tv, go) = _range_inputs(D)
    zoom = torch.exp2(torch.randint(-20, 21, (B, H, L, 1), generator=g).float())
    v, tv = v * zoom, tv * zoom
    s = torch.ones(D)
    s[1], s[2] = 2.0**20, 2.0**-20
    q, tq, k, tk = q * s, tq * s, k / s, tk / s
    dead = torch.rand(B, 1, L, 1, generator=g) > 0.8
    dead[:, :, 0] = False
    mask = (torch.rand(B, 1, L, L, generator=g) > 0.3) & ~dead.transpose(2, 3)
    mask[..., 0] = True
    clean = [x.masked_fill(dead, 0.0) for x in (k, v, tk, tv)]
    ro, rto = orc.sdpa_jvp(q, clean[0], clean[1], tq, clean[2], clean[3], mask.expand(B, H, L, L))[:2]
    grads = orc.grads_through_both(q, clean[0], clean[1], tq, clean[2], clean[3], go, None, attn_mask=mask)[2:]
    k, v, tk, tv = (x.masked_fill(dead, 1e15) for x in (k, v, tk, tv))
    got = _all_results(q, k, v, tq, tk, tv, go, mask)
    scores = (q.double() @ clean[0].double().transpose(-1, -2) * D**-0.5).masked_fill(~mask, -math.inf)
    tops = [torch.softmax(scores, -1) @ clean[1].double().abs(), clean[1].double().abs().amax(dim=(2, 3), keepdim=True)]
    scales = [1.0, 1.0, s.double(), 1 / s.double(), 1.0]
    for n, (x, r) in enumerate(zip(got, (ro, rto, *grads))):
        x, r = x * scales[n], r.double() * scales[n]
        top = tops[n] if n < 2 else r.abs().amax(dim=(2, 3), keepdim=True)
        assert torch.isfinite(x).all() and ((x - r).abs() / top.clamp(min=1e-30)).max().item() <= 1e-5, n


@pytest.mark.gpu
@pytest.mark.parametrize("D", [32, 64, 128])
def test_a_negative_softmax_scale(D):
    (B, H, L), g, ts = _range_inputs(D)
    q, k, v, tq, tk, tv, go = ts
    got = _all_results(*ts, causal=True, sm_scale=-0.2)
    flip = [-q, k, v, -tq, tk, tv]  # the same scores at a positive one
    ref = _all_results(*flip, go, causal=True, sm_scale=0.2)
    for n, (x, r) in enumerate(zip(got, ref)):
        assert torch.equal(x, -r if n == 2 else r), n


def _workspace(B, H, L, D, tangents=0, impl=_lib.IMPL_AUTO, dtype=_lib.FP32, **fields):
    class At(int):
        shape = (B, H, L, D)
    x = At(1 << 20)
    a = _fwd_args([x] * 3, [x] * tangents, _lib.Mask(kind=_lib.MASK_NONE), [x, x if tangents else None, x, x if tangents else None], impl)
    a.dtype = dtype
    for k, v in fields.items():
        setattr(a, k, v)
    lib = _lib.load()
    return lib.jvpfa_fwd_workspace(ctypes.byref(a)), lib.jvpfa_fwd_uses_tcgen05(ctypes.byref(a))


def test_a_backward_that_finds_no_memory_for_its_workspace_goes_without(monkeypatch):
    """Host logic of the Python layer's launch, which a functorch transform of the cotangent takes: no memory, no workspace, no error."""
    spec = _lib.MaskSpec(_lib.MASK_CAUSAL)
    spec.fp32_parts = True
    x, r = torch.zeros(2, 6, 512, 64), torch.zeros(2, 6, 512)
    seen, empty = [], torch.empty

    def launch(t, entry, a):
        seen.append((a.workspace, a.workspace_bytes))
        return 0

    def no_memory(*args, **kw):
        raise torch.OutOfMemoryError("made by this test")

    monkeypatch.setattr(_lib, "_launch", launch)
    for f in (empty, no_memory):
        monkeypatch.setattr(torch, "empty", f)
        _lib.bwd(x, x, x, None, None, None, x, None, r, None, r, r, r, x, x, x, spec, 0.125)
    assert seen[0][0] and seen[0][1] == 24 * x.numel() and seen[1] == (None, 0)


def test_where_fp32_takes_the_tcgen05_kernels():
    """Host logic.  From 384 16-row tiles on at D = 64 (320 at 128, 1024 at 32), and not for one 64-row tile; later for short sequences
    with a mask that is read by element, or at D = 128 a causal one; 18, 24 or 36 bytes an element (three, four or six tensors);
    with a workspace that is large enough and aligned."""
    assert _workspace(2, 6, 512, 64) == (18 * 2 * 6 * 512 * 64, 0)  # (no workspace given: the register-tiled kernels)
    assert _workspace(2, 6, 512, 64, 1)[0] == 24 * 2 * 6 * 512 * 64
    assert _workspace(2, 6, 512, 64, 3)[0] == 36 * 2 * 6 * 512 * 64
    assert _workspace(2, 6, 496, 64)[0] == 0 and _workspace(16, 16, 64, 64)[0] == 0
    assert _workspace(2, 5, 512, 128)[0] > 0 and _workspace(2, 5, 480, 128)[0] == 0
    assert _workspace(4, 16, 256, 32)[0] > 0 and _workspace(4, 16, 128, 32)[0] == 0 and _workspace(2, 16, 448, 32)[0] == 0
    assert _workspace(1, 200, 192, 32)[0] == 0 and _workspace(1, 200, 194, 32)[0] > 0
    assert _workspace(1, 1, 32, 64, impl=_lib.IMPL_TCGEN05)[0] > 0

    def masked(kind, B, H, L, D, offset=0):
        m = _lib.Mask(kind=kind, bias_dtype=_lib.FP32, ptr=(1 << 20) + offset)
        m.stride[:] = [H * L * L, L * L, L, 1]
        return _workspace(B, H, L, D, mask=m)[0] > 0

    for kind, offset in ((_lib.MASK_BIAS, 0), (_lib.MASK_BOOL, 1)):
        assert not masked(kind, 1, 63, 160, 64, offset) and masked(kind, 1, 64, 160, 64, offset) and masked(kind, 1, 32, 192, 64, offset)
        assert not masked(kind, 1, 95, 96, 128, offset) and masked(kind, 1, 96, 96, 128, offset) and masked(kind, 1, 46, 112, 128, offset)
        assert not masked(kind, 1, 98, 208, 32, offset) and masked(kind, 1, 99, 208, 32, offset) and masked(kind, 1, 74, 224, 32, offset)
    assert masked(_lib.MASK_BOOL, 1, 39, 160, 64) and not masked(_lib.MASK_BOOL, 1, 55, 130, 64)
    assert masked(_lib.MASK_CAUSAL, 1, 39, 160, 64) and not masked(_lib.MASK_CAUSAL, 1, 95, 96, 128) and masked(_lib.MASK_NONE, 1, 54, 96, 128)
    for dtype in (_lib.BF16, _lib.FP16, _lib.FP32_TF32):
        assert _workspace(2, 6, 512, 64, dtype=dtype)[0] == 0
    assert _workspace(2, 6, 512, 64, impl=_lib.IMPL_GENERIC)[0] == 0
    need = 18 * 2 * 6 * 512 * 64
    assert _workspace(2, 6, 512, 64, workspace=1 << 20, workspace_bytes=need)[1] == 1
    assert _workspace(2, 6, 512, 64, workspace=1 << 20, workspace_bytes=need - 1)[1] == 0
    assert _workspace(2, 6, 512, 64, workspace=(1 << 20) + 8, workspace_bytes=need)[1] == 0
    assert _workspace(2, 6, 512, 64, workspace=1 << 20, workspace_bytes=need, struct_size=_lib.FwdArgs.workspace.offset)[1] == 0
    assert _workspace(2, 6, 512, 64, struct_size=_lib.FwdArgs.workspace.offset + 8) == (0, 0)
