"""Tiles shared out among CTAs: a tile that is cut leaves partial sums in a workspace, which are added up in a fixed order."""
import ctypes
import math

import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc
from tests.test_fp32_tcgen05 import _fwd_args

DEV = "cuda:0"


def _mask(kind, B, H, L, dt, g):
    if kind == "keys":  # entries of one and of few keys, whole and ragged ones
        lens = torch.tensor([2, 1, L, L // 2 + 3, L - 1] * B)[:B] if B > 1 else torch.tensor([L // 2 + 3])
        return (torch.arange(L)[None, :] < lens[:, None])[:, None, None, :]
    if kind == "bool":
        return (torch.rand(B, H, L, L, generator=g) > 0.5) | torch.eye(L, dtype=torch.bool)
    if kind == "bias":
        return torch.randn(B, H, L, L, generator=g).clamp(-5, 5).to(dt)
    return None


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "causal", "keys", "bool", "bias"])
@pytest.mark.parametrize("B,H,L", [(1, 1, 1024), (1, 3, 1000), (5, 2, 720), (2, 12, 1024), (1, 150, 256)])
@pytest.mark.parametrize("cot,dt", [("o", torch.float16), ("t", torch.bfloat16), ("both", torch.bfloat16)])
def test_backward_of_cut_key_tiles(kind, B, H, L, cot, dt):
    """Against the float64 oracle: 2e-2 of the largest entry at least 1, the 16-bit bound of the parity tests, and in the 2-norm 1e-2 for
    bf16 and 2e-3 for fp16 (operands of 8 and 11 significant bits, four roundings on the longest way); dK and dV bit for bit the same
    from run to run, also in a workspace full of NaN."""
    g = torch.Generator().manual_seed(L + H)
    ts = [(torch.randn(B, H, L, 64, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt) for n in range(8)]
    mask, causal = _mask(kind, B, H, L, dt, g), kind == "causal"
    n = min(H, 2)  # (the oracle looks at some of the heads)
    few = lambda x: None if x is None else x[:, -n:] if x.shape[1] > 1 else x  # noqa: E731
    go, gt = ts[6] if cot != "t" else None, ts[7] if cot != "o" else None
    ref = orc.grads_through_both(*(few(x) for x in (*ts[:6], go, gt)), attn_mask=few(mask), causal=causal)
    a = [x.to(DEV).requires_grad_() for x in ts[:3]]
    m = None if mask is None else mask.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, causal=causal), tuple(a), tuple(x.to(DEV) for x in ts[3:6]))
    outs = [(x, w.to(DEV)) for x, w in ((o, go), (to, gt)) if w is not None]

    def run():
        junk = torch.full((1 << 24,), float("nan"), device=DEV)  # what the next allocations find
        del junk
        return torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs], retain_graph=True)

    first = run()
    for _ in range(3):
        for x, y in zip(run()[1:], first[1:]):
            assert torch.equal(x, y)
    assert _lib.device_status() == 0
    rel = 1e-2 if dt == torch.bfloat16 else 2e-3
    for name, x, r in zip(("dq", "dk", "dv"), first, ref[2:]):
        x = few(x).double().cpu()
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        assert (x - r).norm() <= rel * r.norm() + 1e-6, name


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "causal", "keys", "bool", "bias"])
@pytest.mark.parametrize("B,H,L,D", [(1, 1, 2048, 64), (1, 3, 1000, 64), (5, 2, 1104, 64), (2, 12, 1024, 64), (1, 3, 1330, 32)])
@pytest.mark.parametrize("dual,dt", [(False, torch.bfloat16), (True, torch.float16), (True, torch.bfloat16)])
def test_forward_of_cut_pairs(kind, B, H, L, D, dual, dt):
    """Against the float64 oracle, bounds as above (one rounding fewer on the way), lse and mu as in the parity tests; bit for bit the same
    from run to run, also in a workspace full of NaN.  A row's running maximum is one for each of its pieces."""
    g = torch.Generator().manual_seed(L + H + D)
    ts = [(torch.randn(B, H, L, D, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt) for n in range(6)]
    ts[0][..., ::7, :] *= 4  # rows whose maximum moves from piece to piece
    mask, causal = _mask(kind, B, H, L, dt, g), kind == "causal"
    n = min(H, 2)
    few = lambda x: None if x is None else x[:, -n:] if x.shape[1] > 1 else x  # noqa: E731
    o_ref, to_ref = orc.sdpa_jvp(*(few(x) for x in ts), few(mask), causal, None)[:2]
    dev, m = [x.to(DEV) for x in ts], None if mask is None else mask.to(DEV)

    def run():
        junk = torch.full((1 << 24,), float("nan"), device=DEV)
        del junk
        if not dual:
            return (ja.attention(*dev[:3], attn_mask=m, causal=causal),)
        return torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, causal=causal), tuple(dev[:3]), tuple(dev[3:]))

    first = run()
    for _ in range(3):
        for x, y in zip(run(), first):
            assert torch.equal(x, y)
    assert _lib.device_status() == 0
    rel = 1e-2 if dt == torch.bfloat16 else 2e-3
    for name, x, r in zip(("O", "tO"), first, (o_ref, to_ref)):
        x = few(x).double().cpu()
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        assert (x - r).norm() <= rel * r.norm(), name


def _spec(kind, mask):
    """A mask (on the device) as the C ABI takes it."""
    if kind == "keys":
        return _lib.MaskSpec(_lib.MASK_KVLEN, mask[:, 0, 0].sum(-1).to(torch.int32))
    if mask is None:
        return _lib.MaskSpec(_lib.MASK_CAUSAL if kind == "causal" else _lib.MASK_NONE)
    dt = _lib.BF16 if mask.dtype == torch.bool else _lib.DTYPE_ENUM[mask.dtype]
    return _lib.MaskSpec(_lib.MASK_BOOL if kind == "bool" else _lib.MASK_BIAS, mask, mask.stride(), dt)


class _Forward:
    """jvpfa_fwd on q, k, v and, as far as given, their tangents.  cut: with the workspace that it asks for, full of NaN."""

    def __init__(self, ts, spec, cut):
        B, H, L, D = ts[0].shape
        dual = len(ts) == 6
        nan = lambda *s, dt=torch.float32: torch.full(s, math.nan, device=DEV, dtype=dt)  # noqa: E731
        self.out = [nan(B, H, L, D, dt=ts[0].dtype), nan(B, H, L, D, dt=ts[0].dtype) if dual else None, nan(B, H, L), nan(B, H, L) if dual else None]
        self.args = a = _fwd_args(ts[:3], ts[3:], spec.to_c(), self.out, _lib.IMPL_TCGEN05)
        a.dtype = _lib.DTYPE_ENUM[ts[0].dtype]
        self.kept = ts, spec
        if cut:
            n = _lib.load().jvpfa_fwd_workspace(ctypes.byref(a))
            assert n > 0, "this call is not cut"
            self.workspace = nan(n // 4)
            a.workspace, a.workspace_bytes = self.workspace.data_ptr(), n
            self.ctas = (n - 16384) // (2 * 2 * (33 if dual else 17) * 128 * 16)

    def launch(self):
        _lib.check(_lib.load().jvpfa_fwd(ctypes.byref(self.args), torch.cuda.current_stream().cuda_stream), "jvpfa_fwd")
        return [x for x in self.out if x is not None]


@pytest.mark.gpu
@pytest.mark.parametrize("D", [64, 32])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("kind,B,H,L", [("none", 1, 3, 1040), ("causal", 1, 3, 1040), ("bool", 1, 3, 1040), ("bias", 1, 3, 1040),
                                        ("none", 2, 12, 2048), ("bool", 2, 12, 2048), ("bias", 2, 12, 2048)])
def test_what_is_not_finite_reaches_in_cut_pairs_what_it_reaches_in_whole_ones(kind, B, H, L, dt, D):
    """Entries that are not a number, or Inf; rows without a key, with two in two pieces, and whose bias is the type's lowest value: the
    results that are finite are those of whole pairs, and where lse is +Inf (no key, or no number) it is there."""
    g = torch.Generator(device=DEV).manual_seed(L + D)
    ts = [(torch.randn(B, H, L, D, device=DEV, generator=g) * (0.1 if n > 2 else 1.0)).to(dt) for n in range(6)]
    mask, bad_key = None, L // 3
    if kind == "bool":
        mask = torch.rand(B, H, L, L, device=DEV, generator=g) > 0.5
        mask[:, :, 5] = mask[:, :, 7] = False
        mask[:, :, 7, [bad_key, L - 1]] = True
    elif kind == "bias":
        mask = torch.randn(B, H, L, L, device=DEV, generator=g).to(dt)
        mask[:, :, 5] = torch.finfo(dt).min
        mask[:, :, 6] = -math.inf
        mask[:, :, 7, : L // 2] = -math.inf
    spec = _spec(kind, mask)
    for n in (3, 6):
        for bad in (math.nan, math.inf):
            for where in range(n):
                x = [t.clone() if m == where else t for m, t in enumerate(ts[:n])]
                x[where][:, ::2, bad_key, 7] = bad
                if where == 0:
                    x[0][:, 1] = bad  # a head throughout
                got, want = _Forward(x, spec, True).launch(), _Forward(x, spec, False).launch()
                for m, (u, w) in enumerate(zip(got, want)):
                    assert torch.equal(torch.isfinite(u), torch.isfinite(w)), (n, bad, where, m)
                    assert u.dim() == 4 or torch.equal(torch.isposinf(u), torch.isposinf(w)), (n, bad, where, m)
    assert _lib.device_status() == 0


def _replayed_behind_a_launch_that_gave_up(step):
    """What `step` returns, replayed from a graph over results of 1 with the status word set (from the host, as a thread that gives up a
    wait would) and without."""
    side = torch.cuda.Stream()  # (the legacy stream's graph nodes cannot be captured)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step()
    seen = []
    for code in (5, 0):
        if code:
            _lib.device_status_inject(code)
        try:
            for x in got:
                x.fill_(1.0)
            graph.replay()
            torch.cuda.synchronize()
            seen.append([x.clone() for x in got])
        finally:
            assert _lib.device_status(clear=True) == code
    return seen


@pytest.mark.gpu
@pytest.mark.parametrize("n", [3, 6])
@pytest.mark.parametrize("kind,B,H,L", [("none", 1, 3, 1040), ("causal", 1, 3, 1040), ("none", 2, 12, 2048), ("keys", 5, 2, 1104), ("bias", 1, 3, 1040)])
def test_rows_of_cut_pairs_are_marked_where_the_forward_gave_up(kind, B, H, L, n):
    """lse of every row holds NaN then (jvpfa_device_status), also of a pair whose shares are merged by a later kernel."""
    g = torch.Generator().manual_seed(L)
    ts = [torch.randn(B, H, L, 64, generator=g).to(torch.bfloat16).to(DEV) for _ in range(n)]
    mask = _mask(kind, B, H, L, torch.bfloat16, g)
    f = _Forward(ts, _spec(kind, None if mask is None else mask.to(DEV)), True)
    gave_up, after = _replayed_behind_a_launch_that_gave_up(f.launch)
    assert torch.isnan(gave_up[n // 3]).all()
    f.launch()
    for x, y in zip(after, [x for x in f.out if x is not None]):
        assert torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("through", ["o", "t", "both"])
@pytest.mark.parametrize("kind", ["none", "causal", "keys", "bool", "bias"])
def test_rows_of_cut_key_tiles_are_marked_where_the_backward_gave_up(kind, through):
    """Every row of dQ, dK and dV holds NaN then, also those of keys that are all padding, which weigh nothing on the line."""
    B, H, L = (8, 12, 400) if kind == "bias" else (5, 2, 720)
    g = torch.Generator().manual_seed(L)
    q, k, v, tq, tk, tv, go, gt = (torch.randn(B, H, L, 64, generator=g).to(torch.bfloat16).to(DEV) for _ in range(8))
    mask = _mask(kind, B, H, L, torch.bfloat16, g)
    m = None if mask is None else mask.to(DEV)
    a = [x.requires_grad_() for x in (q, k, v)]

    def step():
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, causal=kind == "causal"), tuple(a), (tq, tk, tv))
        outs = [(o, go)] * (through != "t") + [(to, gt)] * (through != "o")
        return list(torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs]))

    gave_up, after = _replayed_behind_a_launch_that_gave_up(step)
    for name, x in zip(("dq", "dk", "dv"), gave_up):
        assert torch.isnan(x).any(-1).all(), name
    for x, y in zip(after[1:], step()[1:]):  # (dQ has no fixed order of summation)
        assert torch.equal(x, y)


def _bias_forms(B, H, L, dt):
    g = torch.Generator().manual_seed(L)
    r = lambda *s: torch.randn(*s, generator=g).clamp(-5, 5).to(dt).to(DEV)  # noqa: E731
    forms = {"full": r(B, H, L, L), "heads": r(1, H, L, L), "entries": r(B, 1, L, L), "one": r(1, 1, L, L), "row": r(B, 1, 1, L),
             "row of each head": r(B, H, 1, L), "heads first": r(H, B, L, L).transpose(0, 1), "expanded": r(1, 1, L, L).expand(B, H, L, L),
             "wider rows": r(B, H, L, L + 24)[..., :L], "rows apart": r(B, H, L, 2, L)[:, :, :, 1], "at an odd place": r(B, H, L, L + 3)[..., 3:]}
    if L % 16 == 0:  # every row eight elements on from the one before: rows that overlap in memory
        forms["overlapping rows"] = r(1, 1, 8 * L + L).as_strided((1, 1, L, L), (9 * L, 9 * L, 8, 1))
    return forms


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,L,D", [(2, 3, 336, 64), (2, 2, 200, 64), (1, 3, 130, 128), (2, 2, 256, 128), (2, 2, 144, 32)])
def test_every_layout_of_a_bias(B, H, L, D, dt):
    """The forward with and without tangents and the backward: a bias of any layout gives what its row-major copy gives, the forward
    bit for bit, and that is the float64 oracle's within the bounds above."""
    g = torch.Generator().manual_seed(L + D)
    ts = [(torch.randn(B, H, L, D, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt).to(DEV) for n in range(8)]

    def run(m):
        a = [x.detach().requires_grad_() for x in ts[:3]]
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), tuple(a), tuple(ts[3:6]))
        dk, dv = torch.autograd.grad((o, to), a[1:], (ts[6], ts[7]))
        return ja.attention(*ts[:3], attn_mask=m), o.detach(), to.detach(), dk, dv

    for name, m in _bias_forms(B, H, L, dt).items():
        got, want = run(m), run(m.expand(B, H, L, L).contiguous())
        # (rows that begin off 16-byte boundaries, and a ragged one for all queries, are the register-tiled kernels')
        if name != "at an odd place" and (L % 16 == 0 or name not in ("row", "row of each head")):
            for x, y in zip(got[:3], want[:3]):
                assert torch.equal(x, y), name
        ref = orc.sdpa_jvp(*(x.cpu() for x in ts[:6]), m.expand(B, H, L, L).cpu(), False, None)
        for x, r in zip(got[1:3], ref):
            assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        for x, y in zip(got[3:], want[3:]):  # (a broadcast bias may be served by another backward kernel)
            assert (x.double() - y.double()).norm() <= (1e-2 if dt == torch.bfloat16 else 2e-3) * y.double().norm(), name
    assert _lib.device_status() == 0
