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


def _lengths(B, L):
    """Whole and ragged entries, of one and of few keys."""
    return ([L, L // 2 + 3, 2, 1, L - 1] * B)[:B] if B > 1 else [L - 3]


def _mask(kind, B, H, L, dt, g):
    if kind == "keys":
        return (torch.arange(L)[None, :] < torch.tensor(_lengths(B, L))[:, None])[:, None, None, :]
    if kind == "bool":
        return (torch.rand(B, H, L, L, generator=g) > 0.5) | torch.eye(L, dtype=torch.bool)
    if kind == "bias":
        return torch.randn(B, H, L, L, generator=g).clamp(-5, 5).to(dt)
    return None


def _host_mask(kind, H, L, dt):
    """For the host logic alone, with rows as the native layer gives them to the kernels (addresses that nothing follows)."""
    if kind in ("none", "causal", "keys"):
        return _lib.Mask(kind={"none": _lib.MASK_NONE, "causal": _lib.MASK_CAUSAL, "keys": _lib.MASK_KVLEN}[kind], kv_len=1 << 20)
    m = _lib.Mask(kind=_lib.MASK_BOOL if kind == "bool" else _lib.MASK_BIAS, bias_dtype=_lib.DTYPE_ENUM[dt], ptr=1 << 20)
    row = (L + 15) // 16 * 16
    m.stride[:] = [H * L * row, L * row, row, 1]
    return m


def _on_the_host(lengths):
    return (ctypes.c_int32 * len(lengths))(*lengths)


def _backward_is_cut(kind, B, H, L, dt, cot, lengths=None):
    """Whether the workspace that the call asks for holds more than a bias's shares of dQ."""
    lengths = _on_the_host(lengths or _lengths(B, L))
    x = 1 << 20
    a = _lib.BwdArgs(struct_size=ctypes.sizeof(_lib.BwdArgs), dtype=_lib.DTYPE_ENUM[dt], B=B, H=H, L=L, D=64, sm_scale=0.125, q=x, k=x, v=x, lse=x,
                     delta=x, dq=x, dk=x, dv=x, mask=_host_mask(kind, H, L, dt))
    if cot != "o":
        a.tq = a.tk = a.tv = a.gto = a.mu = a.eps = a.cterm = x
    if cot != "t":
        a.go = x
    if kind == "keys":
        a.kv_len_host = ctypes.addressof(lengths)
    parts = 0
    if kind == "bias" and cot != "o":
        parts = (L + 127) // 128 * B * H * L * 64 * 4
    else:
        a.dq_accum = x
    return _lib.load().jvpfa_bwd_workspace(ctypes.byref(a)) > parts


def _forward_is_cut(kind, B, H, L, D, dt, dual, lengths=None):
    lengths = _on_the_host(lengths or _lengths(B, L))
    class At(int):
        shape = (B, H, L, D)
    x = At(1 << 20)
    a = _fwd_args([x] * 3, [x] * 3 * dual, _host_mask(kind, H, L, dt), [x, x if dual else None, x, x if dual else None], _lib.IMPL_AUTO)
    a.dtype, a.mask_bits = _lib.DTYPE_ENUM[dt], x if kind == "bool" else None
    if kind == "keys":
        a.kv_len_host = ctypes.addressof(lengths)
    return _lib.load().jvpfa_fwd_workspace(ctypes.byref(a)) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "causal", "keys", "bool", "bias"])
@pytest.mark.parametrize("B,H,L", [(1, 1, 1024), (1, 3, 1000), (5, 2, 720), (2, 12, 1024), (1, 150, 256), (36, 1, 720)])
@pytest.mark.parametrize("cot,dt", [("o", torch.float16), ("t", torch.bfloat16), ("both", torch.bfloat16)])
def test_backward_of_cut_key_tiles(kind, B, H, L, cot, dt):
    """Against the float64 oracle: 2e-2 of the largest entry at least 1, the 16-bit bound of the parity tests, and in the 2-norm 1e-2 for
    bf16 and 2e-3 for fp16 (operands of 8 and 11 significant bits, four roundings on the longest way); dK and dV bit for bit the same
    from run to run, also in a workspace full of NaN.  (Left whole, by the rule: causal ones of many heads, and short ones of 150; the two
    launches' are a mask whose rows are not whole 16-byte pieces, and a bias through tO below 96 key tiles.)"""
    left = (kind == "causal" and B * H >= 24) or H == 150 or (kind in ("bool", "bias") and L % 16 != 0)
    left = left or (kind == "bias" and cot != "o" and (L + 127) // 128 * B * H < 96)
    assert _backward_is_cut(kind, B, H, L, dt, cot) != left
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
@pytest.mark.parametrize("B,H,L,D", [(1, 1, 2048, 64), (1, 3, 1000, 64), (5, 2, 1104, 64), (2, 12, 1024, 64), (1, 3, 1330, 32), (2, 12, 2048, 64)])
@pytest.mark.parametrize("dual,dt", [(False, torch.bfloat16), (True, torch.float16), (True, torch.bfloat16)])
def test_forward_of_cut_pairs(kind, B, H, L, D, dual, dt):
    """Against the float64 oracle, bounds as above (one rounding fewer on the way); bit for bit the same from run to run, also in a workspace
    full of NaN.  A row's running maximum is one for each of its pieces.  (Left whole, by the rule: 24 heads of L 1024, and causal and padded ones.)"""
    assert _forward_is_cut(kind, B, H, L, D, dt, dual) != (B * H == 24 and (L == 1024 or kind in ("causal", "keys")))
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
    """jvpfa_fwd on q, k, v and, as far as given, their tangents.  cut: with the workspace that it asks for, full of NaN (key padding: that
    it asks for where the host says that no key is padding, which decides nothing else)."""

    def __init__(self, ts, spec, cut):
        B, H, L, D = ts[0].shape
        dual = len(ts) == 6
        nan = lambda *s, dt=torch.float32: torch.full(s, math.nan, device=DEV, dtype=dt)  # noqa: E731
        self.out = [nan(B, H, L, D, dt=ts[0].dtype), nan(B, H, L, D, dt=ts[0].dtype) if dual else None, nan(B, H, L), nan(B, H, L) if dual else None]
        self.args = a = _fwd_args(ts[:3], ts[3:], spec.to_c(), self.out, _lib.IMPL_TCGEN05)
        a.dtype = _lib.DTYPE_ENUM[ts[0].dtype]
        self.kept = ts, spec, _on_the_host([L] * B)  # (what the arguments point to)
        if spec.kind == _lib.MASK_KVLEN:
            a.kv_len_host = ctypes.addressof(self.kept[2])
        if cut:
            n = _lib.load().jvpfa_fwd_workspace(ctypes.byref(a))
            assert n > 0, "this call is not cut"
            self.workspace = nan(n // 4)
            a.workspace, a.workspace_bytes = self.workspace.data_ptr(), n
            self.ctas = (n - 16384) // (2 * 2 * (33 if dual else 17) * 128 * 16)

    def launch(self):
        _lib.check(_lib.load().jvpfa_fwd(ctypes.byref(self.args), torch.cuda.current_stream().cuda_stream), "jvpfa_fwd")
        return [x for x in self.out if x is not None]

    def begins(self):
        """[pair, key tile] where each of the CTAs began."""
        return self.workspace[:4096].view(torch.int32)[:2 * self.ctas].view(-1, 2).tolist()


def _begins(weights, steps, first, G):
    """Where G CTAs begin, [item, step], on the line of the items from `first` on: weights[w] is how long item w is on it (0: it is not), two
    more than the steps that it stands for; it has steps[w].  A cut leaves two steps on either side, or is moved to the item's beginning or its end
    (of an item with fewer than two steps, always to its end)."""
    line = [(w, x) for w, x in enumerate(weights) if w >= first and x > 0]
    total = sum(x for _, x in line)
    begins = []
    for c in range(G):
        pos, at = total * c // G, [len(weights), 0] if c else [first, 0]
        for w, x in line if c else ():
            if pos < x:
                s = pos - 2 if pos >= 4 else 0
                at = [w, s] if s <= steps[w] - 2 else [w + 1, 0]
                break
            pos -= x
        begins.append(at)
    return begins


def _line_of_pairs(kind, B, H, L, lens):
    """(weights, steps) of the forward's query pairs."""
    P, N = (L + 255) // 256, (L + 63) // 64
    steps = [min(N, 4 * r + 4) if kind == "causal" else (lens[b] + 63) // 64 if kind == "keys" else N for b in range(B) for _ in range(H) for r in range(P)]
    stands_for = [4 * r + 4 for _ in range(B * H) for r in range(P)] if kind == "causal" else steps
    return [x + 2 for x in stands_for], steps


@pytest.mark.parametrize("kind", ["none", "causal", "keys"])
def test_pieces_of_a_line_of_pairs(kind):
    """On the model that the kernel is held against below: pieces follow one another, are alike, and no cut leaves fewer than two steps."""
    g = torch.Generator().manual_seed(3)
    r = lambda lo, hi: int(torch.randint(lo, hi + 1, (1,), generator=g))  # noqa: E731
    for _ in range(60):
        B, H, L = r(1, 40), r(1, 12), r(32, 3000)
        lens = [r(0, L) for _ in range(B)]
        weights, steps = _line_of_pairs(kind, B, H, L, lens)
        G = min(148, sum(steps) // 4)
        if G < 2:
            continue
        whole = 0 if kind != "none" else len(steps) // G
        begins = _begins(weights, steps, whole * G, G) + [[len(steps), 0]]
        piece = sum(weights[whole * G:]) / G
        for (w0, s0), (w1, s1) in zip(begins, begins[1:]):
            assert (w0, s0) <= (w1, s1) and (s1 == 0 or 2 <= s1 <= steps[w1] - 2)
            took = sum(weights[w0:w1]) + (s1 + 2 if s1 else 0) - (s0 + 2 if s0 else 0)
            assert took <= piece + 8, (took, piece)  # (a first cut moves back by up to 3, a last one on by up to 4, and rounding)


@pytest.mark.gpu
@pytest.mark.parametrize("dt,n", [(torch.bfloat16, 6), (torch.float16, 3)])
@pytest.mark.parametrize("kind,B,H,L,D,whole", [
    ("none", 1, 1, 2048, 64, 0), ("causal", 1, 3, 1040, 64, 0), ("keys", 5, 2, 1104, 64, 0), ("keys", 38, 1, 1024, 64, 0),
    ("none", 38, 1, 1024, 64, 1), ("none", 2, 12, 2048, 64, 1), ("bool", 2, 12, 2048, 64, 1), ("bias", 2, 12, 2048, 64, 1),
    ("none", 4, 16, 2048, 64, 3), ("bool", 1, 3, 1040, 32, 0), ("bias", 1, 3, 1040, 32, 0),
])
def test_where_pairs_are_cut_and_their_statistics(kind, B, H, L, D, whole, dt, n):
    """O, tO, lse and mu of the first and the last head against the float64 oracle, in the parity tests' bounds and as above, with empty
    sequences and rows that have no key; and every CTA's beginning against the model."""
    g = torch.Generator().manual_seed(L + H + B)
    ts = [(torch.randn(B, H, L, D, generator=g) * (0.1 if m > 2 else 1.0)).to(dt) for m in range(n)]
    ts[0][..., ::7, :] *= 4
    mask = _mask(kind, B, H, L, dt, g)
    if kind == "keys":
        mask[1] = False  # an empty sequence
    if kind == "bool":
        mask[:, :, 5] = False
    f = _Forward([x.to(DEV) for x in ts], _spec(kind, None if mask is None else mask.to(DEV)), True)
    got = dict(zip(("o", "to", "lse", "mu") if n == 6 else ("o", "lse"), f.launch()))
    weights, steps = _line_of_pairs(kind, B, H, L, mask[:, 0, 0].sum(-1).tolist() if kind == "keys" else None)
    assert f.begins() == _begins(weights, steps, whole * f.ctas, f.ctas)
    assert _lib.device_status() == 0
    rel = 1e-2 if dt == torch.bfloat16 else 2e-3
    for b, h in ((0, 0), (B - 1, H - 1)) + (((1, 0),) if kind == "keys" else ()):
        one = lambda x: None if x is None else x[b:b + 1, h:h + 1] if x.shape[1] > 1 else x[b:b + 1]  # noqa: E731
        want = orc.tiled_forward(*(one(x) for x in ts), attn_mask=one(mask), causal=kind == "causal", block=256)
        for name, x in got.items():
            x, r = one(x).double().cpu(), torch.from_numpy(want[name])
            none = torch.isinf(r)  # (lse of a row without a key)
            assert torch.equal(torch.isposinf(x), none), name
            x, r = x.masked_fill(none, 0.0), r.masked_fill(none, 0.0)
            assert orc.max_abs_err(x, r) <= {"mu": 5e-2}.get(name, 2e-2 * max(1.0, r.abs().max().item()) if name != "lse" else 2e-2), name
            assert name in ("lse", "mu") or (x - r).norm() <= rel * r.norm(), name


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
def test_key_padding_is_cut_by_its_lengths():
    """Short entries leave whole tiles the better deal, as if the tensors were that short; so they are where the host does not know the lengths."""
    dt = torch.bfloat16
    for (B, H, L), lengths, forward, backward in (((8, 2, 1024), [1024] * 8, True, False), ((8, 2, 1024), [512] * 8, False, True),
                                                  ((8, 2, 1024), [32] * 8, False, None), ((1, 4, 4096), [4096], True, False), ((1, 4, 4096), [1024], True, True),
                                                  ((1, 4, 4096), [128], False, True), ((2, 20, 1000), [280, 400], False, False),
                                                  ((2, 20, 512), [268, 384], False, False), ((8, 12, 256), [100] * 8, False, False)):
        for dual in (False, True):
            assert _forward_is_cut("keys", B, H, L, 64, dt, dual, lengths) == forward, (B, H, L, lengths)
        for cot in ("o", "t", "both") if backward is not None else ():
            assert _backward_is_cut("keys", B, H, L, dt, cot, lengths) == backward, (B, H, L, lengths, cot)
    x = torch.zeros(1, 4, 4096, 64, dtype=dt, device=DEV)
    f = _Forward([x, x, x], _lib.MaskSpec(_lib.MASK_KVLEN, torch.full((1,), 4096, dtype=torch.int32, device=DEV)), True)
    f.args.kv_len_host = None
    assert _lib.load().jvpfa_fwd_workspace(ctypes.byref(f.args)) == 0
    spec = ja.classify_mask(torch.ones(1, 1, 1, 4096, dtype=torch.bool, device=DEV), False, 3, 4, 4096, dt, True)[0]
    assert spec.kv_len_host == [4096] * 3


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
