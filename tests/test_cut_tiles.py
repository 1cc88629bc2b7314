"""Tiles shared out among CTAs: a tile that is cut leaves partial sums in a workspace, which are added up in a fixed order."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

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
