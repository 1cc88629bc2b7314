"""The D = 32 backward in one pass: dQ's shares, one for each key tile, are summed in their order."""
import ctypes

import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc
from tests.test_cut_tiles import _replayed_behind_a_launch_that_gave_up

DEV = "cuda:0"


def _mask(kind, B, H, L, dt, g):
    if kind == "bool":
        return (torch.rand(B, H, L, L, generator=g) > 0.5) | torch.eye(L, dtype=torch.bool)
    if kind == "bias":
        return torch.randn(B, H, L, L, generator=g).clamp(-5, 5).to(dt)
    return None


def _call(ts, mask, causal, through):
    a = [x.to(DEV).requires_grad_() for x in ts[:3]]
    m = None if mask is None else mask.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, causal=causal), tuple(a), tuple(x.to(DEV) for x in ts[3:6]))
    outs = [(o, ts[6].to(DEV))] * (through != "t") + [(to, ts[7].to(DEV))] * (through != "o")
    return lambda: torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs], retain_graph=True)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "causal", "bool", "bias"])
@pytest.mark.parametrize("B,H,L", [(2, 40, 66), (5, 16, 128), (4, 20, 130), (2, 18, 512), (1, 1, 1024), (1, 2, 1098), (1, 3, 1544)])
@pytest.mark.parametrize("through,dt", [("o", torch.float16), ("t", torch.bfloat16), ("both", torch.float16)])
def test_against_the_oracle(kind, B, H, L, through, dt):
    """2e-2 of the largest entry, at least 1, the 16-bit bound of the parity tests, and in the 2-norm 2e-3 for fp16 and 1e-2 for bf16 (operands of 11
    and 8 significant bits, four roundings on the longest way); bit for bit the same from run to run, also in a workspace full of NaN."""
    g = torch.Generator().manual_seed(L + H)
    ts = [(torch.randn(B, H, L, 32, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt) for n in range(8)]
    mask, causal = _mask(kind, B, H, L, dt, g), kind == "causal"
    run = _call(ts, mask, causal, through)

    def again():
        junk = torch.full((1 << 24,), float("nan"), device=DEV)  # what the next allocations find
        del junk
        return run()

    got = again()
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(again(), got))
    assert _lib.device_status() == 0
    few = lambda x: None if x is None else x[-1:, -1:]  # noqa: E731
    ref = orc.grads_through_both(*(few(x) for x in ts[:6]), few(ts[6]) if through != "t" else None, few(ts[7]) if through != "o" else None,
                                 attn_mask=few(mask), causal=causal)
    rel = 2e-3 if dt == torch.float16 else 1e-2
    for name, x, r in zip(("dq", "dk", "dv"), got, ref[2:]):
        x = few(x).double().cpu()
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        assert (x - r).norm() <= rel * r.norm() + 1e-6, name


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["none", "causal", "bool", "bias"])
@pytest.mark.parametrize("through", ["o", "both"])
def test_rows_are_marked_where_it_gave_up(kind, through):
    """Every row of dQ, dK and dV holds NaN then (jvpfa_device_status)."""
    B, H, L = 2, 18, 520
    g = torch.Generator().manual_seed(L)
    ts = [torch.randn(B, H, L, 32, generator=g).to(torch.bfloat16) for _ in range(8)]
    mask = _mask(kind, B, H, L, torch.bfloat16, g)
    a = [x.to(DEV).requires_grad_() for x in ts[:3]]
    rest, m = [x.to(DEV) for x in ts[3:]], None if mask is None else mask.to(DEV)

    def step():
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m, causal=kind == "causal"), tuple(a), tuple(rest[:3]))
        outs = [(o, rest[3])] + [(to, rest[4])] * (through == "both")
        return list(torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs]))

    gave_up, after = _replayed_behind_a_launch_that_gave_up(step)
    for name, x in zip(("dq", "dk", "dv"), gave_up):
        assert torch.isnan(x).any(-1).all(), name
    assert all(torch.equal(x, y) for x, y in zip(after, step()))


def test_which_calls_take_a_workspace():
    """Host logic: a share of dQ for each key tile, up to a quarter of a GiB; none for key padding, tile bitmaps, dQ alone, and few short key tiles.
    (Where there is a GPU, and key tiles are shared out among its SMs, room for their shares of dK and dV is added.)"""
    x = 1 << 20

    def need(L=1024, B=2, H=4, kind=_lib.MASK_NONE, flags=0, **fields):
        a = _lib.BwdArgs(struct_size=ctypes.sizeof(_lib.BwdArgs), dtype=_lib.BF16, B=B, H=H, L=L, D=32, sm_scale=0.2, q=x, k=x, v=x, lse=x, delta=x,
                         dq=x, dk=x, dv=x, go=x, flags=flags)
        a.mask = _lib.Mask(kind=kind, bias_dtype=_lib.BF16, ptr=x, kv_len=x)
        a.mask.stride[:] = [H * L * L, L * L, L, 1]
        for name, value in fields.items():
            setattr(a, name, value)
        return _lib.load().jvpfa_bwd_workspace(ctypes.byref(a))

    assert need() >= 8 * 8 * 1024 * 32 * 4 and need(kind=_lib.MASK_CAUSAL) > 0 and need(kind=_lib.MASK_BIAS) > 0
    assert need(kind=_lib.MASK_KVLEN) == 0 and need(flags=2) == 0 and need(kind=_lib.MASK_BOOL) == 0
    assert need(kind=_lib.MASK_BOOL, mask_bits=x, mask_bits_t=x) > 0
    assert need(kind=_lib.MASK_BOOL, mask_bits=x, mask_bits_t=x, mask_tile_live=x, mask_tile_live_t=x) == 0
    assert need(L=512, B=1, H=18) == 0 and need(L=512, B=1, H=19) > 0 and need(L=64, B=8, H=16) == 0
    assert need(L=512, B=1, H=35, kind=_lib.MASK_CAUSAL) == 0 and need(L=512, B=1, H=36, kind=_lib.MASK_CAUSAL) > 0
    assert need(L=8192, B=1, H=4) > 0 and need(L=8192, B=1, H=5) == 0 and need(L=1032, kind=_lib.MASK_BIAS) == 0
