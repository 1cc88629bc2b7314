"""Backward through tO with a bias at D = 64: one pass whose dQ is summed key tile by key tile, in a fixed order."""
import ctypes

import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cot", ["both", "t"])
@pytest.mark.parametrize("B,H,L,heads", [(8, 12, 48, 1), (4, 25, 128, 25), (2, 24, 144, 1), (4, 6, 400, 6), (3, 60, 256, 60)])
def test_bias_through_the_tangent(dt, cot, B, H, L, heads):
    """2e-2 of the largest entry at least 1, the 16-bit bound of the parity tests; and bit for bit the same from run to run, also
    in a workspace full of NaN."""
    g = torch.Generator().manual_seed(L + H)
    q, k, v, tq, tk, tv, go, gt = ((torch.randn(B, H, L, 64, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt) for n in range(8))
    mask = torch.randn(B, heads, L, L, generator=g).clamp(-5, 5).to(dt)
    go = go if cot == "both" else None
    n = min(H, 4)  # (the oracle looks at some of the heads)
    few = lambda x: None if x is None else x[:, :n]  # noqa: E731
    ref = orc.grads_through_both(*(few(x) for x in (q, k, v, tq, tk, tv, go, gt)), attn_mask=mask[:, :n])
    a = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    m = mask.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), tuple(a), tuple(x.to(DEV) for x in (tq, tk, tv)))
    outs = [(o, go)] * (cot == "both") + [(to, gt)]

    def run():
        junk = torch.full((1 << 24,), float("nan"), device=DEV)  # what the next allocations find
        del junk
        return torch.autograd.grad([x for x, _ in outs], a, [w.to(DEV) for _, w in outs], retain_graph=True)

    first = run()
    for _ in range(5):
        for x, y in zip(run(), first):
            assert torch.equal(x, y)
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    for name, x, r in zip(("dq", "dk", "dv"), first, ref[2:]):
        assert orc.max_abs_err(few(x), r) <= 2e-2 * max(1.0, r.abs().max().item()), name


def test_which_bias_backwards_take_a_workspace():
    """Host logic: from 96 key tiles on, as many bytes as a (B, H, L, L) bias of 16 bits when L is a multiple of 128; none for
    what the two launches keep.  (Where there is a GPU, and key tiles are shared out among its SMs, room for their shares of dK and dV is
    added: 16 KiB, and 128 KiB for each of the CTAs, one an SM.)"""
    sms = torch.cuda.get_device_properties(0).multi_processor_count if torch.cuda.is_available() else 0
    shares = (0, *(16384 + 131072 * n for n in range(2, sms + 1)))

    def need(L=256, D=64, B=4, H=12, go=True, gto=True, dtype=_lib.BF16, bias=_lib.BF16, flags=0, impl=_lib.IMPL_AUTO):
        x = 1 << 20
        a = _lib.BwdArgs(struct_size=ctypes.sizeof(_lib.BwdArgs), dtype=dtype, B=B, H=H, L=L, D=D, impl=impl, sm_scale=0.125, q=x, k=x, v=x,
                         lse=x, delta=x, dq=x, dk=x, dv=x, flags=flags)
        if gto:
            a.tq = a.tk = a.tv = a.gto = a.mu = a.eps = a.cterm = x
        if go:
            a.go = x
        a.mask = _lib.Mask(kind=_lib.MASK_BIAS, bias_dtype=bias, ptr=x)
        a.mask.stride[:] = [H * L * L, L * L, L, 1]
        return _lib.load().jvpfa_bwd_workspace(ctypes.byref(a))

    for through_both in (True, False):
        assert need(go=through_both) - 2 * 4 * 12 * 256 * 256 in shares
    assert need(L=272) - 3 * 4 * 12 * 272 * 64 * 4 in shares
    assert need(B=5, H=19, L=128) == 0 and need(B=6, H=16, L=16) > 0
    assert need(gto=False) == 0 and need(D=128) == 0 and need(L=264) == 0 and need(flags=2) == 0  # (2: no dK, dV asked for)
    assert need(bias=_lib.FP32) == 0 and need(bias=_lib.FP16) == 0 and need(impl=_lib.IMPL_GENERIC) == 0
    assert need(L=8192, B=1, H=4) - (1 << 29) in shares and need(L=8192, B=1, H=5) == 0
