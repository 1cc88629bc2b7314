"""Key padding at D = 64 with more items than SMs: the persistent kernels take the longest sequences first, of up to 64 of them."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,H,L", [(1, 80, 520), (5, 24, 300), (64, 2, 300), (65, 2, 300)])
@pytest.mark.parametrize("cot", ["both", "t", "o"])
def test_key_padding_longest_first(B, H, L, cot):
    """2e-2 of the largest entry, at least 1: the 16-bit bound of the parity tests.  Equal lengths, one and full length among them."""
    g = torch.Generator().manual_seed(B)
    q, k, v, tq, tk, tv, go, gt = ((torch.randn(B, H, L, 64, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).half() for n in range(8))
    lens = torch.randint(1, L + 1, (B,), generator=g)
    lens[0], lens[B // 2], lens[-1] = L, 1, lens[B // 3]
    mask = (torch.arange(L)[None] < lens[:, None])[:, None, None]
    go, gt = (go if cot != "t" else None), (gt if cot != "o" else None)
    ref = orc.grads_through_both(q, k, v, tq, tk, tv, go, gt, attn_mask=mask.expand(B, 1, L, L))
    a = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    m = mask.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), tuple(a), tuple(x.to(DEV) for x in (tq, tk, tv)))
    outs = [(x, w) for x, w in ((o, go), (to, gt)) if w is not None]
    got = (o, to, *torch.autograd.grad([x for x, _ in outs], a, [w.to(DEV) for _, w in outs]))
    torch.cuda.synchronize()
    assert _lib.device_status() == 0
    for name, x, r in zip(("O", "tO", "dq", "dk", "dv"), got, ref):
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
