"""The D = 64 backward through tO in one pass, of a bias whose length does not fill whole 32-byte pieces: padded rows, and a last
sub-tile whose 16 queries are there in part."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("through", ["t", "both"])
@pytest.mark.parametrize("B,H,L", [(4, 12, 130), (4, 12, 200), (2, 16, 270), (2, 16, 386), (1, 12, 1034)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_against_the_oracle(B, H, L, dt, through):
    """2e-2 of the largest entry, at least 1, the 16-bit bound of the parity tests, and in the 2-norm 2e-3 for fp16 and 1e-2 for bf16 (operands
    of 11 and 8 significant bits, four roundings on the longest way); bit for bit the same from run to run."""
    g = torch.Generator().manual_seed(L)
    q, k, v, tq, tk, tv, go, gt = ((torch.randn(B, H, L, 64, generator=g) * (0.1 if n in (3, 4, 5) else 1.0)).to(dt) for n in range(8))
    bias = torch.randn(B, H, L, L, generator=g).clamp(-5, 5).to(dt)
    go = go if through == "both" else None
    few = lambda x: None if x is None else x[-1:, -2:]  # noqa: E731
    ref = orc.grads_through_both(*(few(x) for x in (q, k, v, tq, tk, tv, go, gt)), attn_mask=few(bias))
    a = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    m = bias.to(DEV)
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), tuple(a), tuple(x.to(DEV) for x in (tq, tk, tv)))
    outs = [(x, w.to(DEV)) for x, w in ((o, go), (to, gt)) if w is not None]

    def run():
        return torch.autograd.grad([x for x, _ in outs], a, [w for _, w in outs], retain_graph=True)

    got = run()
    assert all(torch.equal(x, y) for x, y in zip(run(), got))
    assert _lib.device_status() == 0
    rel = 2e-3 if dt == torch.float16 else 1e-2
    for name, x, r in zip(("dq", "dk", "dv"), got, ref[2:]):
        x = few(x).double().cpu()
        assert orc.max_abs_err(x, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        assert (x - r).norm() <= rel * r.norm() + 1e-6, name
