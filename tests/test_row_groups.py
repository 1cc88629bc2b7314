"""fp32 register-tiled kernels with tangents: every split of a CTA's warps into row groups and loop parts, as the rule chooses them."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("B,H,L,D", [(1, 4, 130, 64), (3, 7, 256, 64), (2, 12, 512, 32), (2, 18, 98, 128), (4, 9, 160, 128), (1, 40, 250, 64)])
def test_against_the_oracle(B, H, L, D, causal):
    """Relative errors in the 2-norm below 1e-5: sums of up to 512 fp32 terms of products that are exact to 2^-21 (measured 3e-7 to 2e-6)."""
    g = torch.Generator().manual_seed(L)
    ts = [torch.randn(B, H, L, D, generator=g) for _ in range(8)]
    few = lambda x: x[-1:, -2:]  # noqa: E731
    ref = orc.grads_through_both(*(few(x) for x in ts), causal=causal)
    a = [x.to(DEV).requires_grad_() for x in ts[:3]]
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, causal=causal), tuple(a), tuple(x.to(DEV) for x in ts[3:6]))
    got = (o, to, *torch.autograd.grad((o, to), a, [x.to(DEV) for x in ts[6:]]))
    assert _lib.device_status() == 0
    for name, x, r in zip(("O", "tO", "dq", "dk", "dv"), got, ref):
        x = few(x.detach()).double().cpu()
        assert (x - r).norm() <= 1e-5 * r.norm(), (name, ((x - r).norm() / r.norm()).item())
