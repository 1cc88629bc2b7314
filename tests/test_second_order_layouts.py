"""Hessian-vector products of views: the incoming gradients' layout against that of q, k and v, which the kernels read in place."""
import pytest
import torch

from jvp_flash_attention_b200 import jvp_attention as ja

DEV = "cuda:0"


@pytest.mark.gpu
@pytest.mark.parametrize("D,dt", [(64, torch.bfloat16), (128, torch.float16), (64, torch.float32)])
@pytest.mark.parametrize("inputs", ["views", "packed", "row-major"])
@pytest.mark.parametrize("direction", ["view", "row-major", "expanded", "odd place"])
def test_layouts_give_what_row_major_tensors_give(D, dt, inputs, direction):
    """Bit for bit: the same launches on the same values (of dQ alone, whose sum has a fixed order)."""
    B, H, L = 2, 3, 130
    g = torch.Generator(device=DEV).manual_seed(D)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dt)  # noqa: E731
    if inputs == "packed":
        q, k, v = r(B, L, 3, H, D).permute(2, 0, 3, 1, 4)
    elif inputs == "views":
        q, k, v = (r(B, L, H, D).transpose(1, 2) for _ in range(3))
    else:
        q, k, v = (r(B, H, L, D) for _ in range(3))
    go = r(B, H, L, D)
    if direction == "expanded":
        u = r(B, H, 1, D).expand(B, H, L, D)
    elif direction == "odd place":
        u = r(B * H * L * D + 1)[1:].view(B, L, H, D).transpose(1, 2)
    else:
        u = r(B, L, H, D).transpose(1, 2) if direction == "view" else r(B, H, L, D)

    def hvp(q, k, v, u):
        x = [t.detach().requires_grad_() for t in (q, k, v)]
        o = ja.attention(*x, causal=True)
        (dq,) = torch.autograd.grad(o, x[0], go, create_graph=True)
        return (dq, *torch.autograd.grad(dq, x[:1], u))

    got, want = hvp(q, k, v, u), hvp(*(t.contiguous() for t in (q, k, v, u)))
    assert all(torch.equal(a, b) for a, b in zip(got, want))
