"""Hessian-vector products of views: the incoming gradients' layout against that of q, k and v, which the kernels read in place."""
import pytest
import torch

from jvp_flash_attention_b200 import jvp_attention as ja
from tests import _oracle_launchers as stand_in
from tests.test_autograd_wiring import cpu_kernels  # noqa: F401

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


@pytest.mark.parametrize("inputs", ["views", "packed", "row-major"])
@pytest.mark.parametrize("direction", ["views", "packed", "row-major", "q alone"])
def test_what_the_kernels_are_handed(cpu_kernels, monkeypatch, inputs, direction):  # noqa: F811
    """Tangents in the layout of q, k and v as far as that takes no copy of q, k or v; else row-major, and never copied where they come so."""
    B, H, L, D = 2, 3, 32, 32
    g = torch.Generator().manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=g, dtype=torch.float64)  # noqa: E731

    def three(layout):
        if layout == "packed":
            return list(r(B, L, 3, H, D).permute(2, 0, 3, 1, 4))
        if layout == "views":
            return [r(B, L, H, D).transpose(1, 2) for _ in range(3)]
        return [r(B, H, L, D) for _ in range(3)]

    seen = []

    def launch_fwd(*a):
        seen.append(a)
        return tuple(None if y is None else y.contiguous() for y in stand_in.launch_fwd(*a))

    monkeypatch.setattr(ja, "_launch_fwd", launch_fwd)
    x = [t.requires_grad_() for t in three(inputs)]
    u = three("row-major" if direction == "q alone" else direction)
    o = ja.attention(*x)
    grads = torch.autograd.grad(o, x, r(B, H, L, D), create_graph=True)
    if direction == "q alone":
        torch.autograd.grad(grads[0], x, u[0])
        u = u[:1]
    else:
        torch.autograd.grad(grads, x, u)
    given, in_place = seen[-1][3:6], inputs == "views" or inputs == direction
    for t in given:
        assert t.stride() == x[0].stride() if in_place else t.is_contiguous()
    for t, y in zip(given, u):
        assert torch.equal(t, y)
        if y.stride() == t.stride():
            assert t.data_ptr() == y.data_ptr()
