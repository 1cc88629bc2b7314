"""A bias on the tensor-core kernels: tiles are given back behind their last read, and rows are copied only where a kernel takes the copy."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja

DEV = "cuda:0"


def _tensors(n, B, H, L, D, dt=torch.bfloat16):
    g = torch.Generator(device=DEV).manual_seed(L)
    return [torch.randn(B, H, L, D, generator=g, device=DEV).to(dt) for _ in range(n)], g


@pytest.mark.gpu
@pytest.mark.parametrize("tangents", [False, True])
@pytest.mark.parametrize("B,H,L,D", [(2, 12, 2048, 64), (2, 20, 1000, 64), (2, 9, 2048, 128), (1, 16, 1000, 32)])
def test_forward_repeats_itself(B, H, L, D, tangents):
    """Bit for bit over 200 launches: a tile that was copied over what threads had yet to read would show in some of them."""
    ts, g = _tensors(6, B, H, L, D)
    bias = torch.randn(B, H, L, L, generator=g, device=DEV).to(torch.bfloat16)

    def run():
        if tangents:
            return torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=bias), tuple(ts[:3]), tuple(ts[3:]))
        return (ja.attention(*ts[:3], attn_mask=bias),)

    want = run()
    same = torch.ones((), dtype=torch.bool, device=DEV)
    for _ in range(200):
        for x, y in zip(run(), want):
            same &= (x == y).all()
    assert same.item() and _lib.device_status() == 0


def _backward_bytes(H, L, D, through, room):
    """What a backward holds at most, beside what was there: its gradients, scratch, workspace and copies; and the bytes of its bias."""
    ts, g = _tensors(8, 1, H, L, D)
    bias = torch.zeros(1, H, L, L + room, device=DEV, dtype=torch.bfloat16)[..., :L]
    a = [x.requires_grad_() for x in ts[:3]]
    o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=bias), tuple(a), tuple(ts[3:6]))
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    torch.autograd.grad(o if through == "o" else to, a, ts[6])
    return torch.cuda.max_memory_allocated() - before, bias.numel() * 2


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,through", [(64, 64, "t"), (61, 32, "o"), (4, 64, "t"), (20, 64, "o"), (20, 128, "t")])
def test_no_copy_for_two_launches(H, D, through):
    """L % 16 == 8: rows that the two launches read in place, more key tiles than the one pass has a workspace for, fewer than it takes, or not its call."""
    held, bias = _backward_bytes(H, 2056, D, through, 0)
    assert held < bias / 2


@pytest.mark.gpu
@pytest.mark.parametrize("H,D,through", [(4, 32, "o"), (8, 64, "t")])
def test_one_pass_reads_rows_with_room_in_place(H, D, through):
    copied, bias = _backward_bytes(H, 2056, D, through, 0)
    in_place, _ = _backward_bytes(H, 2056, D, through, 8)
    assert bias * 0.9 < copied - in_place < bias * 1.1
