"""The D = 128 backward through O alone: loop tiles of 64 queries and 96 keys, the latter in pieces of 16."""
import math

import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _mask(kind, B, H, L, g):
    if kind == "keys":  # ends beside the edges of a piece and of a tile
        return (torch.arange(L)[None] < torch.tensor([L, min(L, 97), max(1, L - 17)])[:B, None])[:, None, None]
    if kind == "bool":
        return (torch.rand(B, H, L, L, generator=g) > 0.5) | torch.eye(L, dtype=torch.bool)
    if kind == "window":  # whole 64-key tiles without an entry, which the kernels step over
        i = torch.arange(L)
        return ((i[:, None] - i[None]).abs() < 40)[None, None]
    return None


def _grads(q, k, v, go, mask, causal):
    a = [x.to(DEV).requires_grad_() for x in (q, k, v)]
    o = ja.attention(*a, attn_mask=None if mask is None else mask.to(DEV), causal=causal)
    return torch.autograd.grad(o, a, go.to(DEV))


@pytest.mark.parametrize("kind", ["none", "causal", "keys", "bool", "window"])
@pytest.mark.parametrize("L", [34, 64, 96, 98, 128, 130, 192, 258, 480])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_edges_of_tiles(kind, L, dt):
    """Against the float64 oracle: 2e-2 of the largest entry, at least 1, the parity tests' bound, and in the 2-norm 2e-3 for fp16 and 1e-2
    for bf16 (operands of 11 and 8 significant bits, three roundings on the longest way)."""
    B, H = 3, 2
    g = torch.Generator().manual_seed(L)
    q, k, v, go = (torch.randn(B, H, L, 128, generator=g).to(dt) for _ in range(4))
    mask, causal = _mask(kind, B, H, L, g), kind == "causal"
    full = None if mask is None else mask.expand(B, mask.shape[1], L, L)
    x = [t.double().requires_grad_() for t in (q, k, v)]
    want = torch.autograd.grad(orc.sdpa_primal(*x, attn_mask=full, causal=causal), x, go.double())
    got = _grads(q, k, v, go, mask, causal)
    assert _lib.device_status() == 0
    rel = 2e-3 if dt == torch.float16 else 1e-2
    for name, y, r in zip(("dq", "dk", "dv"), got, want):
        y = y.double().cpu()
        assert orc.max_abs_err(y, r) <= 2e-2 * max(1.0, r.abs().max().item()), name
        assert (y - r).norm() <= rel * r.norm() + 1e-6, name


@pytest.mark.parametrize("bad", [math.nan, math.inf])
def test_padding_that_is_not_finite_stays_out(bad):
    """Keys behind the last piece of 16 that holds one in range (for the forward: behind its tile of 64) reach no row, whatever tile they lie
    in; nor do those above the diagonal tile of 128 queries."""
    B, H, L, n = 1, 2, 256, 40
    g = torch.Generator().manual_seed(1)
    q, k, v, go = (torch.randn(B, H, L, 128, generator=g).half() for _ in range(4))
    mask = (torch.arange(L) < n)[None, None, None].clone()
    for where in (1, 2):
        ts = [q.clone(), k.clone(), v.clone()]
        ts[where][:, :, 64:] = bad
        dq, dk, dv = _grads(*ts, go, mask, False)
        assert torch.isfinite(dq).all() and torch.isfinite(dk[:, :, :n]).all() and torch.isfinite(dv[:, :, :n]).all()
        ts = [q.clone(), k.clone(), v.clone()]
        ts[where][:, :, 144:] = bad
        dq, dk, dv = _grads(*ts, go, None, True)
        assert torch.isfinite(dq[:, :, :128]).all()
