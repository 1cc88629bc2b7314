"""The register-tiled kernels under boolean masks with tile bitmaps: tiles without a true entry are stepped over."""
import pytest
import torch

from jvp_flash_attention_b200 import _lib
from jvp_flash_attention_b200 import jvp_attention as ja
from oracle import jvp_attention_oracle as orc

DEV = "cuda:0"


def _mask(kind, B, H, L, g):
    i = torch.arange(L)
    if kind == "window":
        return ((i[:, None] - i[None]).abs() < 50)[None, None].expand(B, H, L, L).clone()
    if kind == "documents":
        cuts = torch.sort(torch.randint(1, L, (B, 3), generator=g), dim=1).values
        doc = (i[None, :, None] >= cuts[:, None, :]).sum(-1)
        m = (doc[:, :, None] == doc[:, None, :])[:, None].expand(B, H, L, L).clone()
        m[:, -1, 128:256] = False  # a query tile without a key
        return m
    m = torch.rand(B, 1, 1, L, generator=g) > 0.3  # one row for every query, whole key tiles without an entry
    m[..., 64:192] = False
    m[..., 5] = True
    return m


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["window", "documents", "keys"])
@pytest.mark.parametrize("B,H,L", [(1, 2, 450), (3, 9, 330), (2, 24, 448)])
@pytest.mark.parametrize("D,dt,impl", [(64, torch.float32, "fp32"), (128, torch.float32, "fp32"), (32, torch.float32, "tf32"), (64, torch.float16, "fp32")])
def test_same_as_visiting_every_tile(kind, B, H, L, D, dt, impl):
    """Bit for bit (dead tiles add zeros), at every split of a CTA's warps; and against the float64 oracle, relative errors in the 2-norm below 1e-5
    for fp32, 2e-3 for one TF32 product and fp16 (11 significant bits)."""
    g = torch.Generator().manual_seed(L + D)
    ts = [torch.randn(B, H, L, D, generator=g).to(dt) for _ in range(8)]
    m = _mask(kind, B, H, L, g)
    md = m.to(DEV)
    spec = _lib.MaskSpec(_lib.MASK_BOOL, md.view(torch.uint8), tuple(0 if n == 1 else s for n, s in zip(md.shape, md.stride())))
    if dt == torch.float32:
        spec.fp32_mode = impl
    live, _, live_t = _lib.mask_tiles(spec, L)
    q, k, v, tq, tk, tv, go, gt = (x.to(DEV) for x in ts)
    runs = []
    for bitmaps in ((None, None), (live, live_t)):
        spec.tile_live, spec.tile_live_t = bitmaps
        o, to = torch.empty_like(q), torch.empty_like(q)
        lse, mu = (torch.empty(B, H, L, device=DEV) for _ in range(2))
        _lib.fwd(q, k, v, tq, tk, tv, o, to, lse, mu, spec, D**-0.5, _lib.IMPL_GENERIC)
        stats = torch.empty(3, B, H, L, device=DEV)
        _lib.bwd_preprocess(o, to, go, gt, mu, *stats)
        grads = [torch.empty_like(q) for _ in range(3)]
        _lib.bwd(q, k, v, tq, tk, tv, go, gt, lse, mu, *stats, *grads, spec, D**-0.5, _lib.IMPL_GENERIC)
        runs.append((o, to, lse, mu, *grads))
    for x, y in zip(*runs):
        assert torch.equal(x, y)
    few = lambda x: x[:1, :1]  # noqa: E731
    ref = orc.grads_through_both(*(few(x) for x in ts), attn_mask=few(m).expand(1, 1, L, L))
    rel = 1e-5 if dt == torch.float32 and impl == "fp32" else 2e-3
    for name, x, r in zip(("O", "tO", "dq", "dk", "dv"), (*runs[1][:2], *runs[1][4:]), ref):
        x = few(x).double().cpu()
        assert (x - r).norm() <= rel * r.norm(), (name, ((x - r).norm() / r.norm()).item())


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,L,D", [(1, 2, 450, 64), (2, 24, 448, 32)])
@pytest.mark.parametrize("missing", ["mask_tile_live", "mask_tile_live_t"])
def test_one_bitmap_alone_decides_nothing(monkeypatch, B, H, L, D, missing):
    """The backward takes both bitmaps or neither; here the other one calls every tile dead."""
    g = torch.Generator().manual_seed(L + D)
    q, k, v, _, _, _, go, _ = (torch.randn(B, H, L, D, generator=g).to(DEV) for _ in range(8))
    m = _mask("window", B, H, L, g).to(DEV)
    spec = _lib.MaskSpec(_lib.MASK_BOOL, m.view(torch.uint8), m.stride())
    live, _, live_t = (torch.zeros_like(x) for x in _lib.mask_tiles(spec, L))
    o, lse, stats = torch.empty_like(q), torch.empty(B, H, L, device=DEV), torch.empty(3, B, H, L, device=DEV)
    _lib.fwd(q, k, v, None, None, None, o, None, lse, None, spec, D**-0.5, _lib.IMPL_GENERIC)
    _lib.bwd_preprocess(o, None, go, None, None, *stats)
    launch = _lib._launch

    def one_bitmap(x, fn, a):
        setattr(a, missing, None)
        return launch(x, fn, a)

    runs = []
    for tiles in ((None, None), (live, live_t)):
        spec.tile_live, spec.tile_live_t = tiles
        if tiles[0] is not None:
            monkeypatch.setattr(_lib, "_launch", one_bitmap)
        grads = [torch.empty_like(q) for _ in range(3)]
        _lib.bwd(q, k, v, None, None, None, go, None, lse, None, *stats, *grads, spec, D**-0.5, _lib.IMPL_GENERIC)
        runs.append(grads)
    for x, y in zip(*runs):
        assert torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["data", "graph", "functorch"])
@pytest.mark.parametrize("B,H,L,D", [(1, 2, 450, 64), (2, 6, 448, 128), (1, 3, 300, 32)])
def test_a_window_written_behind_the_version_counter(how, B, H, L, D):
    """fp32: what the kernels read are the mask's present entries, also where the verified ones left tiles dead."""
    g = torch.Generator().manual_seed(D)
    q, k, v, tq, tk, tv, go, gt = (torch.randn(B, H, L, D, generator=g).to(DEV) for _ in range(8))
    first = _mask("window", 1, 1, L, g).to(DEV)
    second = first.flip(-1) | torch.eye(L, dtype=torch.bool, device=DEV)
    a = [x.requires_grad_() for x in (q, k, v)]

    def run(m):
        if how == "functorch":
            o, back = torch.func.vjp(lambda *x: ja.attention(*x, attn_mask=m), *(x.detach() for x in a))
            return (o, *back(go))
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m), tuple(a), (tq, tk, tv))
        return (o, to, *torch.autograd.grad((o, to), a, (go, gt)))

    want = [x.detach().clone() for x in run(second.clone())]
    mask = first.clone()
    if how != "graph":
        run(mask)
        mask.data.copy_(second)
        got = run(mask)
    else:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            run(mask)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = run(mask)
        mask.copy_(second)
        graph.replay()
    for x, y in zip(got, want):
        assert torch.equal(x, y)


@pytest.mark.gpu
@pytest.mark.parametrize("B,H,L,D,tangents,made", [(1, 7, 170, 32, False, False), (4, 1, 370, 64, False, False), (6, 6, 450, 64, True, True), (1, 1, 2600, 32, False, True)])
def test_bitmaps_are_made_where_they_pay(B, H, L, D, tangents, made):
    """fp32: one allocation more than a call without a mask has, or none."""
    g = torch.Generator().manual_seed(L)
    ts = [torch.randn(B, H, L, D, generator=g).to(DEV) for _ in range(6)]
    window = _mask("window", 1, 1, L, g).to(DEV).expand(B, H, L, L)

    def allocations(m):
        call = lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=m) if tangents else ja.attention(*x, attn_mask=m)  # noqa: E731
        for _ in range(2):  # the first verifies the mask
            before = torch.cuda.memory_stats()["allocation.all.allocated"]
            with torch.no_grad():
                torch.func.jvp(call, tuple(ts[:3]), tuple(ts[3:])) if tangents else call(*ts[:3])
        return torch.cuda.memory_stats()["allocation.all.allocated"] - before

    prev = ja.set_fp32_precision("tf32")
    try:
        assert allocations(window) - allocations(None) == made
    finally:
        ja.set_fp32_precision(prev)


@pytest.mark.gpu
@pytest.mark.parametrize("L", [400, 450, 500, 600])
def test_a_captured_backward_leaves_no_bitmaps_to_others(L):
    """fp32, forwards that are too short to make bitmaps: a backward of the same graph runs between another's capture and its replay."""
    g = torch.Generator().manual_seed(L)
    q, k, v, go = (torch.randn(1, 2, L, 64, generator=g).to(DEV) for _ in range(4))
    m = _mask("window", 1, 1, L, g).to(DEV)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        a = [x.requires_grad_() for x in (q, k, v)]
        want = torch.autograd.grad(ja.attention(*a, attn_mask=m), a, go)
        o = ja.attention(*a, attn_mask=m)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            captured = torch.autograd.grad(o, a, go, retain_graph=True)
        got = torch.autograd.grad(o, a, go, retain_graph=True)
        graph.replay()
    torch.cuda.synchronize()
    for x, y, z in zip(got, captured, want):
        assert torch.equal(x, z) and torch.equal(y, z)
