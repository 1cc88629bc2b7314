"""CPU tests of the native call layer (csrc/native.cpp): what the existing wiring tests do not reach.  Launches go to
the float64 stand-ins of tests/_oracle_launchers.py."""
import ctypes

import pytest
import torch
import torch.autograd.forward_ad as fwAD

import jvp_flash_attention_b200.jvp_attention as ja
from jvp_flash_attention_b200 import _lib, build
from oracle import jvp_attention_oracle as orc
from tests import _oracle_launchers as stand_in
from tests.test_autograd_wiring import _inputs, cpu_kernels  # noqa: F401


def test_a_released_graph_refuses_a_second_backward(cpu_kernels):  # noqa: F811
    q, k, v, tq, tk, tv, w, _ = _inputs(11)
    q.requires_grad_()
    o, to = torch.func.jvp(ja.JVPAttn.fwd_dual, (q, k, v), (tq, tk, tv))
    torch.autograd.grad((o * w).sum() + (to * w).sum(), q)
    with pytest.raises(RuntimeError, match="second time"):
        torch.autograd.grad((o * w).sum(), q)


@pytest.mark.parametrize("given", ["q", "kv"])
@pytest.mark.parametrize("route", ["func_jvp", "fwad"])
def test_missing_tangents_count_as_zero(cpu_kernels, given, route):  # noqa: F811
    q, k, v, tq, tk, tv, _, w = _inputs(12)
    z = torch.zeros_like(q)
    t = [tq if given == "q" else z, tk if given == "kv" else z, tv if given == "kv" else z]
    a = [x.clone().requires_grad_() for x in (q, k, v)]
    if route == "fwad":
        with fwAD.dual_level():
            d = [fwAD.make_dual(x, y) if y is not z else x for x, y in zip(a, t)]
            o, to = fwAD.unpack_dual(ja.JVPAttn.fwd_dual(*d))
    elif given == "q":
        o, to = torch.func.jvp(lambda x: ja.JVPAttn.fwd_dual(x, a[1], a[2]), (a[0],), (tq,))
    else:
        o, to = torch.func.jvp(lambda x, y: ja.JVPAttn.fwd_dual(a[0], x, y), (a[1], a[2]), (tk, tv))
    g = torch.autograd.grad((to * w).sum(), a)
    ro, rto, *rg = orc.grads_through_both(q, k, v, *t, None, w)
    assert orc.max_abs_err(o, ro) < 1e-10 and orc.max_abs_err(to, rto) < 1e-10
    for x, y in zip(g, rg):
        assert orc.max_abs_err(x, y) < 1e-9


def test_a_mask_is_verified_once_inside_func_jvp(cpu_kernels, monkeypatch):  # noqa: F811
    """The mask that a function under torch.func.jvp closes over is the caller's own tensor: its memo entry holds."""
    q, k, v, tq, tk, tv, _, _ = _inputs(13)
    mask = torch.rand(1, 2, 32, 32, generator=torch.Generator().manual_seed(1)) > 0.4
    mask[..., 0] = True
    calls = []
    monkeypatch.setattr(_lib, "mask_tiles", lambda *a: (calls.append(1), stand_in.mask_tiles(*a))[1])
    for _ in range(3):
        o, to = torch.func.jvp(lambda x, y, z: ja.JVPAttn.fwd_dual(x, y, z, attn_mask=mask), (q, k, v), (tq, tk, tv))
    ro, rto = orc.sdpa_jvp(q, k, v, tq, tk, tv, attn_mask=mask)
    assert len(calls) == 1 and orc.max_abs_err(o, ro) < 1e-10 and orc.max_abs_err(to, rto) < 1e-10


def test_nested_transforms_take_the_general_route(cpu_kernels):  # noqa: F811
    q, k, v, tq, tk, tv, w, _ = _inputs(14)
    g = torch.func.grad(lambda x: (ja.attention(x, k, v) * w).sum())(q)
    _, _, rdq, _, _ = orc.grads_through_both(q, k, v, tq, tk, tv, w, None)
    assert orc.max_abs_err(g, rdq) < 1e-9


def test_a_remembered_mask_does_not_let_host_tensors_past_the_checks(cpu_kernels, monkeypatch):  # noqa: F811
    q, k, v, *_ = _inputs(15)
    mask = torch.randn(1, 2, 32, 32, dtype=torch.float64)
    ja.attention(q, k, v, attn_mask=mask)
    assert id(mask) in ja._MASK_MEMO

    def require_cuda(*ts):
        raise RuntimeError("runs only on CUDA tensors")

    monkeypatch.setattr(ja, "_require_cuda", require_cuda)
    with pytest.raises(RuntimeError, match="runs only on CUDA tensors"):
        ja.attention(q, k, v, attn_mask=mask)


@pytest.mark.parametrize("kind", ["bias", "bool", "transposed"])
def test_a_mask_whose_data_is_replaced_is_another_mask(cpu_kernels, kind):  # noqa: F811
    """An assignment to ``.data`` leaves object and version counter as they are."""
    q, k, v, *_ = _inputs(17)
    g = torch.Generator().manual_seed(17)
    masks = [torch.randn(1, 2, 32, 32, generator=g, dtype=torch.float64) for _ in range(2)]
    if kind == "bool":
        masks = [(m > 0) | torch.eye(32, dtype=torch.bool) for m in masks]
    mask = masks[0].clone()
    ja.attention(q, k, v, attn_mask=mask)
    mask.data = mask.data.transpose(2, 3) if kind == "transposed" else masks[1]
    got = ja.attention(q, k, v, attn_mask=mask)
    assert torch.equal(got, ja.attention(q, k, v, attn_mask=mask.clone()))


@pytest.mark.parametrize("call", [ja.attention, ja.JVPAttn.fwd_dual])
@pytest.mark.parametrize("route", ["func_jvp", "fwad"])
def test_a_tangent_of_the_mask_alone_is_refused(cpu_kernels, call, route):  # noqa: F811
    """There is no derivative with respect to a bias: a call that is differentiated along the bias alone says so, and does
    not answer with a tangent of zero."""
    q, k, v, *_ = _inputs(18)
    g = torch.Generator().manual_seed(18)
    mask, t = (torch.randn(1, 2, 32, 32, generator=g, dtype=torch.float64) for _ in range(2))
    with pytest.raises(RuntimeError, match="needs tangents at forward time"):
        if route == "fwad":
            with fwAD.dual_level():
                call(q, k, v, attn_mask=fwAD.make_dual(mask, t))
        else:
            torch.func.jvp(lambda m: call(q, k, v, attn_mask=m), (mask,), (t,))


@pytest.mark.parametrize("leaf", ["mask", "mask and q"])
@pytest.mark.parametrize("route", ["attention", "fwad", "func_jvp"])
def test_a_mask_that_requires_a_gradient_is_part_of_the_graph(cpu_kernels, leaf, route):  # noqa: F811
    """A learned bias gets no gradient, but a backward from a call that has one works, whether q needs one or not."""
    q, k, v, tq, tk, tv, w, _ = _inputs(19)
    mask = torch.randn(1, 2, 32, 32, dtype=torch.float64, requires_grad=True)
    q.requires_grad_("q" in leaf)
    if route == "attention":
        o, to = ja.attention(q, k, v, attn_mask=mask), None
    elif route == "fwad":
        with fwAD.dual_level():
            o, to = fwAD.unpack_dual(ja.JVPAttn.fwd_dual(*map(fwAD.make_dual, (q, k, v), (tq, tk, tv)), attn_mask=mask))
    else:
        o, to = torch.func.jvp(lambda *x: ja.JVPAttn.fwd_dual(*x, attn_mask=mask), (q, k, v), (tq, tk, tv))
    assert o.requires_grad and (to is None or to.requires_grad == q.requires_grad)
    (o * w).sum().backward(retain_graph=True)
    ro, rto, rdq, _, _ = orc.grads_through_both(q, k, v, tq, tk, tv, w, None, attn_mask=mask.detach())
    assert mask.grad is None and orc.max_abs_err(o, ro) < 1e-10
    if "q" in leaf:
        assert orc.max_abs_err(q.grad, rdq) < 1e-9
        if to is not None:
            (to * w).sum().backward()
    else:
        assert q.grad is None


def _strided(x):  # the same values, not row-major
    return x.transpose(1, 2).contiguous().transpose(1, 2)


@pytest.mark.parametrize("which", ["all", "o", "to", "lse", "mu", "inputs"])
def test_hooks_on_saved_tensors_that_change_the_layout(cpu_kernels, which):  # noqa: F811
    """q, k, v and their tangents may come back in any layout; what the forward allocated is refused unless row-major."""
    q, k, v, tq, tk, tv, w1, w2 = _inputs(20)
    a = [x.clone().requires_grad_() for x in (q, k, v)]
    packed = []

    def pack(x):
        packed.append(x.detach().clone())
        return len(packed) - 1, x

    def unpack(handle):
        n, x = handle
        own = {k_: any(torch.equal(packed[n], y) for y in ys) for k_, ys in outputs.items() if ys and ys[0].shape == x.shape}
        name = next((k_ for k_, same in own.items() if same), "inputs" if x.dim() == 4 else None)
        if name is None:  # lse and mu: told apart by what is known of lse
            name = "lse" if n == rows[0] else "mu"
        return _strided(x) if which in ("all", name) else x

    outputs = {"o": [], "to": []}
    with torch.autograd.graph.saved_tensors_hooks(pack, unpack):
        o, to = torch.func.jvp(ja.JVPAttn.fwd_dual, tuple(a), (tq, tk, tv))
    outputs["o"].append(o.detach()), outputs["to"].append(to.detach())
    lse = torch.logsumexp(q @ k.transpose(-1, -2) * 32**-0.5, -1) / 0.6931471805599453
    rows = [n for n, x in enumerate(packed) if x.dim() == 3 and torch.allclose(x, lse)]
    assert len(rows) == 1
    if which == "inputs":
        g = torch.autograd.grad((o * w1).sum() + (to * w2).sum(), a)
        for x, y in zip(g, orc.grads_through_both(q, k, v, tq, tk, tv, w1, w2)[2:]):
            assert orc.max_abs_err(x, y) < 1e-9
    else:
        with pytest.raises(ValueError, match="to be contiguous"):
            torch.autograd.grad((o * w1).sum() + (to * w2).sum(), a)


@pytest.fixture()
def unwrapping_cpu_kernels(cpu_kernels, monkeypatch):  # noqa: F811
    """The stand-ins on plain tensors, as the package's own launch helpers run."""
    def plain(launch):
        def run(*args):
            with torch.no_grad(), _lib.native().NoFunctorch():
                return launch(*(ja._unwrap(x).detach() if isinstance(x, torch.Tensor) else x for x in args))
        return run

    monkeypatch.setattr(ja, "_launch_fwd", plain(stand_in.launch_fwd))
    monkeypatch.setattr(ja, "_launch_bwd", plain(stand_in.launch_bwd))


@pytest.mark.parametrize("outputs", ["o", "both"])
def test_a_functorch_transform_of_the_cotangent(unwrapping_cpu_kernels, outputs):
    """d/dw <dq(w), u> of a graph built outside the transform is the tangent of O along u; vmap over w is refused."""
    q, k, v, tq, tk, tv, w, u = _inputs(21)
    a = [x.clone().requires_grad_() for x in (q, k, v)]
    if outputs == "o":
        o, to = ja.attention(*a), None
    else:
        o, to = torch.func.jvp(ja.JVPAttn.fwd_dual, tuple(a), (tq, tk, tv))

    def vjp(x):
        outs, cots = ((o,), (x,)) if to is None else ((o, to), (x, w))
        return torch.autograd.grad(outs, a[0], cots, retain_graph=True, create_graph=True)[0]

    got = torch.func.grad(lambda x: (vjp(x) * u).sum())(w)
    z = torch.zeros_like(q)
    assert orc.max_abs_err(got, orc.sdpa_jvp(q, k, v, u, z, z)[1]) < 1e-9
    if to is None:
        with pytest.raises(RuntimeError, match="vmap"):
            torch.func.vmap(vjp)(torch.stack([w, u]))


def test_another_torch_has_the_call_layer_built_again(monkeypatch, tmp_path):
    monkeypatch.setattr(build, "NATIVE", tmp_path / "_native.so")
    monkeypatch.setattr(build, "NATIVE_STAMP", tmp_path / "native.stamp")
    assert build._native_stale()
    build.NATIVE.touch()
    assert build._native_stale()  # built with nobody knows what
    build.NATIVE_STAMP.write_text(build._native_with())
    assert not build._native_stale()
    monkeypatch.setattr(torch, "__version__", "0.0")
    assert build._native_stale()


def test_misaligned_forms_of_a_mask_are_refused_by_the_library():
    """Checked on the host before anything is launched: the kernels read the bits 8 bytes at a time."""
    lib = _lib.load()
    x = 1 << 20  # an address that is never followed: the kind of the mask is refused as well
    refused = 99

    def fwd(**fields):
        a = _lib.FwdArgs(struct_size=ctypes.sizeof(_lib.FwdArgs), dtype=_lib.BF16, B=1, H=1, L=64, D=64, sm_scale=0.125, q=x, k=x, v=x, o=x,
                         lse=x, **fields)
        a.mask.kind = refused
        return lib.jvpfa_fwd(ctypes.byref(a), None)

    def bwd(**fields):
        a = _lib.BwdArgs(struct_size=ctypes.sizeof(_lib.BwdArgs), dtype=_lib.BF16, B=1, H=1, L=64, D=64, sm_scale=0.125, q=x, k=x, v=x, go=x,
                         lse=x, delta=x, dq=x, dk=x, dv=x, **fields)
        a.mask.kind = refused
        return lib.jvpfa_bwd(ctypes.byref(a), None)

    def tiles(**fields):
        a = _lib.MaskTilesArgs(struct_size=ctypes.sizeof(_lib.MaskTilesArgs), n_b=1, n_h=1, n_rows=64, L=64, **fields)
        a.mask.kind = refused
        return lib.jvpfa_mask_tiles(ctypes.byref(a), None)

    misaligned = -8
    for call, fields in ((fwd, ("mask_bits", "mask_tile_live")), (bwd, ("mask_bits", "mask_bits_t", "mask_tile_live", "mask_tile_live_t")),
                         (tiles, ("bits", "bits_t", "tile_live_t"))):
        for field in fields:
            extra = {"tile_live": x} if call is tiles else {}
            assert call(**extra, **{field: x + 4}) == misaligned, (call.__name__, field)
