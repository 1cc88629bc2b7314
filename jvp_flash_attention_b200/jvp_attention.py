"""Drop-in Python API of ``jvp_flash_attention.jvp_attention`` on hand-written sm_100a kernels.

Public names and signatures mirror upstream (jvp_flash_attention/jvp_attention.py:48-51,
2236-2981): ``MASK_CONST``, ``MIN_SEQUENCE_LENGTH``, ``JVPAttn`` (a ``torch.autograd.Function``
with ``forward / setup_context / jvp / backward`` plus the ``fwd`` and ``fwd_dual``
conveniences) and ``attention = JVPAttn.fwd``.  All arithmetic happens in ``libjvpfa.so``
(see ``include/jvpfa.h``); this module only validates, classifies the mask, allocates outputs
and wires autograd.

Behaviour that goes beyond upstream, on purpose:

* the tangent output is differentiable: ``jvp`` returns it through ``_TangentBridge`` whose
  backward is the gradient of ``<gtO, tO>`` (upstream returns a constant, jvp_attention.py:2828);
* ``backward`` is itself differentiable once (Hessian-vector products) through ``_AttnBwd``;
* masks may be any shape broadcastable to (Z, H, N, N); a boolean (Z|1, 1, 1, N) prefix mask is
  recognised as key padding and its fully padded key tiles are skipped;
* a float mask is an additive bias with SDPA semantics, ``softmax(scale*QK^T + bias)``
  (upstream scales the bias as well and ignores it in backward, jvp_attention.py:247-251,
  1519-1522), and a float mask without ``MASK_CONST`` entries is accepted (upstream raises
  ``UserWarning``, jvp_attention.py:2459-2462).

Calls of one shape give the same bits from run to run, but for dQ of 16-bit calls at head dimension 64 (see
``_lib.bwd``, ``dq_accum``).  16-bit calls at head dimension 64 and below cut their tiles among the SMs by the number
of heads, so a head's last bits may differ between calls that compute it beside different numbers of others.
"""
from __future__ import annotations

import copy
import inspect
import sys
import types
import weakref
from typing import Any, Literal, NamedTuple

import torch
import torch.autograd.forward_ad as fwAD
from torch import Tensor
from torch.autograd import Function
from torch.autograd.function import FunctionCtx, once_differentiable

from . import _lib

MASK_CONST = -100.0  # same constant as upstream (jvp_attention.py:48-50)
MIN_SEQUENCE_LENGTH = 32  # jvp_attention.py:51
# Upstream refuses sequence lengths that are odd or below 32 (its block sizes); the kernels here take any length >= 1.
# The check is kept so that the same calls fail the same way; set this to False to lift it.
STRICT_SEQUENCE_LENGTH = True

_SUPPORTED_HEAD_DIMS = (32, 64, 128)
_UPSTREAM_HEAD_DIMS = {16, 32, 64, 128, 256}

# Kernel family used by the launches of this module (see jvpfa_impl in include/jvpfa.h).
# Tests flip it to cross-check the two families against each other.
KERNEL_IMPL = _lib.IMPL_AUTO

# The backward of head-dimension-64 16-bit calls runs as one pass that sums dQ with floating-point reductions (reproducible
# to rounding) where the mask is none, causal, key padding, or, with rows of whole 16-byte pieces, boolean without dead
# tiles or (through O alone) a bias of the tensors' type.  False: always the two-launch kernels, whose results are bitwise
# reproducible from run to run, as those of all other calls are.
SINGLE_PASS_BACKWARD = True


def is_hip() -> bool:
    """Upstream's backend probe (jvp_attention.py:54-59).  This build has one target, NVIDIA sm_100a."""
    return False


def is_cuda() -> bool:
    """True when a CUDA device is present (upstream: jvp_attention.py:62-67)."""
    return torch.cuda.is_available()


def is_blackwell() -> bool:
    """True on a compute-capability-10 device, the only kind these kernels run on (upstream: jvp_attention.py:86-91)."""
    try:
        return is_cuda() and torch.cuda.get_device_capability()[0] == 10
    except Exception:  # noqa: BLE001
        return False


def supports_host_descriptor() -> bool:
    """Upstream asks this before building host-side TMA descriptors (jvp_attention.py:70-75); here every tcgen05 kernel
    takes host-encoded tensor maps, so the answer is that of is_blackwell()."""
    return is_blackwell()


def supports_tma() -> bool:
    """See supports_host_descriptor (upstream: jvp_attention.py:78-83)."""
    return is_blackwell()


def _unwrap(x):
    """Strips functorch wrappers so that ``data_ptr()`` is available (cf. jvp_attention.py:2846-2855)."""
    fc = torch._C._functorch
    while isinstance(x, Tensor) and fc.is_functorch_wrapped_tensor(x):
        x = fc.get_unwrapped(x)
    return x


def _require_cuda(*ts: Tensor) -> None:
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError(
                "jvp_flash_attention_b200 runs only on CUDA tensors of a compute-capability-10 GPU; "
                "there is no CPU or PyTorch fallback"
            )


def set_fp32_precision(mode: str) -> str:
    """How fp32 inputs are multiplied from now on; returns the previous mode.

    ``"3xtf32"`` (default): every product as three TF32 MMAs on a hi/lo split, about 1e-6 relative error.
    ``"tf32"``: one TF32 MMA per product, about 5e-4 -- what upstream's fp32 path computes (its ``tl.dot`` calls
    run on TF32 tensor cores, jvp_attention.py:233-236; its fp32 tolerance is 2.35e-2), 1.7 to 2.2 times
    as fast (B2 H8 L2048 D64: O 479 -> 241 us, its backward 1885 -> 988, fwd_dual 1280 -> 605).
    A call's backward (and double backward) runs at the precision its forward ran at: the mode is recorded with the
    call, so changing it in between affects later forwards only."""
    if mode not in ("3xtf32", "tf32"):
        raise ValueError("fp32 precision is '3xtf32' or 'tf32'")
    prev, _lib.FP32_PRECISION = _lib.FP32_PRECISION, mode
    return prev


# What classify_mask found out about a mask tensor, kept while the same tensor object is passed again unmodified
# (same Python object, same version counter, which every in-place operation of torch bumps, and still the same memory and
# layout, which an assignment to `.data` changes).  A mask is typically built once and used by every layer and step; its
# verification is a pass over B*H*L*L elements and a read-back.
# What is kept: that the mask is a valid one, which tiles of a boolean mask are stepped over, and the lengths of a
# key-padding mask.  Writes that bypass torch's counter (a foreign kernel, a captured graph that is replayed after the mask
# was changed) are not seen by these; the entries themselves are read by every launch.  MASK_MEMO_ENABLED = False turns the
# memo off.
MASK_MEMO_ENABLED = True
_MASK_MEMO: dict = {}
_MASK_MEMO_MAX = 16


def _mask_state(m: Tensor) -> tuple:
    """What tells a mask tensor's present contents from those that were verified."""
    return m._version, m.data_ptr(), m.stride(), m.dtype


def _remembered_mask(attn_mask: Tensor, q_shape) -> _lib.MaskSpec | None:
    """The description classify_mask found for this very tensor, unmodified since, or None."""
    hit = _MASK_MEMO.get(id(attn_mask)) if MASK_MEMO_ENABLED else None
    if hit is not None and hit[0]() is attn_mask and hit[1] == (*q_shape[:3], True, *_mask_state(attn_mask)):
        return hit[2][0]
    return None


def classify_mask(attn_mask: Tensor | None, causal: bool, Z: int, H: int, N: int, qdtype: torch.dtype,
                  verify: bool) -> tuple[_lib.MaskSpec, int, Tensor | None]:
    """Turns the user's mask into the kernel's description.

    Returns ``(spec, MASK_TYPE, mask_tensor)`` where MASK_TYPE follows upstream's numbering
    (0 none, 1 boolean, 2 additive; jvp_attention.py:2430-2446).  Pure host logic apart from
    the optional verification reductions, which mirror jvp_attention.py:2438-2457.
    """
    if causal:
        return _lib.MaskSpec(_lib.MASK_CAUSAL), 0, None
    if attn_mask is None:
        return _lib.MaskSpec(_lib.MASK_NONE), 0, None
    if not MASK_MEMO_ENABLED:
        return _classify_mask_tensor(attn_mask, Z, H, N, verify)
    key = (Z, H, N, verify, *_mask_state(_unwrap(attn_mask)))
    hit = _MASK_MEMO.get(id(attn_mask))
    if hit is not None and hit[0]() is attn_mask and hit[1] == key:
        spec, mask_type = hit[2]
        return copy.copy(spec), mask_type, attn_mask  # a copy: the caller writes per-call state into the description
    spec, mask_type, _ = _classify_mask_tensor(attn_mask, Z, H, N, verify)
    if len(_MASK_MEMO) >= _MASK_MEMO_MAX:
        _MASK_MEMO.clear()
    try:
        # the entry goes when the caller's tensor object does (the description holds a view of the mask's storage and
        # must not keep it alive)
        k_id = id(attn_mask)
        _MASK_MEMO[k_id] = (weakref.ref(attn_mask, lambda _r, k_id=k_id, pop=_MASK_MEMO.pop: pop(k_id, None)), key,
                            (copy.copy(spec), mask_type))
    except TypeError:  # an object that cannot be weakly referenced: no memo
        pass
    return spec, mask_type, attn_mask


def _classify_mask_tensor(attn_mask: Tensor, Z: int, H: int, N: int, verify: bool):
    """classify_mask for a mask tensor: shape checks, key-padding recognition, verification passes."""
    assert attn_mask.dim() == 4, "The provided attention mask must have 4 dimensions (Z, H, N_CTX, N_CTX)."
    mz, mh, mi, mj = attn_mask.shape
    assert mz in (1, Z) and mh in (1, H) and mi in (1, N) and mj == N, (
        "The provided attention mask must be broadcastable to (Z, H, N_CTX, N_CTX)."
    )
    assert attn_mask.dtype == torch.bool or attn_mask.dtype.is_floating_point, (
        "The attention mask must be of the dtype bool or a floating-point dtype."
    )
    m = _unwrap(attn_mask).detach()  # the description keeps the storage, not the caller's tensor object (see the memo)

    def bstrides(t: Tensor) -> tuple[int, int, int, int]:
        return tuple(0 if t.shape[d] == 1 else t.stride(d) for d in range(4))

    if m.dtype == torch.bool:
        if mh == 1 and mi == 1:
            # Candidate key-padding mask: valid keys form a prefix of each row.  Lengths, the prefix test and
            # upstream's "no head all False" check come back in one read-back.
            rows = m.reshape(mz, N)
            lens = rows.sum(dim=-1, dtype=torch.int32)
            prefix = torch.arange(N, device=m.device).unsqueeze(0) < lens.unsqueeze(1)
            is_prefix, *host_lens = torch.cat(((prefix == rows).all().to(torch.int32).view(1), lens)).tolist()
            if is_prefix:
                if verify:
                    assert min(host_lens) > 0, "The attention mask cannot be all False for any head."
                kv_len = lens.expand(Z).contiguous() if mz == 1 else lens.contiguous()
                spec = _lib.MaskSpec(_lib.MASK_KVLEN, kv_len)
                spec.kv_len_host = host_lens * Z if mz == 1 else host_lens
                return spec, 1, attn_mask
        m8 = m.view(torch.uint8) if m.is_contiguous() or m.stride(-1) == 1 else m.contiguous().view(torch.uint8)
        spec = _lib.MaskSpec(_lib.MASK_BOOL, m8, bstrides(m8))
        every_head_live = True
        if verify:
            # One pass answers upstream's check and says which 128 x 64 tiles have a True at all; forward and
            # backward step over the others.  (Without verification the mask is not looked at beforehand, so
            # there is no block skipping either: whether it would pay is known only from the pass's counts.)
            spec.tile_live, head_live, spec.tile_live_t = _lib.mask_tiles(spec, N)
            *heads, n_live = head_live.tolist()  # the one read-back
            every_head_live = all(heads)
            n_entries = spec.tile_live.numel() // (((N + 63) // 64 + 63) // 64)
            spec.tile_dead = 1.0 - n_live / (n_entries * ((N + 63) // 64))
            if n_live > 0.85 * n_entries * ((N + 63) // 64):
                spec.tile_live = spec.tile_live_t = None  # (nearly) every tile is live: the plain loops are quicker
        assert every_head_live, "The attention mask cannot be all False for any head."
        return spec, 1, attn_mask

    if m.dtype not in _lib.DTYPE_ENUM:
        m = m.to(torch.float32)
    spec = _lib.MaskSpec(_lib.MASK_BIAS, m, bstrides(m), _lib.DTYPE_ENUM[m.dtype])
    if verify:
        # one pass and one read-back for upstream's isinf / isnan / "all MASK_CONST" sweeps (jvp_attention.py:2447-2457)
        every_head_live, has_inf, has_nan = _lib.mask_check(spec, m.shape)
        assert not has_inf, "The attention mask cannot contain -inf or inf."
        assert not has_nan, "The attention mask cannot contain NaNs."
        assert every_head_live, f"The attention mask cannot be all {MASK_CONST} (the masking constant) for any head."
    return spec, 2, attn_mask


def _in_place_layout(ts):
    """``(tensors, in_stride)`` for the kernels: the tensors as they are together with their common (batch, head,
    row) strides when they share a layout the kernels can read in place (e.g. the (B,H,L,D) view of a
    (B,L,H,D) tensor; upstream always copies, jvp_attention.py:2733-2734), else contiguous copies and None."""
    try:
        return ts, _lib.common_strides(*ts)
    except ValueError:
        return [None if t is None else t.contiguous() for t in ts], None


def _without_old_tiles(spec: _lib.MaskSpec, q: Tensor) -> _lib.MaskSpec:
    """fp32 launches visit every tile here: the bitmaps are those of the mask's verification, and what these kernels read
    are its present entries (the native layer makes bitmaps of these for them)."""
    if spec.tile_live is None or q.dtype != torch.float32:
        return spec
    spec = copy.copy(spec)
    spec.tile_live = spec.tile_live_t = None
    return spec


def _launch_fwd(q, k, v, tq, tk, tv, spec: _lib.MaskSpec, sm_scale: float):
    """Allocates outputs and runs the fused forward.  Returns (o, to | None, lse, mu | None)."""
    spec = _without_old_tiles(spec, q)
    ins, st = _in_place_layout([_unwrap(x) for x in (q, k, v, tq, tk, tv)])
    Z, H, N, _ = ins[0].shape
    o = torch.empty(ins[0].shape, device=ins[0].device, dtype=ins[0].dtype)
    lse = torch.empty((Z, H, N), device=o.device, dtype=torch.float32)
    dual = ins[3] is not None
    to = torch.empty_like(o) if dual else None
    mu = torch.empty_like(lse) if dual else None
    _lib.fwd(*ins, o, to, lse, mu, spec, sm_scale, KERNEL_IMPL, in_stride=st)
    return o, to, lse, mu


def _launch_bwd(q, k, v, tq, tk, tv, o, to, lse, mu, go, gto, spec: _lib.MaskSpec, sm_scale: float):
    """Runs preprocess + backward for cotangents ``go`` (of O) and/or ``gto`` (of tO)."""
    spec = _without_old_tiles(spec, q)
    q, k, v, tq, tk, tv, o, to, lse, mu, go, gto = (
        _unwrap(x) for x in (q, k, v, tq, tk, tv, o, to, lse, mu, go, gto)
    )
    if go is not None and not go.is_contiguous():
        go = go.contiguous()
    if gto is not None and not gto.is_contiguous():
        gto = gto.contiguous()
    if gto is None:
        tq = tk = tv = to = mu = None
    ins, st = _in_place_layout([q, k, v, tq, tk, tv])
    Z, H, N, _ = q.shape
    stats = torch.empty((3, Z, H, N), device=q.device, dtype=torch.float32)
    delta, eps, cterm = stats[0], stats[1], stats[2]
    _lib.bwd_preprocess(o, to, go, gto, mu, delta, eps, cterm, spec.fp32_mode)
    dq, dk, dv = (torch.empty(q.shape, device=q.device, dtype=q.dtype) for _ in range(3))
    # fp32 scratch for dQ: with it the library forms every score tile once (head dimension 64, 16-bit, index masks or a
    # boolean mask without dead tiles)
    acc = None
    dense_bool = spec.kind == _lib.MASK_BOOL and spec.tile_live is None and spec.tile_live_t is None  # no tiles to step over
    bias_o = spec.kind == _lib.MASK_BIAS and gto is None and spec.bias_dtype == _lib.DTYPE_ENUM.get(q.dtype)  # through O alone
    if SINGLE_PASS_BACKWARD and q.shape[-1] == 64 and q.dtype != torch.float32 and (
            spec.kind in _lib.INDEX_MASKS or dense_bool or bias_o):
        acc = torch.empty(q.shape, device=q.device, dtype=torch.float32)
    _lib.bwd(*ins, go, gto, lse, mu, delta, eps, cterm, dq, dk, dv, spec, sm_scale, KERNEL_IMPL, in_stride=st, dq_accum=acc)
    return dq, dk, dv


def _check_bwd_layout(q, k, v, o):
    """Upstream refuses non-contiguous saved tensors in backward (jvp_attention.py:2858-2877).  Here q, k, v may
    keep the strided layout they had in forward (they are read in place or copied by _launch_bwd); the
    output, which this library allocated itself, must still be row-major."""
    if not o.is_contiguous():
        raise ValueError(f"JVPAttn expected o to be contiguous; got o.is_contiguous()={o.is_contiguous()}")


class _AttnBwd(Function):
    """(dq, dk, dv) = d<do, O>/d(q, k, v), as a node that can be differentiated once more.

    Its own backward uses the identity (u = incoming grads of dq, dk, dv)
        d<(dq,dk,dv), u>/d(q,k,v) = d<tO(q,k,v; u), do>/d(q,k,v),   d<...>/d(do) = tO(q,k,v; u)
    so a Hessian-vector product costs one fused primal+tangent forward with tangents u and one
    backward through the tangent output; no further kernels exist for it.
    """

    @staticmethod
    def forward(q, k, v, o, lse, do, spec, sm_scale):
        return _launch_bwd(q, k, v, None, None, None, o, None, lse, None, do, None, spec, sm_scale)

    @staticmethod
    def setup_context(ctx, inputs, outputs):
        q, k, v, o, lse, do, spec, sm_scale = inputs
        ctx.save_for_backward(q, k, v, o, lse, do)
        ctx.spec, ctx.sm_scale = spec, sm_scale

    @staticmethod
    @once_differentiable
    def backward(ctx, uq, uk, uv):
        q, k, v, o, lse, do = ctx.saved_tensors
        us = [torch.zeros_like(q) if u is None else u.contiguous() for u in (uq, uk, uv)]
        o2, to_u, lse2, mu_u = _launch_fwd(q, k, v, us[0], us[1], us[2], ctx.spec, ctx.sm_scale)
        need_qkv = any(ctx.needs_input_grad[:3])
        hq = hk = hv = None
        if need_qkv:
            hq, hk, hv = _launch_bwd(q, k, v, us[0], us[1], us[2], o2, to_u, lse2, mu_u, None, do, ctx.spec,
                                     ctx.sm_scale)
        gdo = to_u if ctx.needs_input_grad[5] else None
        return hq, hk, hv, None, None, gdo, None, None


class _TangentBridge(Function):
    """Hands the tangent output computed by the fused forward to autograd with a real gradient.

    forward returns the precomputed tO; backward is the gradient of <gtO, tO> with respect to the
    primals (the tangent-path backward kernel) and, when asked for, with respect to the tangents
    (ordinary attention backward with do = gtO).
    """

    @staticmethod
    def forward(q, k, v, tq, tk, tv, to, o, lse, mu, spec, sm_scale, relay=None, link=None):
        return to.detach()

    @staticmethod
    def setup_context(ctx, inputs, output):
        q, k, v, tq, tk, tv, to, o, lse, mu, spec, sm_scale, relay, link = inputs
        ctx.save_for_backward(q, k, v, tq, tk, tv, to, o, lse, mu)
        ctx.spec, ctx.sm_scale, ctx.link = spec, sm_scale, link

    @staticmethod
    @once_differentiable
    def backward(ctx, gto):
        q, k, v, tq, tk, tv, to, o, lse, mu = ctx.saved_tensors
        _check_bwd_layout(q, k, v, o)
        gq = gk = gv = gtq = gtk = gtv = grelay = None
        if ctx.link is not None and ctx.needs_input_grad[12]:
            # The node of the primal output runs after this one (it produced `relay`) and takes the cotangent of tO
            # along with its own: one preprocess and one backward launch for a loss on both outputs.
            ctx.link.value = (gto, tq, tk, tv, to, mu)
            grelay = _zero_scalar(gto.device)
        elif any(ctx.needs_input_grad[:3]):
            gq, gk, gv = _launch_bwd(q, k, v, tq, tk, tv, o, to, lse, mu, None, gto, ctx.spec, ctx.sm_scale)
        if any(ctx.needs_input_grad[3:6]):
            gtq, gtk, gtv = _launch_bwd(q, k, v, None, None, None, o, None, lse, None, gto, None, ctx.spec,
                                        ctx.sm_scale)
        return gq, gk, gv, gtq, gtk, gtv, None, None, None, None, None, None, grelay, None


class _BwdThroughTangent(Function):
    """(dq, dk, dv) of <gtO, tO> while a graph is being recorded for a second differentiation: like
    ``_TangentBridge.backward``, this part cannot be differentiated again, and says so when asked."""

    @staticmethod
    def forward(q, k, v, tq, tk, tv, o, to, lse, mu, gto, spec, sm_scale):
        return _launch_bwd(q, k, v, tq, tk, tv, o, to, lse, mu, None, gto, spec, sm_scale)

    @staticmethod
    def setup_context(ctx, inputs, outputs):
        pass

    @staticmethod
    def backward(ctx, *grads):
        raise RuntimeError("the gradient through the tangent output of JVPAttn cannot be differentiated a second time")


_ZERO_SCALARS: dict = {}


def _zero_scalar(device) -> Tensor:
    """A fresh tensor object over one cached fp32 zero per device (no kernel launch)."""
    z = _ZERO_SCALARS.get(device)
    if z is None:
        z = _ZERO_SCALARS[device] = torch.zeros((), dtype=torch.float32, device=device)
    return z.detach()


def _check_args(q, k, v, q_t, k_t, v_t, attn_mask, causal):
    """Upstream's argument checks, with its wording (jvp_attention.py:2356-2400)."""
    Z, H, N_CTX, HEAD_DIM_Q = q.shape
    HEAD_DIM_K = k.shape[-1]
    HEAD_DIM_V = v.shape[-1]
    assert HEAD_DIM_Q == HEAD_DIM_K and HEAD_DIM_K == HEAD_DIM_V, (
        "JVP attention requires HEAD_DIM_Q == HEAD_DIM_K == HEAD_DIM_V"
        f" but got HEAD_DIM_Q={HEAD_DIM_Q}, HEAD_DIM_K={HEAD_DIM_K}, HEAD_DIM_V={HEAD_DIM_V}"
    )
    assert HEAD_DIM_K in _UPSTREAM_HEAD_DIMS, (
        "JVP attention only supports HEAD_DIM_K in {16, 32, 64, 128, 256},"
        f" but got HEAD_DIM_K={HEAD_DIM_K}"
    )
    if HEAD_DIM_K not in _SUPPORTED_HEAD_DIMS:
        raise NotImplementedError(
            f"HEAD_DIM_K={HEAD_DIM_K} has no sm_100a kernel in this build (supported: {_SUPPORTED_HEAD_DIMS})"
        )
    assert not STRICT_SEQUENCE_LENGTH or (N_CTX % 2 == 0 and N_CTX >= MIN_SEQUENCE_LENGTH), (
        "JVP attention requires N_CTX to be a multiple of 2 and >= 32,"
        f" but got N_CTX={N_CTX}"
    )
    assert k.shape == q.shape and v.shape == q.shape, "q, k, v must share one (Z, H, N_CTX, HEAD_DIM) shape"
    if causal and attn_mask is not None:
        raise ValueError("Causal attention does not support an attention mask.")
    if q.dtype not in _lib.DTYPE_ENUM:
        raise TypeError(f"unsupported dtype {q.dtype}; expected bfloat16, float16 or float32")
    _require_cuda(q, k, v, q_t, k_t, v_t, attn_mask)


def _forward_impl(q, k, v, q_t, k_t, v_t, attn_mask, dropout_p, causal, sm_scale, verify_attn_mask):
    """Checks, mask classification and the launch of the fused forward, shared by JVPAttn.forward and its lean twin
    (JVPAttn's nested types are looked up when it is called).
    Returns (o, o_t, M, mu, mask_spec, MASK_TYPE, mask_tensor, sm_scale, HEAD_DIM_K, grid)."""
    if dropout_p != 0.0:
        raise NotImplementedError("Dropout is not currently supported in JVP attention.")
    _check_args(q, k, v, q_t, k_t, v_t, attn_mask, causal)
    Z, H, N_CTX, HEAD_DIM_K = q.shape

    if sm_scale is None:
        sm_scale = HEAD_DIM_K**-0.5

    tangents = [q_t, k_t, v_t]
    if any(t is not None for t in tangents):
        tangents = [torch.zeros_like(q) if t is None else t for t in tangents]
    qc, kc, vc = q, k, v  # strided views are read in place where the kernels can (_launch_fwd)
    tq, tk, tv = (None if t is None else t.to(q.dtype) for t in tangents)

    spec, MASK_TYPE, mask_tensor = classify_mask(attn_mask, causal, Z, H, N_CTX, q.dtype, verify_attn_mask)
    # the backward of this call recomputes the scores at the precision they had here, whatever the process-wide
    # setting is by then
    spec.fp32_mode = _lib.FP32_PRECISION
    o, o_t, M, mu = _launch_fwd(qc, kc, vc, tq, tk, tv, spec, sm_scale)
    grid = JVPAttn.Grid((N_CTX + 63) // 64, Z * H, 1)
    return o, o_t, M, mu, spec, MASK_TYPE, mask_tensor, sm_scale, HEAD_DIM_K, grid



class JVPAttn(Function):
    """JVP (Jacobian-Vector Product) for Attention Mechanism (same interface as upstream's JVPAttn)."""

    class Grid(NamedTuple):
        M_BLOCKS: int
        Z_H: int
        ONE: Literal[1]

    class FnCtx(FunctionCtx):
        sm_scale: float
        HEAD_DIM_K: int
        causal: bool
        grid: "JVPAttn.Grid"
        mask_tensor: Tensor
        MASK_TYPE: int
        dropout_p: float
        philox_seed: int
        ENABLE_DROPOUT: bool

    class FwdOutCtxContrib(NamedTuple):
        """Second element of the forward output; the first ten fields are upstream's (jvp_attention.py:2259-2271)."""

        o_t: Tensor | None
        M: Tensor
        grid: "JVPAttn.Grid"
        HEAD_DIM_K: int
        sm_scale: float
        mask_tensor: Tensor | None
        MASK_TYPE: int
        dropout_p: float
        philox_seed: int
        ENABLE_DROPOUT: bool
        mu: Tensor | None = None  # rowsum(P * tS), needed to differentiate through o_t
        mask_spec: Any = None     # kernel-side mask description

    class FwdOut(NamedTuple):
        o: Tensor
        ctx: "JVPAttn.FwdOutCtxContrib"

    class JVPOut(NamedTuple):
        o: Tensor
        ctx: None

    class BwdOut(NamedTuple):
        q: Tensor
        k: Tensor
        v: Tensor
        q_t: None
        k_t: None
        v_t: None
        attn_mask: None
        dropout_p: None
        causal: None
        sm_scale: None
        warp_specialize: None
        USE_TMA: None
        verify_attn_mask: None

    class Strides(NamedTuple):
        z: int
        h: int
        n_ctx: int
        head_dim: int

    @staticmethod
    def forward(
        q: Tensor,
        k: Tensor,
        v: Tensor,
        q_t: Tensor | None,
        k_t: Tensor | None,
        v_t: Tensor | None,
        attn_mask: Tensor | None = None,
        dropout_p: float = 0.0,
        causal: bool = False,
        sm_scale: float | None = None,
        warp_specialize: bool = True,
        USE_TMA: bool = True,
        verify_attn_mask: bool = True,
    ) -> "JVPAttn.FwdOut":
        """Fused primal (+ tangent) forward; argument meaning as upstream (jvp_attention.py:2311-2355).

        ``warp_specialize`` and ``USE_TMA`` are accepted for signature compatibility and ignored:
        there is one sm_100a code path.
        """
        o, o_t, M, mu, spec, MASK_TYPE, mask_tensor, sm_scale, HEAD_DIM_K, grid = _forward_impl(
            q, k, v, q_t, k_t, v_t, attn_mask, dropout_p, causal, sm_scale, verify_attn_mask)
        return JVPAttn.FwdOut(
            o,
            JVPAttn.FwdOutCtxContrib(o_t, M, grid, HEAD_DIM_K, sm_scale, mask_tensor, MASK_TYPE, dropout_p, 0,
                                     False, mu, spec),
        )

    @staticmethod
    def setup_context(ctx: "JVPAttn.FnCtx", inputs, outputs: "JVPAttn.FwdOut") -> None:
        (q, k, v, q_t, k_t, v_t, attn_mask, dropout_p, causal, sm_scale, warp_specialize, USE_TMA,
         *rest) = inputs
        o, c = outputs
        ctx.grid = c.grid
        ctx.save_for_forward(c.o_t, q, k, v, q_t, k_t, v_t, o, c.M, c.mu)
        ctx.save_for_backward(q, k, v, o, c.M)
        ctx.sm_scale = c.sm_scale
        ctx.HEAD_DIM_K = c.HEAD_DIM_K
        ctx.causal = causal
        ctx.mask_tensor = c.mask_tensor
        ctx.MASK_TYPE = c.MASK_TYPE
        ctx.mask_spec = c.mask_spec
        ctx.dropout_p = c.dropout_p
        ctx.philox_seed = c.philox_seed
        ctx.ENABLE_DROPOUT = c.ENABLE_DROPOUT
        ctx.set_materialize_grads(False)

    @staticmethod
    def fwd(
        q: Tensor,
        k: Tensor,
        v: Tensor,
        attn_mask: Tensor | None = None,
        dropout_p: float = 0.0,
        causal: bool = False,
        sm_scale: float | None = None,
        warp_specialize: bool = True,
        USE_TMA: bool = True,
    ) -> Tensor:
        """Primal-only attention (upstream: jvp_attention.py:2701-2752).  Returns O."""
        if dropout_p != 0.0:
            raise NotImplementedError("Dropout is not currently supported in JVP attention.")
        return _attend(q, k, v, attn_mask, causal, sm_scale, False)

    @staticmethod
    def fwd_dual(
        q: Tensor,
        k: Tensor,
        v: Tensor,
        attn_mask: Tensor | None = None,
        dropout_p: float = 0.0,
        causal: bool = False,
        sm_scale: float | None = None,
        warp_specialize: bool = True,
        USE_TMA: bool = True,
    ) -> Tensor:
        """Attention on forward-AD dual tensors (upstream: jvp_attention.py:2755-2813).

        q, k, v may be dual tensors (``fwAD.make_dual`` or inside ``torch.func.jvp``); the result
        is a dual tensor whose tangent is tO.  Tangents are unpacked here, before autograd sees
        them, and travel to the kernel as explicit arguments.
        """
        if dropout_p != 0.0:
            raise NotImplementedError("Dropout is not currently supported in JVP attention.")
        return _attend(q, k, v, attn_mask, causal, sm_scale, True)

    @staticmethod
    def jvp(ctx: "JVPAttn.FnCtx", gq: Tensor, gk: Tensor, gv: Tensor, *_) -> "JVPAttn.JVPOut":
        """Returns the tangent computed by the fused forward (upstream: jvp_attention.py:2816-2828),
        routed through ``_TangentBridge`` so that it carries a gradient."""
        return JVPAttn.JVPOut(_jvp_impl(ctx, gq, gk, gv), None)

    @staticmethod
    def backward(ctx, do, _) -> "JVPAttn.BwdOut":
        """Gradient of <do, O> w.r.t. q, k, v (upstream: jvp_attention.py:2831-2978)."""
        if do is None:
            return JVPAttn.BwdOut(*([None] * 13))
        dq, dk, dv = _backward_impl(ctx, do)
        return JVPAttn.BwdOut(dq, dk, dv, None, None, None, None, None, None, None, None, None, None)


def _jvp_impl(ctx, gq, gk, gv, relay=None, link=None):
    """The tangent output of a call whose forward has run: the kernel's tangent, behind ``_TangentBridge`` when a
    gradient of it can be asked for."""
    o_t, q, k, v, q_t, k_t, v_t, o, M, mu = ctx.saved_for_forward[:10]
    if o_t is None:
        raise RuntimeError(
            "JVPAttn.jvp needs tangents at forward time: call JVPAttn.fwd_dual (or pass q_t, k_t, v_t to apply)"
        )
    # Nobody can ask for a gradient of the tangent when no input takes part in a graph: hand the kernel's tangent
    # over as it is and skip the bridging node.  (Looked up on the unwrapped tensors: inside torch.func.jvp the
    # wrappers do not say.)
    if not any(x is not None and _unwrap(x).requires_grad for x in (q, k, v, q_t, k_t, v_t, gq, gk, gv)):
        return o_t
    tq = gq if gq is not None else (q_t if q_t is not None else torch.zeros_like(q))
    tk = gk if gk is not None else (k_t if k_t is not None else torch.zeros_like(k))
    tv = gv if gv is not None else (v_t if v_t is not None else torch.zeros_like(v))
    return _TangentBridge.apply(q, k, v, tq, tk, tv, o_t, o, M, mu, ctx.mask_spec, ctx.sm_scale, relay, link)


def _backward_impl(ctx, do):
    """(dq, dk, dv) of <do, O>, as a node that can be differentiated once more."""
    # Inside fwAD.dual_level() the saved q, k, v are still dual; only their primal parts (which
    # keep the backward graph needed for double backward) may enter the next Function.
    q, k, v, o, M = (fwAD.unpack_dual(x).primal for x in ctx.saved_tensors)
    _check_bwd_layout(q, k, v, o)
    return _AttnBwd.apply(q, k, v, o.detach(), M, fwAD.unpack_dual(do).primal, ctx.mask_spec, ctx.sm_scale)


def _backward_under_functorch(q, k, v, o, M, do, spec, sm_scale, tf32, parts):
    """The native layer's backward through O where the cotangent is a tensor of a functorch transform (``torch.func.grad``
    over a vector-Jacobian product, say): ``_AttnBwd`` takes part in it."""
    spec = copy.copy(spec)
    spec.fp32_mode, spec.fp32_parts = "tf32" if tf32 else "3xtf32", parts
    return _AttnBwd.apply(q, k, v, o, M, do, spec, sm_scale)


_NO_MASK = _lib.MaskSpec(_lib.MASK_NONE)
_CAUSAL = _lib.MaskSpec(_lib.MASK_CAUSAL)
_functorch = torch._C._functorch
_peek_functorch = _functorch.peek_interpreter_stack
_JVP = _functorch.TransformType.Jvp
_is_tracing = torch._C._is_tracing


def _attend(q, k, v, attn_mask, causal, sm_scale, dual):
    """The call behind ``fwd`` and ``fwd_dual``: the mask is looked up or classified here, everything else happens in
    the native layer (csrc/native.cpp).  What that does not take (bad arguments, nested transforms) goes through the
    Python Function, which words the errors."""
    interp = _peek_functorch()
    # no transform, or torch.func.jvp alone (a torch.jit.trace would record the native call's result as a constant)
    if (interp is None or (dual and interp.level() == 1 and interp.key() == _JVP)) and not _is_tracing():
        native = _lib.native()
        if attn_mask is None:
            spec = _CAUSAL if causal else _NO_MASK
        else:
            mask = attn_mask
            if interp is not None and _functorch.is_functorch_wrapped_tensor(mask):
                mask = _functorch._unwrap_for_grad(mask, 1)
            spec = None if causal else _remembered_mask(mask, q.shape)
        if spec is None or not q.is_cuda:  # (the native layer checks CUDA tensors itself, for a mask that is known to fit)
            _check_args(q, k, v, None, None, None, attn_mask, causal)
            if spec is None:
                with native.NoFunctorch():  # the mask is a plain tensor, and so is what is found out about it
                    spec = classify_mask(mask, causal, *q.shape[:3], q.dtype, True)[0]
        out = native.attend(q, k, v, attn_mask, spec.native(), sm_scale, _lib.FP32_PRECISION == "tf32", dual, STRICT_SEQUENCE_LENGTH)
        if out is not None:
            return out
    q_t, k_t, v_t = (fwAD.unpack_dual(x).tangent for x in (q, k, v)) if dual else (None, None, None)
    # every positional argument given: the quick signature binding applies
    return _Attn.apply(q, k, v, q_t, k_t, v_t, attn_mask, causal, sm_scale, True)[0]


class _Box:
    """One-slot holder that passes through ``Function.apply`` and the pytree handling of torch.func transforms as
    a single opaque leaf."""

    __slots__ = ("value",)

    def __init__(self, value=None):
        self.value = value


class _Attn(Function):
    """The general route of ``JVPAttn.fwd`` and ``JVPAttn.fwd_dual`` (functorch transforms other than a lone
    ``torch.func.jvp``): the same forward, jvp and backward as ``JVPAttn``, whose second output is one opaque holder of
    (o_t, M, mu, mask description, scale) instead of upstream's nested NamedTuples.  Under ``torch.func.jvp`` every output of a custom Function is wrapped and unwrapped as a pytree once
    per transform level; the NamedTuples (some twenty leaves) made that the larger part of a call's host time.
    ``JVPAttn.apply`` keeps upstream's output structure for callers that use it directly."""

    @staticmethod
    def forward(q, k, v, q_t, k_t, v_t, attn_mask, causal, sm_scale, verify_attn_mask):
        o, o_t, M, mu, spec, _, _, sm_scale, _, _ = _forward_impl(q, k, v, q_t, k_t, v_t, attn_mask, 0.0, causal, sm_scale,
                                                                 verify_attn_mask)
        # Third output (with tangents only): a scalar that the tangent's node takes as an input, so that autograd runs
        # that node before this one and the cotangent of tO can be handed over here (see backward).
        # The holder through which that hand-over goes is made here, once per call: under torch.func transforms
        # setup_context runs once per level, each time with another ctx.
        relay = _zero_scalar(o.device) if o_t is not None else None
        link = _Box(None) if o_t is not None else None
        return o, _Box((o_t, M, mu, spec, sm_scale, link)), relay

    @staticmethod
    def setup_context(ctx, inputs, outputs):
        q, k, v, q_t, k_t, v_t, *_ = inputs
        o, aux, relay = outputs
        o_t, M, mu, ctx.mask_spec, ctx.sm_scale, ctx.link = aux.value
        ctx.save_for_forward(o_t, q, k, v, q_t, k_t, v_t, o, M, mu, relay)
        ctx.save_for_backward(q, k, v, o, M)
        ctx.set_materialize_grads(False)

    @staticmethod
    def jvp(ctx, gq, gk, gv, *_):
        relay = ctx.saved_for_forward[10]
        return _jvp_impl(ctx, gq, gk, gv, relay, ctx.link), None, _zero_scalar(relay.device)

    @staticmethod
    def backward(ctx, do, _, _relay=None):
        handed = None
        if ctx.link is not None:
            handed, ctx.link.value = ctx.link.value, None
        if handed is None:
            if do is None:
                return (None,) * 10
            dq, dk, dv = _backward_impl(ctx, do)
            return (dq, dk, dv) + (None,) * 7
        gto, tq, tk, tv, to, mu = handed
        q, k, v, o, M = (fwAD.unpack_dual(x).primal for x in ctx.saved_tensors)
        _check_bwd_layout(q, k, v, o)
        if do is not None and torch.is_grad_enabled():
            # a second differentiation was asked for: the part through O stays a differentiable node of its own
            dq, dk, dv = _backward_impl(ctx, do)
            hq, hk, hv = _BwdThroughTangent.apply(q, k, v, tq, tk, tv, o, to, M, mu, gto, ctx.mask_spec, ctx.sm_scale)
            return (dq + hq, dk + hk, dv + hv) + (None,) * 7
        go = None if do is None else fwAD.unpack_dual(do).primal
        with torch.no_grad():
            dq, dk, dv = _launch_bwd(q.detach(), k.detach(), v.detach(), tq, tk, tv, o.detach(), to, M, mu, go, gto,
                                     ctx.mask_spec, ctx.sm_scale)
        return (dq, dk, dv) + (None,) * 7


attention = JVPAttn.fwd

# torch.autograd.Function.apply calls inspect.signature(cls.forward).bind(...) on every call of a
# Function that defines setup_context (to fill in default arguments): ~45 us to build the signature and
# ~35 us to bind, per apply, of the ~0.3 ms that the host side of one fwd_dual call used to take.
# inspect.signature returns a function's __signature__ attribute when there is one; the signature
# object below also short-cuts the binding of a complete positional argument list.
class _BoundPositional:
    __slots__ = ("args",)

    def __init__(self, args):
        self.args = args

    def apply_defaults(self):
        pass


class _ForwardSignature(inspect.Signature):
    def bind(self, *args, **kwargs):
        if not kwargs and len(args) == len(self.parameters):
            return _BoundPositional(args)
        return super().bind(*args, **kwargs)


for _fn in (JVPAttn, _Attn, _TangentBridge, _AttnBwd):
    _sig = inspect.signature(_fn.forward)
    _fn.forward.__signature__ = _ForwardSignature(list(_sig.parameters.values()), return_annotation=_sig.return_annotation)
del _fn, _sig


def scaled_dot_product_attention(query: Tensor, key: Tensor, value: Tensor, attn_mask: Tensor | None = None,
                                 dropout_p: float = 0.0, is_causal: bool = False,
                                 scale: float | None = None) -> Tensor:
    """``torch.nn.functional.scaled_dot_product_attention``-shaped entry point.

    Accepts plain or forward-AD dual (B, H, L, D) tensors and forwards to ``JVPAttn.fwd_dual``
    with SDPA's argument names, which is how upstream's README wires the kernel into a model.
    """
    return JVPAttn.fwd_dual(query, key, value, attn_mask=attn_mask, dropout_p=dropout_p, causal=is_causal,
                            sm_scale=scale)


class _Module(types.ModuleType):
    """Forwards the launch switches to the native layer when they are set."""

    def __setattr__(self, name, value):
        super().__setattr__(name, value)
        if name == "KERNEL_IMPL":
            _lib.native().set_impl(value)
        elif name == "SINGLE_PASS_BACKWARD":
            _lib.native().set_single_pass(value)


sys.modules[__name__].__class__ = _Module
