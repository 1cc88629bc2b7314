"""jvpfa_pad_bias: a ragged bias of 16-bit elements with its rows padded to whole 16-byte pieces."""
import ctypes

import pytest
import torch

from jvp_flash_attention_b200 import _lib

DEV = "cuda:0"


def _args(m, padded, **fields):
    spec = _lib.MaskSpec(_lib.MASK_BIAS, m, tuple(0 if n == 1 else s for n, s in zip(m.shape, m.stride())), _lib.DTYPE_ENUM[m.dtype])
    a = _lib.PadBiasArgs(struct_size=ctypes.sizeof(_lib.PadBiasArgs), n_b=m.shape[0], n_h=m.shape[1], L=m.shape[2], width=padded.shape[3], mask=spec.to_c(),
                         out=padded.data_ptr())
    a.mask.stride[3] = m.stride(3)
    for name, value in fields.items():
        setattr(a, name, value)
    return a


@pytest.mark.gpu
@pytest.mark.parametrize("L", [33, 66, 130, 255, 1026, 1033])
@pytest.mark.parametrize("layout", ["rows", "offset", "wider rows", "keys first", "keys apart"])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
def test_rows_are_padded(L, layout, dt):
    """Entries bit for bit, zeros behind them, of rows that begin at even and odd places, the last one at the end of its storage."""
    g = torch.Generator(device=DEV).manual_seed(L)
    want = torch.randn(2, 2, L, L, generator=g, device=DEV).to(dt)
    m = want
    if layout == "offset":
        m = torch.cat([want.new_ones(1), want.flatten()])[1:].view(want.shape)
    elif layout == "wider rows":
        m = torch.nn.functional.pad(want, (3, 2), value=7.0)[..., 3:-2]
    elif layout == "keys first":
        m = want.transpose(2, 3).contiguous().transpose(2, 3)
    elif layout == "keys apart":
        m = want.repeat_interleave(2, -1)[..., ::2]
    for width in ((L + 7) // 8 * 8, (L + 31) // 8 * 8):
        out = torch.full((2, 2, L, width), 3.0, dtype=dt, device=DEV)
        _lib.check(_lib.load().jvpfa_pad_bias(ctypes.byref(_args(m, out)), torch.cuda.current_stream().cuda_stream), "jvpfa_pad_bias")
        assert torch.equal(out[..., :L], want) and not out[..., L:].any()


@pytest.mark.gpu
@pytest.mark.parametrize("L,width", [(1, 8), (33, 128), (113, 120), (120, 128), (121, 128), (128, 136), (129, 136), (249, 256), (250, 256), (255, 264), (505, 512), (506, 520), (1023, 1024), (1025, 1032)])
@pytest.mark.parametrize("heads", [(1, 1), (3, 5)])
def test_edges_of_what_a_warp_takes(L, width, heads):
    """Rows of up to 128, 256, 512 and more elements, and heads that end within a block's rows: entries bit for bit, zeros behind them, nothing elsewhere."""
    g = torch.Generator(device=DEV).manual_seed(L)
    m = torch.randn(*heads, L, L, generator=g, device=DEV).to(torch.bfloat16)
    out = torch.full((heads[0] * heads[1] * L * width + 64,), 3.0, dtype=m.dtype, device=DEV)
    view = out[:-64].view(*heads, L, width)
    _lib.check(_lib.load().jvpfa_pad_bias(ctypes.byref(_args(m, view)), torch.cuda.current_stream().cuda_stream), "jvpfa_pad_bias")
    assert torch.equal(view[..., :L], m) and not view[..., L:].any() and (out[-64:] == 3).all()


def test_what_is_refused():
    """Host logic, before anything is launched."""
    m, out = torch.zeros(1, 1, 66, 66, dtype=torch.float16), torch.zeros(1, 1, 66, 72, dtype=torch.float16)
    lib = _lib.load()
    for status, fields in (("STRUCT", {"struct_size": 8}), ("SHAPE", {"width": 70}), ("SHAPE", {"width": 64}), ("SHAPE", {"L": 0}), ("NULL", {"out": None}),
                           ("ALIGN", {"out": out.data_ptr() + 2})):
        rc = lib.jvpfa_pad_bias(ctypes.byref(_args(m, out, **fields)), None)
        word = {"STRUCT": "struct_size", "SHAPE": "shape", "NULL": "NULL", "ALIGN": "aligned"}[status]
        assert rc != 0 and word in lib.jvpfa_strerror(rc).decode(), (status, fields)
    a = _args(m, out)
    a.mask.bias_dtype = _lib.FP32
    assert "dtype" in lib.jvpfa_strerror(lib.jvpfa_pad_bias(ctypes.byref(a), None)).decode()
