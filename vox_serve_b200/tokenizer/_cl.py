"""Vocoder convolutions over channels-last activations [B, T, C] (csrc/cl_conv.cu), shared by the SNAC and Mimi decoders: layers
whose widths are multiples of 32 channels run as one product per tap on tcgen05 (two fp16 parts a value, fp32 accumulation)."""
from __future__ import annotations

from typing import Optional

import torch

from .. import _lib, ops
from .._lib import VoxB200Error, call

EPI = {"plain": 0, "resid": 1, "scale_resid": 2, "noise": 3}
ACT = {None: 0, "snake": 1, "elu": 2, "gelu": 3}


def pack(w: torch.Tensor) -> torch.Tensor:
    """w fp32 [N, K] on the device (K tap-major, the tap furthest back first) -> packed tiles"""
    N, K = w.shape
    dst = torch.empty(_lib.load().vb_cl_pack_bytes(N, K), dtype=torch.uint8, device=w.device)
    call("vb_cl_pack", dst.data_ptr(), w.contiguous().data_ptr(), N, K, ops._stream())
    return dst


def pack_conv(w: torch.Tensor, cin: int, ksize: int) -> torch.Tensor:
    """w [Cout, Cin * ksize], channel-major and tap-minor (a flattened Conv1d weight)"""
    cout = w.shape[0]
    return pack(w.view(cout, cin, ksize).permute(0, 2, 1).reshape(cout, ksize * cin))


def pack_convtr(wp: torch.Tensor) -> torch.Tensor:
    """wp [stride, Cout, 2 Cin]: per output phase the tap on the input position itself, then the one on its predecessor"""
    s, cout, k = wp.shape
    return pack(torch.cat((wp[..., k // 2:], wp[..., :k // 2]), -1).reshape(s * cout, k))


class Act:
    """An activation [B, T, C] inside a buffer: entry b starts at offset + b * bstride floats.  ``parts``: kept as what the convolutions
    multiply, two fp16 parts a value in the place of a float, with a code byte per 32 channels behind them (written by the kernels
    that produce them, read by ``conv`` and ``conv_transposed`` only)."""
    __slots__ = ("buf", "B", "T", "C", "offset", "bstride", "parts")

    def __init__(self, buf: torch.Tensor, B: int, T: int, C: int, offset: int = 0, bstride: Optional[int] = None, parts: bool = False):
        self.buf, self.B, self.T, self.C, self.offset, self.parts = buf, B, T, C, offset, parts
        self.bstride = T * C if bstride is None else bstride

    @classmethod
    def empty(cls, B: int, T: int, C: int, device, parts: bool = False, offset: int = 0, bstride: Optional[int] = None) -> "Act":
        n = B * (T * C if bstride is None else bstride)
        return cls(torch.empty(n + n // 128 + 1 if parts else n, dtype=torch.float32, device=device), B, T, C, offset, bstride, parts)

    @property
    def ptr(self) -> int:
        return self.buf.data_ptr() + 4 * self.offset

    @property
    def codes(self) -> Optional[int]:
        return self.buf.data_ptr() + 4 * self.B * self.bstride + self.offset // 32 if self.parts else None

    def tensor(self) -> torch.Tensor:
        """[B, T, C] view"""
        if self.parts:
            raise VoxB200Error("an activation kept as parts has no view as floats")
        return self.buf.as_strided((self.B, self.T, self.C), (self.bstride, self.C, 1), self.offset)


def _ptr(t) -> Optional[int]:
    return None if t is None else (t.ptr if isinstance(t, Act) else t.data_ptr())


def _outputs(both: bool, out: str, new):
    """(plain fp32, activated fp32, activated parts) of a convolution, and what it returns"""
    if out not in ("f32", "parts"):
        raise VoxB200Error(f"unknown form {out!r} of a convolution's result")
    last = new(out == "parts")
    plain = new(False) if both else None
    if out == "parts":
        return (plain, None, last), ((plain, last) if both else last)
    return ((plain, last, None), (plain, last)) if both else ((last, None, None), last)


def conv(x: Act, w: torch.Tensor, N: int, bias=None, ksize: int = 1, dil: int = 1, epi: str = "plain", resid: Optional[Act] = None,
         scale=None, noise=None, act: Optional[str] = None, alpha=None, lo: int = 0, hi: Optional[int] = None,
         both: bool = False, out: str = "f32"):
    """Causal convolution (zeros before the start) of rows [lo, hi) -> Act [B, T, N]; ``both``: (plain, activated).  ``out``: the
    activated values as floats or as parts for the next convolution."""
    hi = x.T if hi is None else hi
    (y, y2, yp), ret = _outputs(both, out, lambda parts: Act.empty(x.B, x.T, N, x.buf.device, parts))
    call("vb_cl_conv_parts", _ptr(y), _ptr(y2), _ptr(yp), yp.codes if yp else None, x.ptr, x.codes, x.bstride, x.T, w.data_ptr(), _ptr(bias),
         _ptr(resid), resid.bstride if resid else 0, _ptr(scale), _ptr(noise), noise.shape[-1] if noise is not None else 0, _ptr(alpha), EPI[epi],
         ACT[act], x.B, x.C, N, N, ksize, dil, lo, hi, x.T * N, ops._stream())
    return ret


def conv_transposed(x: Act, w: torch.Tensor, cout: int, stride: int, bias, pad: int = 0, o_lo: int = 0, o_hi: Optional[int] = None,
                    act: Optional[str] = None, both: bool = False, out: str = "f32"):
    """Transposed convolution with 2 * stride taps -> Act [B, T * stride, cout]; ``pad`` positions are dropped in front.  Output
    positions [o_lo, o_hi) are computed."""
    T_out = x.T * stride
    o_hi = T_out if o_hi is None else o_hi
    n_lo, n_hi = (o_lo + pad) // stride, (o_hi - 1 + pad) // stride + 1
    N = stride * cout
    rows = x.T + (1 if pad else 0)
    (y, y2, yp), ret = _outputs(both, out, lambda parts: Act.empty(x.B, T_out, cout, x.buf.device, parts, pad * cout, rows * N))
    base = lambda a: None if a is None else a.buf.data_ptr()                 # noqa: E731  (the kernel's rows start before the padding)
    call("vb_cl_conv_parts", base(y), base(y2), base(yp), yp.codes - yp.offset // 32 if yp else None, x.ptr, x.codes, x.bstride, x.T, w.data_ptr(),
         _ptr(bias), None, 0, None, None, 0, None, EPI["plain"], ACT[act], x.B, x.C, N, cout, 2, 1, n_lo, n_hi, rows * N, ops._stream())
    return ret


def depthwise7(x: Act, w: torch.Tensor, bias, alpha_in, alpha_out, dil: int, lo: int, hi: int, parts: bool = False) -> Act:
    """w [7, C]; alpha tables [2, C]: values, then 1 / (alpha + 1e-9)"""
    y = Act.empty(x.B, x.T, x.C, x.buf.device, parts)
    call("vb_cl_dwconv7_parts", y.ptr, y.codes, x.ptr, x.bstride, w.data_ptr(), _ptr(bias), _ptr(alpha_in), _ptr(alpha_out), x.B, x.C, x.T, dil, lo, hi,
         ops._stream())
    return y


def dw_unit_pays(x: Act, dil: int, rows: int) -> bool:
    """whether ``dw_unit`` is the faster way (the results are the same bits)"""
    return bool(_lib.load().vb_cl_dw_unit_pays(x.B, x.C, rows, dil))


def dw_unit(x: Act, dw_w: torch.Tensor, dw_b, alpha_in, alpha_mid, w: torch.Tensor, bias, dil: int, lo: int, hi: int, alpha_out=None,
            out: str = "f32") -> Act:
    """x + 1x1(Snake(depthwise7(Snake(x)))) for rows [lo, hi), then a Snake if ``alpha_out``: ``depthwise7`` and ``conv`` in one launch"""
    y = Act.empty(x.B, x.T, x.C, x.buf.device, out == "parts")
    call("vb_cl_dw_unit", None if y.parts else y.ptr, y.ptr if y.parts else None, y.codes, x.ptr, x.bstride, dw_w.data_ptr(), dw_b.data_ptr(),
         alpha_in.data_ptr(), alpha_mid.data_ptr(), w.data_ptr(), bias.data_ptr(), _ptr(alpha_out), x.B, x.C, x.T, dil, lo, hi, ops._stream())
    return y


def res_tail(x: Act, w1: torch.Tensor, b1, w3: torch.Tensor, b3, wl: torch.Tensor, bl) -> torch.Tensor:
    """The last residual unit of 64 channels (three taps to 32, ELU, 1x1 back), ELU and the convolution of three taps to one channel -> [B, 1, T]"""
    y = torch.empty(x.B, 1, x.T, dtype=torch.float32, device=x.buf.device)
    call("vb_cl_res_tail", y.data_ptr(), x.ptr, x.bstride, w1.data_ptr(), b1.data_ptr(), w3.data_ptr(), b3.data_ptr(), wl.data_ptr(), bl.data_ptr(), x.B, x.T,
         ops._stream())
    return y


def last_conv(x: Act, w: torch.Tensor, bias, ksize: int, left: int, t0: int, t1: int, tanh: bool) -> torch.Tensor:
    """one output channel -> [B, 1, t1 - t0]; w [C, ksize]"""
    y = torch.empty(x.B, 1, t1 - t0, dtype=torch.float32, device=x.buf.device)
    call("vb_cl_last_conv", y.data_ptr(), x.ptr, x.bstride, w.data_ptr(), _ptr(bias), x.B, x.C, x.T, ksize, left, t0, t1, int(tanh), ops._stream())
    return y
