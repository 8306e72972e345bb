"""Device-side quantizers for the `sb6` and `sym` layouts.

The counterpart of the reference's host-side packer for its block formats
(`formats/writer.py:236-269` `_make_qt_gw_sb6` over `calibration/groupwise.py:207-300`): the
scale search, the code selection and the bit packing into the file buffers run in one CUDA kernel
(`rwkvq_quantize_sb6_packed`, a thread per block of 32 weights).
The result is a `QuantizedTensor` a `.rwkvq` file can hold and the kernels can read.
"""
from __future__ import annotations

import functools
from typing import Optional

import torch

from . import _lib
from .formats import QuantizedTensor

MODES = {"asym_sb6": False, "asym_sb6_search": True, "asym_sb6_aw": True}
SYM_MODES = ("sym", "sym_aw", "sym_plain")


def sym_factors() -> torch.Tensor:
    """The scale factors the reference's symmetric search visits: the float32 nodes of
    torch.linspace(0.7, 1.15, 19) (calibration/groupwise.py:305)."""
    return torch.linspace(0.7, 1.15, 19, dtype=torch.float32, device="cpu")


@functools.lru_cache(maxsize=16)
def _factors(search: bool, device: torch.device) -> torch.Tensor:
    """The search's scale factors on a device (19 constants: uploaded once)."""
    return (sym_factors() if search else torch.ones(1, dtype=torch.float32, device="cpu")).to(device)


def _prepared(who: str, w: torch.Tensor, ex2: Optional[torch.Tensor]):
    """(w fp32 contiguous, ex2 fp32 on its device or None) of a quantizer call."""
    if not w.is_cuda or w.dim() != 2:
        raise ValueError(f"{who}: a 2-D CUDA tensor is required")
    n = w.shape[1]
    if n % 256:
        raise ValueError(f"{who}: IN={n} is not a multiple of 256")
    e = None
    if ex2 is not None:
        e = ex2.to(device=w.device, dtype=torch.float32).contiguous()
        if e.numel() != n:
            raise ValueError(f"{who}: ex2 needs one value per input channel")
    return w.float().contiguous(), e


def quantize_sb6_parts(w: torch.Tensor, bits: int, search: bool = True, ex2: Optional[torch.Tensor] = None):
    """(q u8 [OUT, IN], qs u8 [OUT, IN/32], qm i8 [OUT, IN/32], d f16 [OUT, IN/256], dm f16) on the device."""
    w32, e = _prepared("quantize_sb6", w, ex2)
    o, n = w32.shape
    dev = w.device
    q = torch.empty((o, n), dtype=torch.uint8, device=dev)
    qs = torch.empty((o, n // 32), dtype=torch.uint8, device=dev)
    qm = torch.empty((o, n // 32), dtype=torch.int8, device=dev)
    d = torch.empty((o, n // 256), dtype=torch.float16, device=dev)
    dm = torch.empty((o, n // 256), dtype=torch.float16, device=dev)
    lib = _lib.load(check_device=True)
    with torch.cuda.device(dev):
        _lib.check(lib.rwkvq_quantize_sb6(w32.data_ptr(), n, o, n, bits, 1 if search else 0,
                                          e.data_ptr() if e is not None else None, q.data_ptr(), qs.data_ptr(),
                                          qm.data_ptr(), d.data_ptr(), dm.data_ptr(), _lib.stream_ptr()), "rwkvq_quantize_sb6")
    return q, qs, qm, d, dm


def quantize_sb6(key: str, group: str, w: torch.Tensor, bits: int, mode: str = "asym_sb6_search",
                 ex2: Optional[torch.Tensor] = None) -> QuantizedTensor:
    """`w` [OUT, IN] -> a packed sb6 `QuantizedTensor` (buffers stay on w's device).  mode: one of
    asym_sb6 (min / max scales), asym_sb6_search (scale search + least-squares refit), asym_sb6_aw
    (the search weighted by `ex2`, E[x^2] per input channel)."""
    if mode not in MODES:
        raise ValueError(f"quantize_sb6: mode {mode!r}")
    if (mode == "asym_sb6_aw") != (ex2 is not None):
        raise ValueError("quantize_sb6: ex2 goes with mode asym_sb6_aw, and only with it")
    w32, e = _prepared("quantize_sb6", w, ex2)
    (o, n), dev = w32.shape, w32.device
    u8 = dict(dtype=torch.uint8, device=dev)
    packed = torch.empty((o, n // 2), **u8)
    qh = torch.empty((o, n // 8), **u8) if bits >= 5 else None
    qh2 = torch.empty((o, n // 8), **u8) if bits >= 6 else None
    qsqm = torch.empty((o, n // 256, 12), **u8)
    d = torch.empty((o, n // 256), dtype=torch.float16, device=dev)
    dm = torch.empty_like(d)
    lib = _lib.load(check_device=True)
    with torch.cuda.device(dev):
        _lib.check(lib.rwkvq_quantize_sb6_packed(w32.data_ptr(), n, o, n, bits, 1 if MODES[mode] else 0, _lib.ptr(e) or None,
                                                 packed.data_ptr(), _lib.ptr(qh) or None, _lib.ptr(qh2) or None, qsqm.data_ptr(),
                                                 d.data_ptr(), dm.data_ptr(), _lib.stream_ptr()), "rwkvq_quantize_sb6_packed")
    return QuantizedTensor(key=key, group=group, bits=bits, shape=(o, n), gw_mode="sb6", gw_gs=32, gw_sb=8,
                           codes_packed=packed, gw_qh=qh, gw_qh2=qh2, gw_qsqm=qsqm, gw_d=d, gw_dm=dm)


def quantize_sym_parts(w: torch.Tensor, bits: int, search: bool = True, ex2: Optional[torch.Tensor] = None):
    """(q i8 [OUT, IN], qs i8 [OUT, IN/16], d f16 [OUT, IN/256]) on the device."""
    w32, e = _prepared("quantize_sym", w, ex2)
    (o, n), dev = w32.shape, w32.device
    f = _factors(search, dev)
    q = torch.empty((o, n), dtype=torch.int8, device=dev)
    qs = torch.empty((o, n // 16), dtype=torch.int8, device=dev)
    d = torch.empty((o, n // 256), dtype=torch.float16, device=dev)
    lib = _lib.load(check_device=True)
    with torch.cuda.device(dev):
        _lib.check(lib.rwkvq_quantize_sym(w32.data_ptr(), n, o, n, bits, f.data_ptr(), f.numel(),
                                          e.data_ptr() if e is not None else None, q.data_ptr(), qs.data_ptr(), d.data_ptr(),
                                          _lib.stream_ptr()), "rwkvq_quantize_sym")
    return q, qs, d


def quantize_sym(key: str, group: str, w: torch.Tensor, bits: int, mode: str = "sym",
                 ex2: Optional[torch.Tensor] = None) -> QuantizedTensor:
    """`w` [OUT, IN] -> a packed sym `QuantizedTensor` (bits 6 or 8).  mode: sym (scale search), sym_aw (the
    search weighted by `ex2`), sym_plain (no search); the counterpart of `formats/writer.py::_make_qt_gw_sym`."""
    if mode not in SYM_MODES:
        raise ValueError(f"quantize_sym: mode {mode!r}")
    if (mode == "sym_aw") != (ex2 is not None):
        raise ValueError("quantize_sym: ex2 goes with mode sym_aw, and only with it")
    if bits != 6:                                        # 8; the library refuses others
        q, qs, d = quantize_sym_parts(w, bits, mode != "sym_plain", ex2)
        return QuantizedTensor(key=key, group=group, bits=bits, shape=tuple(w.shape), gw_mode="sym", gw_gs=16, gw_sb=16, gw_qs=qs, gw_d=d, codes=q)
    w32, e = _prepared("quantize_sym", w, ex2)
    (o, n), dev = w32.shape, w32.device
    f = _factors(mode != "sym_plain", dev)
    packed = torch.empty((o, n // 2), dtype=torch.uint8, device=dev)
    qh = torch.empty((o, n // 8), dtype=torch.uint8, device=dev)
    qh2 = torch.empty_like(qh)
    qs = torch.empty((o, n // 16), dtype=torch.int8, device=dev)
    d = torch.empty((o, n // 256), dtype=torch.float16, device=dev)
    lib = _lib.load(check_device=True)
    with torch.cuda.device(dev):
        _lib.check(lib.rwkvq_quantize_sym6_packed(w32.data_ptr(), n, o, n, f.data_ptr(), f.numel(), _lib.ptr(e) or None,
                                                  packed.data_ptr(), qh.data_ptr(), qh2.data_ptr(), qs.data_ptr(), d.data_ptr(),
                                                  _lib.stream_ptr()), "rwkvq_quantize_sym6_packed")
    return QuantizedTensor(key=key, group=group, bits=6, shape=(o, n), gw_mode="sym", gw_gs=16, gw_sb=16, codes_packed=packed,
                           gw_qh=qh, gw_qh2=qh2, gw_qs=qs, gw_d=d)
