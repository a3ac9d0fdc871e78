"""Host <-> device plumbing shared by the reference-shaped classes."""
from __future__ import annotations

import numpy as np

from . import _native as nv

_U8, _I8 = -2, -3                                       # element codes of nv.host().upload beside the float codes
_UPLOAD_FLOAT = (np.dtype(np.float16), np.dtype(np.float32), np.dtype(np.float64))
_UPLOAD_INT = (np.dtype(np.int64), np.dtype(np.int32), np.dtype(np.uint8), np.dtype(np.int8))
_DOWNLOAD = _UPLOAD_FLOAT + _UPLOAD_INT


def _index(torch, dev):
    return torch.cuda.current_device() if dev.index is None else dev.index


def to_device(x, device=None, allow_f64=False):
    """(tensor on the GPU, was_numpy, original float dtype or None).

    NumPy arrays are uploaded; CUDA tensors are used in place.  fp64 survives only where the
    caller's kernel takes it (dense mode); everything else that is not fp16/bf16/fp32 becomes fp32.
    """
    torch = nv.require_cuda()
    was_numpy = not isinstance(x, torch.Tensor)
    dev = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    if was_numpy:
        arr = np.asarray(x)
        src_dtype = arr.dtype if arr.dtype.kind == "f" else None
        if arr.dtype.kind != "f":
            arr = arr.astype(np.float64)
        arr = np.ascontiguousarray(arr)
        if arr.dtype in _UPLOAD_FLOAT:
            code = nv.F16 if arr.dtype.itemsize == 2 else nv.F64 if arr.dtype.itemsize == 8 and allow_f64 else nv.F32
            return nv.host().upload(arr, _index(torch, dev), code), True, src_dtype
        t = torch.from_numpy(arr)
    else:
        t, src_dtype = x, None
    if t.device.type != "cuda":
        t = t.to(dev)
    keep = (torch.float16, torch.bfloat16, torch.float32) + ((torch.float64,) if allow_f64 else ())
    if t.dtype not in keep:
        t = t.to(torch.float32)
    return t.contiguous(), was_numpy, src_dtype


def ints_to_device(a, device, dtype):
    torch = nv.require_cuda()
    if isinstance(a, torch.Tensor):
        return a.to(device=device, dtype=dtype).contiguous()
    arr = np.ascontiguousarray(np.asarray(a))
    if arr.dtype in _UPLOAD_INT and dtype in (torch.uint8, torch.int8):
        return nv.host().upload(arr, _index(torch, device), _U8 if dtype == torch.uint8 else _I8)
    return torch.from_numpy(arr).to(device=device, dtype=dtype).contiguous()


def floats_to_device(a, device):
    torch = nv.require_cuda()
    if isinstance(a, torch.Tensor):
        return a.to(device=device, dtype=torch.float32).contiguous()
    arr = np.asarray(a)
    if arr.dtype not in _UPLOAD_FLOAT:
        arr = arr.astype(np.float64)
    return nv.host().upload(np.ascontiguousarray(arr), _index(torch, device), nv.F32)


def to_numpy(*pairs):
    """(tensor, NumPy type) pairs -> arrays of those types, all behind one wait for the device."""
    out, jobs = [], []
    for t, dtype in pairs:
        dtype = np.dtype(dtype)
        if dtype in _DOWNLOAD:
            a = np.empty(tuple(t.shape), dtype)
            jobs += (t, a)
        else:
            a = t.cpu().numpy().astype(dtype)
        out.append(a)
    nv.host().download(*jobs)
    return out
