"""Stand-alone codec kernels on local memory (no communicator): what the compression
hook ABIs are built from. Wire layout of `count` elements: pad = count rounded up to 512,
[payload: pad elements][scales: pad / group entries]."""
from __future__ import annotations

import ctypes
import functools

import torch

from .. import constants as K
from .._lib import calls, lib
from ..comm import _check, _DTYPES, current_stream_ptr as _stream, taken, wire_bytes


@functools.cache   # the declarations once: plain integers then go straight through
def _lib():
    L = lib()
    i, u, vp = ctypes.c_int, ctypes.c_uint64, ctypes.c_void_p
    for f in (L.ccb_encode, L.ccb_decode, L.ccb_decode_reduce):
        f.argtypes = [i, i, vp, u, vp, vp]
    L.ccb_reduce_recode.argtypes = [i, ctypes.POINTER(vp), i, u, vp, vp]
    L.ccb_refwire_encode.argtypes = L.ccb_refwire_decode.argtypes = [i, vp, u, i, vp, vp]
    return L


def encode(x: torch.Tensor, codec: str) -> torch.Tensor:
    """Returns the wire bytes (uint8 tensor) of a contiguous CUDA tensor."""
    if (c := calls()) is not None and (made := c.encode(x, codec)) is not None:
        return taken(made)
    wire = torch.empty(wire_bytes(codec, x.dtype, x.numel()), dtype=torch.uint8, device=x.device)
    _check(_lib().ccb_encode(K.CODECS[codec], _DTYPES[x.dtype], x.data_ptr(), x.numel(), wire.data_ptr(), _stream()))
    return wire


def decode(wire: torch.Tensor, codec: str, count: int, dtype: torch.dtype) -> torch.Tensor:
    if (c := calls()) is not None and (made := c.decode(wire, codec, count, dtype)) is not None:
        return taken(made)
    out = torch.empty(count, dtype=dtype, device=wire.device)
    _check(_lib().ccb_decode(K.CODECS[codec], _DTYPES[dtype], wire.data_ptr(), count, out.data_ptr(), _stream()))
    return out


def decode_reduce(wire: torch.Tensor, codec: str, inout: torch.Tensor) -> torch.Tensor:
    """inout += decode(wire), one kernel."""
    _check(_lib().ccb_decode_reduce(K.CODECS[codec], _DTYPES[inout.dtype], wire.data_ptr(), inout.numel(), inout.data_ptr(),
                                   _stream()))
    return inout


def reduce_recode(wires, codec: str, count: int) -> torch.Tensor:
    """encode(sum_k decode(wires[k])) without leaving the compressed domain in memory."""
    if (c := calls()) is not None and (made := c.reduce_recode(wires, codec, count)) is not None:
        return taken(made)
    arr = (ctypes.c_void_p * len(wires))(*[w.data_ptr() for w in wires])
    out = torch.empty_like(wires[0])
    _check(_lib().ccb_reduce_recode(K.CODECS[codec], arr, len(wires), count, out.data_ptr(), _stream()))
    return out


def refwire_bytes(count: int, group: int) -> int:
    return (count + group - 1) // group * 4 + count


def refwire_encode(x: torch.Tensor, group: int = 256) -> torch.Tensor:
    """The reference wrapper's int8 wire: [f32 127/absmax per group][int8 x count]."""
    wire = torch.empty(refwire_bytes(x.numel(), group), dtype=torch.uint8, device=x.device)
    _check(_lib().ccb_refwire_encode(_DTYPES[x.dtype], x.data_ptr(), x.numel(), group, wire.data_ptr(), _stream()))
    return wire


def refwire_decode(wire: torch.Tensor, count: int, dtype: torch.dtype, group: int = 256) -> torch.Tensor:
    out = torch.empty(count, dtype=dtype, device=wire.device)
    _check(_lib().ccb_refwire_decode(_DTYPES[dtype], wire.data_ptr(), count, group, out.data_ptr(), _stream()))
    return out
