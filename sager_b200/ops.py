"""The reference's launcher names on torch device tensors.

`ops.<name>(...)` calls `sgr_<name>` of the C ABI with the same argument order
as `sager::cuda::<name>` (include/sager/kernels/cuda_ops.hpp of the reference);
tensors are passed as raw device pointers and the trailing stream argument is
torch's current stream. Nothing here computes: a missing library raises.
"""
from __future__ import annotations

import ctypes as C
import sys

import torch

from .capi import SagerError, kinds_of, lib


_raw_stream = torch._C._cuda_getCurrentRawStream
_device = torch._C._cuda_getDevice


def _stream() -> int:
    """torch's current stream as an address (0 is the default stream), without building a Stream object."""
    if not torch.cuda.is_initialized():
        torch.cuda.init()
    return _raw_stream(_device())


def stream_ptr():
    return C.c_void_p(_stream())


_fast = None


def _fastcall():
    """The extension module that makes the calls (csrc/fastcall.c); False where it was not built for this interpreter."""
    global _fast
    if _fast is None:
        try:
            from . import _fastcall
        except ImportError:
            _fast = False
        else:
            _fastcall.setup(torch.Tensor, torch.nn.Parameter, _stream, _raw_stream, _device)
            _fast = _fastcall
    return _fast


def _bind(name: str):
    """The entry point as a callable: tensors go as device addresses, the current stream last. A decode step issues
    hundreds of these: the extension module makes the call; `slow` takes the arguments that it does not know, and parameter
    lists that it was not built with."""
    L = lib()
    cfn = getattr(L.cdll, "sgr_" + name)
    tensor, stream = torch.Tensor, _stream

    def fail(rc):
        raise SagerError("sgr_" + name, rc)

    def slow(*args):
        rc = cfn(*[a.data_ptr() if isinstance(a, tensor) else a for a in args], stream())
        if rc != 0:
            fail(rc)

    slow.__name__ = name
    kinds = kinds_of(L.protos["sgr_" + name])
    fast = None if kinds is None else _fastcall()
    fn = fast.bind(kinds, C.cast(cfn, C.c_void_p).value, slow, fail, name) if fast else None
    return slow if fn is None else fn


def call(name: str, *args):
    getattr(sys.modules[__name__], name)(*args)


def __getattr__(name):
    if name.startswith("_"):
        raise AttributeError(name)
    if "sgr_" + name not in lib().protos:
        raise AttributeError(f"no entry point sgr_{name}")
    fn = globals()[name] = _bind(name)
    return fn


def ptr_table(tensors, device):
    """int64 device tensor of data pointers (0 for None)."""
    return torch.tensor([0 if t is None else t.data_ptr() for t in tensors], dtype=torch.int64,
                        device=device)
