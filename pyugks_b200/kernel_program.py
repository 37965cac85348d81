"""The reference's kernel-call surface, served by libugks_b200.so.

pyUGKS launches every kernel as ``self.prg.<name>(queue, global_size,
local_size, *args)`` on a per-block ``cl.Program`` (``ugks_block.py:184``).
``KernelProgram`` keeps that surface: attribute names are the reference kernel
names, arguments come in the reference order, buffers are torch CUDA tensors
in the reference layout and scalars are Python ints / floats.  Each call
forwards to ``ugks_<name>(desc, g0, g1, *args, stream)``; the per-block
``ugks_block_desc`` takes the place of the generated OpenCL header.

``queue`` is a ``torch.cuda.Stream`` (or None for the current stream);
``local_size`` is accepted and ignored (the CUDA launch shape is fixed by the
library).
"""
from __future__ import annotations

import ctypes as C

import torch

from . import _lib


class KernelProgram:
    def __init__(self, desc: "_lib.BlockDesc"):
        self.desc = desc
        self._lib = _lib.lib()
        self._calls = {}

    def __getattr__(self, name):
        if name.startswith("_"):
            raise AttributeError(name)
        if name not in _lib.KERNEL_SIGNATURES:
            raise AttributeError("no kernel %r in the UGKS program" % name)
        call = self._calls.get(name)
        if call is None:
            call = self._make(name)
            self._calls[name] = call
        return call

    def _make(self, name):
        fn = getattr(self._lib, "ugks_" + name)
        sig = _lib.KERNEL_SIGNATURES[name]
        desc = C.byref(self.desc)
        count = len(sig)

        def pointer(a):
            if not a.is_cuda or not a.is_contiguous():
                raise ValueError("%s: buffers must be contiguous CUDA tensors" % name)
            return a.data_ptr()

        convert = [pointer if k == "p" else int if k == "i" else float for k in sig]

        def call(queue, global_size, local_size, *args):
            if len(args) != count:
                raise TypeError("%s takes %d kernel arguments, got %d" % (name, count, len(args)))
            conv = [f(a) for f, a in zip(convert, args)]
            g0 = int(global_size[0])
            g1 = int(global_size[1]) if len(global_size) > 1 else 1
            rc = fn(desc, g0, g1, *conv, _stream_ptr(queue))
            if rc:
                _lib.check(rc, name)

        call.__name__ = name
        return call


# the current device's current stream, without the Stream object that
# torch.cuda.current_stream() makes (13 us of a 26 us call); names of torch's own
# that not every version has to have
_get_device = getattr(torch._C, "_cuda_getDevice", None)
_get_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr(queue):
    if queue is None:
        if _get_device is None or _get_raw_stream is None:
            return torch.cuda.current_stream().cuda_stream
        return _get_raw_stream(_get_device())
    if isinstance(queue, int):
        return queue
    return queue.cuda_stream
