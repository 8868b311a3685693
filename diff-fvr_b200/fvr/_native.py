"""The native autograd binding (``_fvr_autograd``, built from
csrc/fvr_autograd.cpp next to the CUDA library), bound to the loaded library.

Its nodes run the same library calls as the Python autograd nodes, which stay
for what the binding does not cover: a checkout without it, launches being
timed one by one, and calls under a functorch transform (where a C++ node
would see wrapped tensors).
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib as L
from . import profiling

try:
    from . import _fvr_autograd as _MOD
except ImportError:
    _MOD = None
if hasattr(_MOD, "set_error_type"):
    _MOD.set_error_type(L.FvrError)

_ENTRIES = ("fvr_status_string", "fvr_pou_pinhole_forward", "fvr_pou_pinhole_backward_chunked",
            "fvr_pou_pinhole_backward_chunked_workspace", "fvr_pou_rays_forward", "fvr_pou_rays_backward",
            "fvr_pou_rays_backward_workspace", "fvr_tc_image", "fvr_tc_image_backward", "fvr_cncc_image",
            "fvr_cncc_image_workspace", "fvr_reg_loss_forward", "fvr_reg_loss_backward", "fvr_reg_loss_workspace")
_bound = None  # the loaded library the binding's addresses belong to


def module():
    """The bound module, or None where the Python nodes have to run."""
    global _bound
    if _MOD is None or profiling.active() or torch._C._functorch.peek_interpreter_stack() is not None:
        return None
    lib = L.load()
    if _bound is not lib:
        if not hasattr(_MOD, "bind"):  # built before these nodes existed
            return None
        _MOD.bind({n: ctypes.cast(getattr(lib, n), ctypes.c_void_p).value for n in _ENTRIES},
                  int(lib.fvr_pou_geo_stride()), int(lib.fvr_reg_loss_stats_count()))
        _bound = lib
    return _MOD


def tensor_keys(tensors):
    """(identity, versions) of tensors that a preparation is kept for: addresses,
    shapes, strides and types; versions, which a write in place advances
    (inference tensors have none).  In Python this takes 3.5 us for a lattice."""
    if _MOD is not None:
        return _MOD.tensor_keys(tensors)
    return (tuple((t.data_ptr(), t.shape, t.stride(), t.dtype) for t in tensors),
            tuple(0 if t.is_inference() else t._version for t in tensors))


def call(fn, launches, *args):
    """``fn(*args)``; ``launches``: kernels of the call.  A library status is an
    FvrError, in the backward too; torch's errors keep their types."""
    L.launch_count[0] += launches
    return fn(*args)
