"""A recurrent mixer enqueued by one call into the library.

``GatedDeltaRule.forward_into`` and ``MatrixMemory.forward_into`` run their products, convolution and recurrence one after the other,
each a call into a library with checks, slices and allocations around it: about 110 us of host time, twice what the kernels of a
decode step take.  In bfloat16 ``NativeMixer`` hands the whole mixer to ``coheryn_recurrent_mixer_bf16`` (csrc/mixer_runner.cu), which
makes the same choices of kernels from the same thresholds and calls the same entry points.  Anything that it does not cover takes
the parts' own path: ``run`` returns False, with nothing launched.
"""
from __future__ import annotations

import ctypes
from ctypes import c_float, c_int, c_long, c_void_p
from typing import Optional

import torch

from .. import ops
from .native_block import block_tuning

P = c_void_p
UNSUPPORTED, RECURRENT_FAILED = 3, 2

# Mixers enqueued through the library since the module was loaded (tests look at it).
runs = 0


class CoMixerLayer(ctypes.Structure):
    _fields_ = [(n, P) for n in ("w_in", "w_second", "w_o", "conv_w", "bias_a", "bias_b", "norm_w", "conv", "delta", "memory",
                                 "chunk_floats", "chunks_pay")] + \
               [(n, c_float) for n in ("eps", "out_scale", "cap")] + \
               [(n, c_int) for n in ("memory_kind", "width", "columns", "heads", "kv_heads", "dk", "dv", "taps", "decay_channels", "gate_act",
                                     "in_chunks", "chunk_from", "chunk_tokens", "at_q", "at_k", "at_v", "at_g", "at_a", "at_b", "second_n",
                                     "second_k", "second_rows", "second_columns", "conv_dtype", "bias_a_dtype", "bias_b_dtype", "norm_dtype")]


class CoMixerStep(ctypes.Structure):
    _fields_ = [(n, P) for n in ("token_req", "cu_q", "state_slots", "tc_status", "stream")] + [("T", c_int), ("B", c_int), ("q_lens", P)]


_entry = None


def _entry_point():
    global _entry
    if _entry is None:
        fn = ops.core().coheryn_recurrent_mixer_bf16
        fn.argtypes = [P, P, P, P, c_long, P, c_long, P, c_long, P, P, c_long, c_int, P]
        fn.restype = c_int
        _entry = fn
    return _entry


def _i32(device, *sized) -> bool:
    """Whether every (tensor, entries it must have) is a contiguous int32 tensor on ``device``."""
    return all(t is not None and t.dtype == torch.int32 and t.device == device and t.is_contiguous() and t.numel() >= n for t, n in sized)


def shapes_fit(specs, tensors) -> bool:
    """Whether every tensor has the shape that its specification names (-1: any size).  The library takes sizes from the part's
    description alone, so a tensor of another size must not reach it."""
    return all(t.dim() == len(specs[n].shape) and all(want in (-1, got) for want, got in zip(specs[n].shape, t.shape))
               for n, t in tensors.items() if n in specs)


class NativeMixer:
    """``fields``: what ``CoMixerLayer`` holds beside the pointers; ``tensors``: its tensors by field (kept alive here);
    ``state_width``: floats of a request's state."""

    def __init__(self, fields: dict, tensors: dict, memory: bool, state_width: int):
        lib = ops.recurrent()
        fn = lambda f: ctypes.cast(f, c_void_p).value
        code = lambda t: ops._code(t) if t is not None else ops.F32
        pointers = {n: t.data_ptr() if t is not None else None for n, t in tensors.items()}
        self.layer = CoMixerLayer(**fields, **pointers, memory_kind=1 if memory else 0, conv=fn(lib.coheryn_short_conv_silu),
                                  delta=fn(lib.coheryn_gated_delta_scan), memory=fn(lib.coheryn_matrix_memory_scan),
                                  chunk_floats=fn(lib.coheryn_memory_chunk_floats if memory else lib.coheryn_delta_chunk_floats),
                                  chunks_pay=fn(lib.coheryn_memory_chunks_pay if memory else lib.coheryn_delta_chunks_pay),
                                  chunk_from=lib.chunk_from, chunk_tokens=lib.chunk_tokens, conv_dtype=code(tensors.get("conv_w")),
                                  bias_a_dtype=code(tensors["bias_a"]), bias_b_dtype=code(tensors["bias_b"]), norm_dtype=code(tensors["norm_w"]))
        self.tensors, self.lib, self.device, self.state_width = tensors, lib, tensors["w_in"].device, state_width
        self.layer_ref = ctypes.addressof(self.layer)

    @classmethod
    def build(cls, fields: dict, tensors: dict, memory: bool, state_width: int) -> Optional["NativeMixer"]:
        """None when a tensor is not as the library's sequence takes it (its shapes are the caller's to check: ``shapes_fit``)."""
        if len({t.device for t in tensors.values() if t is not None}) != 1:
            return None
        matrices = [tensors[n] for n in ("w_in", "w_second", "w_o") if tensors.get(n) is not None]
        if any(not t.is_cuda or t.dtype != torch.bfloat16 or not t.is_contiguous() for t in matrices):
            return None
        vectors = [tensors[n] for n in ("conv_w", "bias_a", "bias_b", "norm_w") if tensors.get(n) is not None]
        if any(not t.is_cuda or t.dtype not in (torch.bfloat16, torch.float32) or not t.is_contiguous() for t in vectors):
            return None
        return cls(fields, tensors, memory, state_width)

    def run(self, x: torch.Tensor, step, state: torch.Tensor, opened: Optional[torch.Tensor], out: Optional[torch.Tensor]) -> bool:
        """The mixer on ``x``, continued from and left in ``state``: the activations in front of the output product into ``opened``
        (bfloat16) and / or the output into ``out`` (float32 [T, width]).  Everything is compared with the part's sizes first; what does
        not fit is left to the part's own path, whose operations check it again and raise."""
        L, T, B = self.layer, x.shape[0], step.num_requests
        width = L.heads * L.dv
        if x.dtype != torch.bfloat16 or x.device != self.device or x.dim() != 2 or x.shape[1] != L.width or x.stride(1) != 1:
            return False
        if (state.dtype != torch.float32 or state.device != self.device or state.dim() != 2 or state.shape[1] != self.state_width
                or state.stride(1) != 1):
            return False
        if not _i32(self.device, (getattr(step, "token_req", None), T), (step.cu_q, B + 1), (step.state_slots, B)):
            return False
        if opened is not None and (opened.dtype != torch.bfloat16 or opened.device != self.device or opened.shape != (T, width) or opened.stride(1) != 1):
            return False
        if out is not None and (out.dtype != torch.float32 or out.device != self.device or out.shape != (T, L.width) or not out.is_contiguous()):
            return False
        lens = None
        if L.in_chunks and T - B + 1 >= L.chunk_from:      # (else no run is as long)
            got = getattr(step, "q_lens", None)
            if got is not None and len(got) == B:
                lens = (c_int * B)(*got)
        described = CoMixerStep(step.token_req.data_ptr(), step.cu_q.data_ptr(), step.state_slots.data_ptr(), ops.tc_status(x.device).data_ptr(),
                                ops._stream().value or 0, T, B, ctypes.addressof(lens) if lens is not None else None)
        tuning, needed, call = block_tuning(), c_long(0), _entry_point()
        args = (self.layer_ref, ctypes.addressof(described), ctypes.addressof(tuning), x.data_ptr(), x.stride(0), state.data_ptr(), state.stride(0),
                opened.data_ptr() if opened is not None else None, opened.stride(0) if opened is not None else 0,
                out.data_ptr() if out is not None else None)
        needed_ref = ctypes.addressof(needed)
        rc = call(*args, None, 0, 1, needed_ref)
        if rc == UNSUPPORTED:
            return False
        if not rc:
            scratch = torch.empty(needed.value + 256, dtype=torch.uint8, device=x.device)
            at = scratch.data_ptr()
            rc = call(*args, at + -at % 256, needed.value, 0, needed_ref)
        if rc:
            raise ops.KernelError((self.lib if rc == RECURRENT_FAILED else ops.core()).coheryn_last_error().decode("utf-8", "replace"))
        global runs
        runs += 1
        return True
