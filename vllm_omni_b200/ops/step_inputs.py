"""Inputs of a decoder step in one launch each (csrc/step_inputs.cu): static tensors of a captured step, embedding rows with
rotation tables.  The PyTorch forms stay where the callers are (CPU, other types and layouts)."""
from __future__ import annotations

import ctypes

import torch

from . import _native as nv

c_int, c_long, c_void_p = ctypes.c_int, ctypes.c_long, ctypes.c_void_p
_JOBS = 16


class _Job(ctypes.Structure):
    _fields_ = [("src", c_void_p), ("dst", c_void_p), ("src_pitch", c_long), ("dst_pitch", c_long), ("src_bytes", c_int),
                ("dst_bytes", c_int), ("ordered", c_int), ("pad", c_int)]


class _Fill(ctypes.Structure):
    _fields_ = [("jobs", _Job * _JOBS), ("order", c_void_p), ("n_jobs", c_int), ("n", c_int), ("rows", c_int)]


class _Tokens(ctypes.Structure):
    _fields_ = [(n, c_void_p) for n in ("ids", "table", "given", "mask", "out", "pos", "freq", "axis", "cosv", "sinv")] + \
        [("axis_pitch", c_long), ("vocab", c_int), ("vecs", c_int), ("half", c_int)]


class StepFill:
    """Copies of ``n`` rows into static tensors of ``rows`` rows.  ``put`` queues one; ``run`` launches them all.  A source that the
    kernel does not take (another type, device, shape or a last dimension with gaps) makes ``put`` return False: the caller
    then fills by PyTorch operations."""

    def __init__(self, n: int, rows: int):
        self.a, self.n, self.rows, self.count, self.keep = _Fill(), n, rows, 0, []

    def put(self, dst: torch.Tensor, src: torch.Tensor | None, ordered: bool, pad_ones: bool = False, narrow: bool = False,
            pad_to: int | None = None) -> bool:
        """dst [rows] or [rows, c]; src the same with n rows and c columns, or with ``narrow`` fewer (the rest of a row is zeroed).  Rows past n repeat
        row 0 of src, or are -1 (``pad_ones``), or the int32 ``pad_to``, 0 or 1."""
        if self.count == _JOBS:
            return False
        j = self.a.jobs[self.count]
        size = dst.element_size()
        j.dst, j.dst_pitch, j.dst_bytes = dst.data_ptr(), dst.stride(0) * size, (dst.shape[1] if dst.dim() == 2 else 1) * size
        if src is None:
            j.src, j.src_pitch, j.src_bytes = None, 0, 0
        else:
            if src.dtype != dst.dtype or src.device != dst.device or src.dim() != dst.dim() or src.shape[0] != self.n \
                    or (src.dim() == 2 and (src.stride(1) != 1 or src.shape[1] > dst.shape[1] or (src.shape[1] < dst.shape[1] and not narrow))):
                return False
            j.src, j.src_pitch, j.src_bytes = src.data_ptr(), src.stride(0) * size, (src.shape[1] if src.dim() == 2 else 1) * size
            self.keep.append(src)
        assert pad_to is None or (pad_to in (0, 1) and dst.dtype == torch.int32)
        j.ordered, j.pad = int(ordered), 1 if pad_ones else {None: 0, 1: 2, 0: 3}[pad_to]
        self.count += 1
        return True

    def run(self, order: torch.Tensor) -> None:
        """``order`` int64 [n]: row i < n of an ordered destination takes the source's row order[i]."""
        self.a.order, self.a.n_jobs, self.a.n, self.a.rows = order.data_ptr(), self.count, self.n, self.rows
        nv.check_rc(nv.lib("step_inputs").omni_fill_step(ctypes.byref(self.a), nv.stream_ptr()), "omni_fill_step")


def token_rows(ids, table, positions, freq, axis=None, given=None, mask=None):
    """(x [T, D], cos, sin fp32 [T, half]): x[t] = given[t] where ``mask`` (everywhere without one), else table[ids[t]] with ids held
    inside the table; angles positions * freq in fp32, frequency i by the position on axis[i] of ``positions`` [axes, T] (or [T]).
    None when an operand is not of a form the kernel takes."""
    T, (vocab, D) = ids.numel(), table.shape
    if not table.is_cuda or any(t is not None and t.device != table.device for t in (ids, positions, freq, axis, given, mask)):
        return None
    if not (T and ids.dtype == positions.dtype == torch.int64 and ids.is_contiguous()
            and table.is_contiguous() and positions.stride(-1) == 1 and positions.shape[-1] == T and (axis is None) == (positions.dim() == 1)
            and D * table.element_size() % 16 == 0 and table.data_ptr() % 16 == 0):
        return None
    if given is not None and not (given.dtype == table.dtype and given.is_contiguous() and given.shape == (T, D) and given.data_ptr() % 16 == 0
                                  and (mask is None or (mask.dtype == torch.bool and mask.is_contiguous() and mask.numel() == T))):
        return None
    half = freq.numel()
    x = torch.empty(T, D, dtype=table.dtype, device=table.device)
    cos, sin = torch.empty(2, T, half, dtype=torch.float32, device=table.device)
    a, P = _Tokens(), lambda t: None if t is None else t.data_ptr()
    a.ids, a.table, a.given, a.mask, a.out, a.pos, a.freq, a.axis = P(ids), P(table), P(given), P(mask if given is not None else None), P(x), \
        P(positions), P(freq), P(axis)
    a.cosv, a.sinv, a.axis_pitch, a.vocab, a.vecs, a.half = P(cos), P(sin), positions.stride(0) if axis is not None else 0, vocab, \
        D * table.element_size() // 16, half
    nv.check_rc(nv.lib("step_inputs").omni_token_rows(ctypes.byref(a), c_long(T), nv.stream_ptr()), "omni_token_rows")
    return x, cos, sin
