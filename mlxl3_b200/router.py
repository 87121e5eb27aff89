"""Stable MoE top-k (``router::topk``, native/src/router.rs:37-120) over the C ABI."""
from __future__ import annotations

from ctypes import c_void_p

import numpy as np

from . import _lib
from ._lib import B200Exl3Error, F16, F32
from .runtime import DEFAULT_STREAM, Scratch, Stream


def topk_device(d_values: int, dtype: int, rows: int, experts: int, top_k: int, normalize: bool, d_indices: int,
                d_scores: int, stream: Stream = DEFAULT_STREAM) -> None:
    _lib.call("b200exl3_router_topk", c_void_p(d_values), dtype, rows, experts, top_k, int(normalize), c_void_p(d_indices),
              c_void_p(d_scores), c_void_p(stream.handle))


def topk(values: np.ndarray, top_k: int, normalize: bool, stream: Stream = DEFAULT_STREAM):
    """``values [rows, experts]`` (float16 or float32) -> ``(indices [rows, top_k] uint32, scores [rows, top_k])``:
    per row the ``top_k`` largest values in ascending order, ties to the higher index; with ``normalize`` the
    scores are divided by their sum (added in slot order in the values' dtype)."""
    values = np.asarray(values)
    if values.ndim != 2:
        raise B200Exl3Error("router values must have rank 2")
    if values.dtype not in (np.float16, np.float32):
        raise B200Exl3Error("native router expects FP16 or FP32 values")
    rows, experts = values.shape
    slots = max(rows * top_k, 1)
    at_v, at_i, at_s, end = Scratch.offsets(values.nbytes, slots * 4, slots * values.dtype.itemsize)
    with Scratch(end, stream) as s:
        s.upload(values, at_v)
        topk_device(s.ptr + at_v, F16 if values.dtype == np.float16 else F32, rows, experts, top_k, normalize, s.ptr + at_i, s.ptr + at_s, stream)
        return s.download((rows, top_k), np.uint32, at_i), s.download((rows, top_k), values.dtype, at_s)


def softmax_topk(logits: np.ndarray, top_k: int, normalize: bool = True, stream: Stream = DEFAULT_STREAM):
    """``router::topk(&logits.softmax_precise(), top_k, normalize)`` (native/src/qwen35.rs:214): returns
    ``(indices, scores, probabilities)``; the softmax runs in fp32 and is rounded to the logits' dtype."""
    logits = np.asarray(logits)
    if logits.ndim != 2:
        raise B200Exl3Error("router values must have rank 2")
    if logits.dtype not in (np.float16, np.float32):
        raise B200Exl3Error("native router expects FP16 or FP32 values")
    rows, experts = logits.shape
    slots = max(rows * top_k, 1)
    at_l, at_i, at_s, at_p, end = Scratch.offsets(logits.nbytes, slots * 4, slots * logits.dtype.itemsize, logits.nbytes)
    with Scratch(end, stream) as s:
        s.upload(logits, at_l)
        _lib.call("b200exl3_router_softmax_topk", s.ptr + at_l, F16 if logits.dtype == np.float16 else F32, rows, experts, top_k,
                  int(normalize), s.ptr + at_i, s.ptr + at_s, s.ptr + at_p, stream.handle)
        return (s.download((rows, top_k), np.uint32, at_i), s.download((rows, top_k), logits.dtype, at_s),
                s.download((rows, experts), logits.dtype, at_p))


def gate(x: np.ndarray, weight: np.ndarray, stream: Stream = DEFAULT_STREAM) -> np.ndarray:
    """fp16 router logits ``x [rows, in] @ weight [experts, in].T`` with fp32 accumulation."""
    x, weight = np.ascontiguousarray(x, np.float16), np.ascontiguousarray(weight, np.float16)
    if x.ndim != 2 or weight.ndim != 2 or x.shape[1] != weight.shape[1]:
        raise B200Exl3Error("invalid router gate dimensions")
    rows, n_in = x.shape
    experts = weight.shape[0]
    at_x, at_w, at_l, end = Scratch.offsets(x.nbytes, weight.nbytes, rows * experts * 2)
    with Scratch(end, stream) as s:
        s.upload(x, at_x)
        s.upload(weight, at_w)
        _lib.call("b200exl3_router_gate", s.ptr + at_x, F16, s.ptr + at_w, rows, n_in, experts, s.ptr + at_l, stream.handle)
        return s.download((rows, experts), np.float16, at_l)
