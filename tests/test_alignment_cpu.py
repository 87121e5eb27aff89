"""Pointers that no element can start at are refused before anything is launched (no GPU needed)."""
import pytest

from mlxl3_b200 import _lib

F16, F32 = 9, 10
BASE = 1 << 20                                       # stands for a device address; nothing may look behind it


@pytest.mark.parametrize("name,args", [
    ("b200exl3_prepare", (BASE + 1, F16, BASE, 1, 1, 128, BASE, None)),
    ("b200exl3_prepare", (BASE + 2, F32, BASE, 1, 1, 128, BASE, None)),
    ("b200exl3_prepare", (BASE, F16, BASE + 1, 1, 1, 128, BASE, None)),
    ("b200exl3_finish", (BASE, 1, BASE + 1, 1, None, 1, 128, F16, BASE, None)),
    ("b200exl3_finish", (BASE, 1, BASE, 1, BASE + 1, 1, 128, F16, BASE, None)),
    ("b200exl3_finish", (BASE, 1, BASE, 1, None, 1, 128, F32, BASE + 2, None)),
    ("b200exl3_expert_mapped", (BASE + 1, F16, BASE, 8, BASE, BASE, BASE, 1, 128, 128, 1, 0, 4, 0, 0, 0, BASE, None)),
    ("b200exl3_expert_mapped", (BASE, F16, BASE, 8, BASE, BASE, BASE + 2, 1, 128, 128, 1, 0, 4, 0, 0, 0, BASE, None)),
    ("b200exl3_expert_mapped", (BASE, F16, BASE, 8, None, None, BASE, 1, 128, 128, 1, 0, 4, 0, 1, 1, BASE + 1, None)),
])
def test_refused_before_a_launch(name, args):
    lib = _lib.load()
    assert getattr(lib, name)(*args) == -1
    assert b"aligned to their elements" in lib.b200exl3_last_error()


@pytest.mark.parametrize("name,args,bytes_", [
    ("b200exl3_rms_norm", (BASE + 2, None, BASE, 1, 128, 1e-5, None, BASE, None), 4),
    ("b200exl3_rms_norm", (BASE, BASE + 2, BASE, 1, 128, 1e-5, None, BASE, None), 4),
    ("b200exl3_rms_norm", (BASE, None, BASE, 1, 128, 1e-5, BASE + 2, BASE, None), 4),
    ("b200exl3_swiglu", (BASE, BASE + 2, 128, BASE, None), 4),
    ("b200exl3_rope_append", (BASE, BASE, BASE + 2, 1, 1, 128, BASE, 1e4, 8, BASE, BASE, None), 4),
    ("b200exl3_rope_append", (BASE, BASE, BASE, 1, 1, 128, BASE + 2, 1e4, 8, BASE, BASE, None), 4),
    ("b200exl3_attention_decode", (BASE, BASE, BASE, 1, 1, 128, BASE, 8, 1.0, BASE + 4, BASE, 1 << 30, None), 8),
    ("b200exl3_head_argmax", (BASE, BASE, 128, 128, 0, None, BASE, BASE + 4, BASE, 1 << 30, None), 8),
    ("b200exl3_embed", (BASE, BASE + 2, 1, 128, 128, BASE, None), 4),
    ("b200exl3_finish_and_reduce", (BASE, BASE + 4, BASE, 1, BASE, F16, 1, 1, 128, BASE, None), 8),
    ("b200exl3_finish_and_reduce", (BASE, BASE, BASE + 2, 1, BASE, F16, 1, 1, 128, BASE, None), 4),
    ("b200exl3_swiglu_down_input", (BASE, BASE + 1, BASE, BASE, 1, 1, 128, BASE, None), 2),
    ("b200exl3_router_topk", (BASE + 2, F32, 1, 8, 2, 1, BASE, BASE, None), 4),
    ("b200exl3_router_softmax_topk", (BASE, F16, 1, 8, 2, 1, BASE + 2, BASE, None, None), 4),
    ("b200exl3_router_gate", (BASE, F16, BASE + 2, 1, 128, 8, BASE, None), 4),
    ("b200exl3_expert_mapped", (BASE, F16, BASE + 2, 8, BASE, BASE, BASE, 1, 128, 128, 1, 0, 4, 0, 0, 0, BASE, None), 4),
    ("b200exl3_expert_mapped", (BASE, F16, BASE, 8, None, None, BASE, 1, 128, 128, 1, 0, 4, 0, 1, 1, BASE + 8, None), 16),
    ("b200exl3_unpack_states", (BASE + 1, 1, 4, 0, BASE, None, None), 2),
    ("b200exl3_unpack_states", (BASE + 2, 1, 4, 0, BASE, None, None), 4),
    ("b200exl3_codebook", (None, 8, 0, BASE + 1, None), 2),
])
def test_what_a_kernel_reads_several_at_a_time_lies_on_that_many_bytes(name, args, bytes_):
    lib = _lib.load()
    assert getattr(lib, name)(*args) == -1
    assert b"device pointers must be %d-byte aligned" % bytes_ in lib.b200exl3_last_error()
