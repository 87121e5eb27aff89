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
    ("b200exl3_expert_mapped", (BASE, F16, BASE, 8, None, None, BASE, 1, 128, 128, 1, 0, 4, 0, 1, 1, BASE + 2, None)),
])
def test_refused_before_a_launch(name, args):
    lib = _lib.load()
    assert getattr(lib, name)(*args) == -1
    assert b"aligned to their elements" in lib.b200exl3_last_error()
