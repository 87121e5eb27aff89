"""Which form the expert block takes (no GPU needed): of measured calls the form that the rule takes is the faster one, or close to
it where the two are level.  The times are those of profiles/expert_block_slots_or_sorted.md, us per call: one row per slot, sorted."""
import ctypes

import pytest

from mlxl3_b200 import _lib


def query(experts, n_in, hidden, top_k, k, rows):
    out = (ctypes.c_int64 * 4)()
    _lib.call("b200exl3_moe_plan_query", experts, n_in, hidden, top_k, k, rows, out, 4)
    return list(out)


MEASURED = [
    # experts, top-k, in, hidden, bits, tokens, one row per slot, sorted
    (8, 1, 4096, 14336, 4, 1, 89.6, 68.2), (8, 2, 4096, 14336, 3, 1, 127.6, 114.8), (8, 2, 4096, 14336, 4, 8, 729.7, 320.2),
    (32, 8, 7168, 2048, 4, 1, 98.2, 111.6), (32, 8, 7168, 2048, 3, 1, 106.8, 119.2), (32, 8, 7168, 2048, 4, 3, 242.3, 183.4),
    (8, 2, 4096, 2048, 4, 2, 31.8, 46.9), (8, 2, 4096, 2048, 4, 8, 104.0, 64.9), (8, 2, 4096, 2048, 2, 1, 24.8, 41.4),
    (64, 6, 2048, 1408, 4, 2, 43.9, 54.4), (64, 6, 2048, 1408, 4, 5, 77.8, 84.7), (64, 6, 2048, 1408, 4, 8, 109.9, 99.5),
    (64, 6, 2048, 1408, 8, 5, 79.8, 91.5), (64, 6, 2048, 1408, 2, 5, 75.5, 86.6), (64, 6, 2048, 1408, 6, 10, 153.2, 129.9),
    (128, 8, 2048, 768, 3, 1, 23.6, 42.3), (128, 8, 2048, 768, 3, 7, 85.3, 94.9), (128, 8, 2048, 768, 3, 16, 165.4, 133.5),
    (128, 8, 2048, 768, 1, 7, 76.6, 90.9), (128, 8, 2048, 768, 4, 7, 79.2, 89.2), (128, 8, 2048, 768, 6, 12, 136.6, 129.2),
    (128, 1, 2048, 768, 3, 32, 56.4, 61.0), (128, 1, 2048, 768, 3, 128, 163.5, 129.8), (32, 4, 1024, 256, 3, 16, 32.9, 40.1),
    (32, 4, 1024, 256, 3, 48, 57.0, 40.9), (8, 1, 512, 256, 4, 64, 25.1, 30.0), (8, 1, 512, 256, 4, 300, 65.3, 32.6),
    (60, 1, 1024, 512, 2, 48, 36.5, 44.4), (60, 1, 1024, 512, 2, 140, 67.1, 52.9), (32, 2, 3072, 1024, 4, 4, 31.7, 47.7),
    (8, 2, 14336, 512, 3, 8, 103.3, 74.2), (16, 1, 512, 2048, 6, 64, 71.5, 45.9), (60, 4, 1408, 1024, 5, 8, 55.4, 62.1),
]


@pytest.mark.parametrize("experts,top_k,n_in,hidden,k,tokens,slots_us,sorted_us", MEASURED)
def test_the_faster_form(experts, top_k, n_in, hidden, k, tokens, slots_us, sorted_us):
    is_sorted, _, one_per_slot, by_expert = query(experts, n_in, hidden, top_k, k, tokens)
    assert (sorted_us if is_sorted else slots_us) <= 1.03 * min(slots_us, sorted_us)
    assert is_sorted == (by_expert < one_per_slot)


def test_passes_and_refused_shapes():
    assert query(128, 2048, 768, 8, 3, 4096)[:2] == [1, 2048]                 # 16384 slots a pass, equal passes
    assert query(65536, 128, 128, 1, 4, 4096)[0] == 0                         # the route plan's ids are 16 bits wide
    lib, out = _lib.load(), (ctypes.c_int64 * 4)()
    for args in ((0, 128, 128, 1, 4, 1), (4, 100, 128, 1, 4, 1), (4, 128, 128, 5, 4, 1), (4, 128, 128, 1, 7, 1), (4, 128, 128, 1, 4, 0)):
        assert lib.b200exl3_moe_plan_query(*args, out, 4) == -1 and b"invalid plan query" in lib.b200exl3_last_error()
    assert lib.b200exl3_moe_plan_query(4, 128, 128, 1, 4, 1, out, 3) == -1
