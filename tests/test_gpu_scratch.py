"""The pool behind calls with host arrays (b200exl3_scratch_*)."""
from ctypes import byref, c_void_p

import pytest

from mlxl3_b200 import _lib
from tests.gpu_util import gpu  # noqa: F401

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def acquire(nbytes):
    p, host = c_void_p(), c_void_p()
    _lib.call("b200exl3_scratch_acquire", nbytes, byref(p), byref(host))
    return p.value, host.value


def release(ptr):
    _lib.call("b200exl3_scratch_release", ptr)


def free_bytes():
    import torch
    return torch.cuda.mem_get_info(0)[0]


@pytest.mark.parametrize("mib", [65, 300, 1100])
def test_a_block_too_large_to_keep_is_as_large_as_asked(gpu, mib):
    before = free_bytes()
    ptr, host = acquire(mib * MIB + 1)
    taken = before - free_bytes()
    release(ptr)
    assert host is None and mib * MIB < taken <= (mib + 8) * MIB      # the driver hands out steps of 2 MiB
    assert before - free_bytes() <= 2 * MIB                           # and it is given back


def test_a_new_size_finds_a_kept_block(gpu):
    """What a call of one size left serves the first call of another: nothing is allocated or page-locked again."""
    first, first_host = acquire(300)
    release(first)
    assert first_host
    for nbytes in (1, 4096, 70_000, MIB // 2 + 1, MIB):
        ptr, host = acquire(nbytes)
        release(ptr)
        assert (ptr, host) == (first, first_host)
    release(acquire(9 * MIB)[0])
    for nbytes in (5 * MIB, 2 * MIB + 1, 16 * MIB):
        before = free_bytes()
        ptr, host = acquire(nbytes)
        assert host is None and free_bytes() == before
        release(ptr)


def test_blocks_in_use_are_never_handed_out_twice(gpu):
    held = [acquire(n)[0] for n in (100, 100, MIB, MIB + 1, 3 * MIB)]
    assert len(set(held)) == len(held)
    for ptr in held:
        release(ptr)
    with pytest.raises(gpu.B200Exl3Error, match="not a scratch block"):
        release(held[0])


def test_a_kept_large_block_does_not_push_small_ones_out(gpu):
    """64 MiB kept, then a small call: the large block makes room, the small one is there for the next call."""
    small = acquire(300)[0]
    before = free_bytes()
    large = acquire(60 * MIB)[0]
    release(large)
    release(small)
    assert before - free_bytes() < 32 * MIB
    again = acquire(300)[0]
    release(again)
    assert again == small
