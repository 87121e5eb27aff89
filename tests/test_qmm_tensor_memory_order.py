"""The many-row kernel passes tensor memory between threads through barriers (no GPU needed: its source is read).  A wait
orders a later tcgen05 instruction of the waiting thread only together with ``tcgen05.fence::after_thread_sync``, so in the
kernel's text such a fence has to lie between a wait and the next instruction that touches tensor memory."""
import re

from tests.conftest import ROOT

WAIT = ("qmm_wait(", "mbar_test_wait(", "__syncthreads(")
FENCE = "tcgen05.fence::after_thread_sync"
USE = ("tmem_st_tile<", "tmem_ld16(", "umma_f16_ts(", "tmem_dealloc(")


def kernel_body():
    text = (ROOT / "mlxl3_b200" / "csrc" / "kernels_qmm.cu").read_text()
    at = text.index("qmm_kernel(const __grid_constant__")
    end = text.index("\n}\n", at)
    return re.sub(r"//[^\n]*", "", text[at:end])


def unordered(body):
    """The uses of tensor memory that follow a wait with no fence in between."""
    tokens = re.finditer("|".join(re.escape(t) for t in (*WAIT, FENCE, *USE)), body)
    ordered, out = True, []
    for m in tokens:
        if m.group() == FENCE:
            ordered = True
        elif m.group() in WAIT:
            ordered = False
        elif not ordered:
            out.append(body[m.start():m.start() + 60])
    return out


def test_a_fence_lies_between_a_wait_and_tensor_memory():
    body = kernel_body()
    assert all(t in body for t in (*USE, FENCE, "qmm_wait("))
    assert unordered(body) == []


def test_the_check_sees_a_missing_fence():
    body = kernel_body()
    without = body.replace(FENCE, "removed")
    assert len(unordered(without)) >= 4
