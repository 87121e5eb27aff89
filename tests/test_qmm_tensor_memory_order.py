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


# instructions that all lanes of a warp execute as one (.sync.aligned), and what lets lanes go ways of their own before them
ALIGNED = ("tmem_alloc(", "tmem_st_tile<", "tcgen05.wait::st.sync.aligned", "tmem_ld16(", "tmem_dealloc(")
TOGETHER = ("__syncwarp(", "group_sync(")
APART = ("qmm_wait(", "if (lane", "lane == 0) {", "threadIdx.x == 0) {", "elect_one()", "while (global_ns()")


def not_converged(body):
    tokens = re.finditer("|".join(re.escape(t) for t in (*ALIGNED, *TOGETHER, *APART)), body)
    together, out = True, []
    for m in tokens:
        if m.group() in TOGETHER:
            together = True
        elif m.group() in APART:
            together = False
        elif not together:
            out.append(body[m.start():m.start() + 60])
    return out


def test_a_warp_barrier_lies_before_every_warp_wide_instruction():
    body = kernel_body()
    assert all(t in body for t in (*ALIGNED, *TOGETHER, *APART))
    assert not_converged(body) == []
    assert len(not_converged(body.replace("__syncwarp(", "removed(").replace("group_sync(", "removed("))) >= 4
