"""Expert segments lie one after the other in the workspace: rows around the 64 a segment holds, batches whose plan does not
fit the grouped planner, ids past the bank, and the room the rows take."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import gpu  # noqa: F401
from tests.test_gpu_moe import check, make_bank, routes

pytestmark = pytest.mark.gpu


def counts_to_routes(rng, counts):
    """One slot per token, expert e chosen counts[e] times, tokens in random order."""
    selected = np.repeat(np.arange(len(counts), dtype=np.uint32), counts)
    return rng.permutation(selected)[:, None]


@pytest.mark.parametrize("counts", [[64, 64], [65, 1, 63], [1, 130, 0, 2], [0, 0, 35], [15, 16, 17, 33], [128, 0, 64, 129]])
def test_rows_around_a_segment(gpu, counts):
    rng = np.random.default_rng(sum(counts))
    n_in, hidden, k = 384, 128, 3
    bank = make_bank(rng, len(counts), n_in, hidden, k)
    moe = gpu.Exl3SwitchGlu(*bank, 1, k, 1, exact_weights=True)
    selected = counts_to_routes(rng, counts)
    x = rng.standard_normal((len(selected), n_in)).astype(np.float16)
    scores = rng.uniform(0.5, 1.0, selected.shape).astype(np.float32)
    got = moe.forward(x, selected, scores)
    check(got, oracle.switch_glu_forward(*bank, 1, k, 1, x, selected, scores), rms=3e-3)
    assert gpu.workspace_status(moe._workspace) == 0
    moe.close()


@pytest.mark.parametrize("experts,top_k,rows", [(1000, 2, 1000), (24, 8, 200)])
def test_sorted_rows_equal_one_row_per_slot(gpu, experts, top_k, rows):
    """1000 experts: the planner that walks the slots per expert; ids past the bank count as the last expert's."""
    rng = np.random.default_rng(experts)
    n_in, hidden, k = 128, 256, 2
    bank = make_bank(rng, experts, n_in, hidden, k)
    moe = gpu.Exl3SwitchGlu(*bank, top_k, k, 0, exact_weights=True)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    selected, scores = routes(rng, rows, experts, top_k)
    selected[::7, 0] = np.uint32(2 ** 31 + 5)
    got = moe.forward(x, selected, scores)
    assert np.array_equal(got.view(np.uint16), moe.forward(x, selected, scores).view(np.uint16))
    gpu.set_option("moe_sorted", 0)
    try:
        plain = moe.forward(x, selected, scores)
    finally:
        gpu.set_option("moe_sorted", 1)
    check(got, plain)
    assert gpu.workspace_status(moe._workspace) == 0
    moe.close()


@pytest.mark.parametrize("rows", [37, 256])
def test_workspace_holds_the_slots_and_no_padding(gpu, rows):
    rng = np.random.default_rng(rows)
    experts, top_k, n_in, hidden, k = 128, 8, 1024, 256, 1
    moe = gpu.Exl3SwitchGlu(*make_bank(rng, experts, n_in, hidden, k), top_k, k, 0)
    slots = rows * top_k
    per_slot = 2 * n_in * 2 + 2 * hidden * 4 + hidden * 2 + n_in * 4
    shared = 148 * 2 * 64 * 128 * 4                          # parts of items that CTAs share, two per CTA
    assert moe.workspace_bytes(rows) <= slots * (per_slot + 64) + shared + (1 << 16)
    moe.close()


@pytest.mark.parametrize("experts,top_k,rows", [(64, 8, 1), (128, 4, 9), (5, 1, 3)])
def test_sorted_form_with_few_slots(gpu, experts, top_k, rows):
    """The sorted form is taken from far fewer than a row per expert on: experts without rows, segments of one row."""
    rng = np.random.default_rng(experts + rows)
    n_in, hidden, k = 256, 384, 3
    bank = make_bank(rng, experts, n_in, hidden, k)
    moe = gpu.Exl3SwitchGlu(*bank, top_k, k, 0, exact_weights=True)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    selected, scores = routes(rng, rows, experts, top_k)
    gpu.set_option("moe_sorted", 2)
    try:
        got = moe.forward(x, selected, scores)
    finally:
        gpu.set_option("moe_sorted", 1)
    check(got, oracle.switch_glu_forward(*bank, top_k, k, 0, x, selected, scores), rms=3e-3)
    assert gpu.workspace_status(moe._workspace) == 0
    moe.close()


@pytest.mark.parametrize("experts,top_k,n_in,hidden", [(128, 8, 512, 256), (8, 2, 256, 640), (300, 1, 128, 128)])
def test_a_workspace_covers_smaller_batches(gpu, experts, top_k, n_in, hidden):
    """Made for the largest batch, used for any: below the sizes where the forms change, and where a pass ends."""
    from mlxl3_b200 import ep
    from mlxl3_b200.runtime import DeviceBuffer, Stream
    rng = np.random.default_rng(experts)
    bank = make_bank(rng, experts, n_in, hidden, 2)
    moe = gpu.Exl3SwitchGlu(*bank, top_k, 2, 0)
    sizes = [moe.workspace_bytes(r) for r in range(1, 700)]
    assert all(a <= b for a, b in zip(sizes, sizes[1:]))
    most = 400
    selected, scores = routes(rng, most, experts, top_k)
    stream, ws = Stream(), gpu.new_workspace(moe.workspace_bytes(most))
    d_x, d_y = DeviceBuffer.from_numpy(rng.standard_normal((most, n_in)).astype(np.float16)), DeviceBuffer(most * n_in * 2)
    d_sel, d_scores = DeviceBuffer.from_numpy(selected), DeviceBuffer.from_numpy(scores)
    for rows in (400, 257, 256, 255, 128, 65, 37, 33, 32, 31, 16, 9, 4, 3, 2, 1):
        moe.forward_device(d_x.ptr, gpu.F16, rows, d_sel.ptr, d_scores.ptr, gpu.F16, d_y.ptr, ws, stream)
    stream.sync()
    assert gpu.workspace_status(ws) == 0
    ctx = ep.EpContext(0, 1, 256, n_in, lambda raw: [raw])
    sharded = ep.Exl3SwitchGluEp(*bank, top_k, 2, 0, ctx)
    sizes = [sharded.workspace_bytes(r) for r in range(1, 300)]
    assert all(a <= b for a, b in zip(sizes, sizes[1:]))
    ws = gpu.new_workspace(sharded.workspace_bytes(256))
    for rows in (256, 200, 31, 30, 7, 1):
        sharded.forward_device(d_x.ptr, gpu.F16, rows, d_sel.ptr, d_scores.ptr, gpu.F16, d_y.ptr, ws, stream)
    stream.sync()
    assert ctx.status() == 0 and gpu.workspace_status(ws) == 0
    sharded.close(), ctx.close(), moe.close()
