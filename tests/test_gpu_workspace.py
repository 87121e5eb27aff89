"""What a workspace holds: the rows, parts and sums that some kernel of the call touches, and no more."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import gpu, random_layer  # noqa: F401
from tests.test_plan_invariants import query

pytestmark = pytest.mark.gpu

HEADER, SLACK = 16384, 4096                      # arrival counters; the areas are rounded to 256 bytes
SHARD_SUMS = 32 << 20                            # a row shard keeps this many bytes of fp32 sums at a time (at least 256 rows)


def rows_and_parts(n_in, n_out, k, rows, members=1):
    """Bytes of the rotated rows of a pass and of the parts of shared items."""
    pass_rows, part_bytes = query("qmm", n_in, n_out, k, rows)[6:]
    return HEADER + members * min(rows, pass_rows) * n_in * 2 + part_bytes + SLACK


@pytest.mark.parametrize("rows", [64, 2048])
def test_no_room_for_sums_that_nobody_stores(gpu, rows):
    rng = np.random.default_rng(rows)
    n_in, n_out, k = 256, 8192, 2
    layers = [gpu.Exl3Linear(*random_layer(rng, n_in, n_out, k), None, k, 0) for _ in range(2)]
    group = gpu.Exl3Group(layers)
    few_rows = HEADER + 2 * rows * n_in * 2 + 128 * 16 * 512 * 4 + SLACK      # the few-row kernel's parts, 16 rows of a launch
    assert group.workspace_bytes(rows) <= max(rows_and_parts(n_in, 2 * n_out, k, rows, 2), few_rows)
    shard = min(rows * n_out * 4, max(SHARD_SUMS, 256 * n_out * 4))
    assert layers[0].workspace_bytes(rows) <= rows_and_parts(n_in, n_out, k, rows) + shard
    group.close()


def test_a_row_shard_of_more_rows_than_one_pass(gpu):
    """1100 rows of 8192 outputs: sums of 1024 rows fit, the rest follows in a second pass of the same call."""
    from mlxl3_b200.runtime import DeviceBuffer, Stream
    from mlxl3_b200.tp import TpContext
    rng = np.random.default_rng(11)
    n_in, n_out, k, rows = 256, 8192, 3, 1100
    trellis, suh, svh = random_layer(rng, n_in, n_out, k)
    layer = gpu.Exl3Linear(trellis, suh, svh, None, k, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    stream = Stream()
    ctx = TpContext(0, 1, rows * n_out // 128, lambda raw: [raw])
    d_x, d_y = DeviceBuffer.from_numpy(x), DeviceBuffer(rows * n_out * 2)
    ws = gpu.new_workspace(layer.workspace_bytes(rows))
    pick = np.array([0, 500, 1023, 1024, 1025, 1099])
    want = oracle.linear_forward(trellis, k, 0, suh, svh, None, x[pick]).astype(np.float32)
    for _ in range(3):                                   # both slots of every unit get used
        d_y.fill(0, stream)
        ctx.forward(layer, d_x.ptr, gpu.F16, rows, d_y.ptr, ws, stream)
        got = d_y.download((rows, n_out), np.float16, stream)[pick].astype(np.float32)
        assert (np.abs(got - want) <= 1e-2 * np.abs(want).max(axis=1, keepdims=True)).all()
    assert gpu.workspace_status(ws) == 0 and ctx.status() == 0
    ctx.close()
    layer.close()
