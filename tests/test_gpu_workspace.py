"""What a workspace holds: the rows, parts and sums that some kernel of the call touches, and no more."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import gpu, random_layer  # noqa: F401
from tests.test_plan_invariants import query

pytestmark = pytest.mark.gpu

HEADER, SLACK = 16384, 4096                      # arrival counters; the areas are rounded to 256 bytes
SHARD_SUMS = 32 << 20                            # a row shard keeps this many bytes of fp32 sums at a time (at least 256 rows)


def rows_and_parts(n_in, n_out, k, rows, members=1, shard=False):
    """Bytes of the rotated rows of a pass and of the parts of shared items, of a row shard also of its sums: the most that a
    batch of up to `rows` rows takes, because a workspace covers the smaller batches too."""
    def need(r):
        pass_rows, part_bytes = query("qmm", n_in, n_out, k, r)[6:]
        return members * min(r, pass_rows) * n_in * 2 + part_bytes + shard * min(r * n_out * 4, max(SHARD_SUMS, 256 * n_out * 4))
    return HEADER + SLACK + max(need(r) for r in range(9, rows + 1))


@pytest.mark.parametrize("rows", [64, 2048])
def test_no_room_for_sums_that_nobody_stores(gpu, rows):
    rng = np.random.default_rng(rows)
    n_in, n_out, k = 256, 8192, 2
    layers = [gpu.Exl3Linear(*random_layer(rng, n_in, n_out, k), None, k, 0) for _ in range(2)]
    group = gpu.Exl3Group(layers)
    few_rows = HEADER + 2 * rows * n_in * 2 + 128 * 16 * 512 * 4 + SLACK      # the few-row kernel's parts, 16 rows of a launch
    assert group.workspace_bytes(rows) <= max(rows_and_parts(n_in, 2 * n_out, k, rows, 2), few_rows)
    assert layers[0].workspace_bytes(rows) <= rows_and_parts(n_in, n_out, k, rows, shard=True)
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


@pytest.mark.parametrize("n_in,n_out,k,members", [(14336, 4096, 1, 1), (4096, 3072, 2, 2), (256, 8192, 2, 1), (128, 128, 4, 1)])
def test_a_workspace_covers_smaller_batches(gpu, n_in, n_out, k, members):
    """Made for the largest batch, used for any: 1024 rows of 14336 -> 4096 leave fewer parts than 768."""
    from mlxl3_b200.runtime import DeviceBuffer, Stream
    rng = np.random.default_rng(n_in)
    layers = [gpu.Exl3Linear(*random_layer(rng, n_in, n_out, k), None, k, 0) for _ in range(members)]
    op = gpu.Exl3Group(layers) if members > 1 else layers[0]
    sizes = [op.workspace_bytes(r) for r in range(1, 1100)]
    assert all(a <= b for a, b in zip(sizes, sizes[1:]))
    stream, ws = Stream(), gpu.new_workspace(op.workspace_bytes(1024))
    d_x, d_ys = DeviceBuffer(1024 * n_in * 2), [DeviceBuffer(1024 * n_out * 2) for _ in range(members)]
    d_x.fill(0, stream)
    for rows in (1024, 896, 768, 640, 576, 300, 150, 40, 16, 15, 9, 8, 3, 1):
        ys = [y.ptr for y in d_ys]
        op.forward_device(d_x.ptr, gpu.F16, rows, ys if members > 1 else ys[0], ws, stream)
    stream.sync()
    assert gpu.workspace_status(ws) == 0
    for m in layers:
        m.close()


def test_an_mlp_block_takes_smaller_batches_after_larger_ones(gpu):
    from mlxl3_b200.decoder import DenseMlp
    from mlxl3_b200.runtime import DeviceBuffer
    rng = np.random.default_rng(3)
    hidden, ffn = 4096, 14336
    block = DenseMlp(*(gpu.Exl3Linear(*random_layer(rng, a, b, 1), None, 1, 0) for a, b in ((hidden, ffn), (hidden, ffn), (ffn, hidden))))
    d_x, d_y = DeviceBuffer(1024 * hidden * 2), DeviceBuffer(1024 * hidden * 2)
    d_x.fill(0)
    for rows in (1024, 768, 33, 1):
        block.forward_device(d_x.ptr, rows, d_y.ptr)
