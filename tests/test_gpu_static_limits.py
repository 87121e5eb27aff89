"""The allocation-free entry point stays inside its 4 MiB whatever path its rows take."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import bits, gpu, random_layer  # noqa: F401
from tests.test_gpu_linear import _check_out

pytestmark = pytest.mark.gpu


def static(gpu, layer, x, n_out):
    from mlxl3_b200.runtime import DeviceBuffer
    rows = x.shape[0]
    d_x, d_y = DeviceBuffer.from_numpy(x), DeviceBuffer(rows * n_out * 2)
    layer.forward_static_device(d_x.ptr, gpu.F16, rows, d_y.ptr)
    return d_y.download((rows, n_out), np.float16)


def test_few_row_path_is_held_to_the_limit(gpu):
    """16 rows of 33024 outputs: the rows and the result fit, the parts the fused kernel keeps (4.2 MB) do not."""
    rng = np.random.default_rng(1)
    n_in, n_out, rows = 128, 33024, 16
    trellis, suh, svh = random_layer(rng, n_in, n_out, 2)
    layer = gpu.Exl3Linear(trellis, suh, svh, None, 2, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    want = oracle.linear_forward(trellis, 2, 0, suh, svh, None, x)
    _check_out(static(gpu, layer, x, n_out), want)               # tensor cores: fits
    try:
        gpu.set_option("qmm", 0)
        with pytest.raises(gpu.B200Exl3Error, match="allocation-free entry point owns"):
            static(gpu, layer, x, n_out)
    finally:
        gpu.set_option("qmm", 1)
    layer.close()


@pytest.mark.parametrize("rows,n_in,n_out", [(9, 128, 128), (64, 1024, 4096), (200, 512, 2048), (240, 256, 4096)])
def test_many_rows_on_the_fixed_array(gpu, rows, n_in, n_out):
    """Shapes whose shared items' parts fit the array and shapes that fall back to whole items."""
    rng = np.random.default_rng(rows)
    trellis, suh, svh = random_layer(rng, n_in, n_out, 3)
    layer = gpu.Exl3Linear(trellis, suh, svh, None, 3, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    pick = np.unique([0, rows // 2, rows - 1])
    want = oracle.linear_forward(trellis, 3, 0, suh, svh, None, x[pick])
    try:
        for qmm in (1, 0):                                       # tensor cores; batches of the fused kernel
            gpu.set_option("qmm", qmm)
            _check_out(static(gpu, layer, x, n_out)[pick], want)
            assert gpu.static_status() == 0
    finally:
        gpu.set_option("qmm", 1)
    layer.close()
