"""Rows that a caller cut out of a larger buffer: they start at an element, not on 16 bytes.  Inputs read element by element
give the same bits as aligned ones; many output rows go through the few-row kernel, which multiplies unrounded weights."""
import numpy as np
import pytest

from tests.gpu_util import bits, gpu, random_layer, to_bf16_bits  # noqa: F401
from tests.test_gpu_linear import _check_out
from tests.test_gpu_moe import make_bank, routes

pytestmark = pytest.mark.gpu

SHIFT = 3                                            # elements between a 256-byte boundary and the rows


def at(gpu, array, shift=SHIFT):
    """(buffer, address of the array's first element inside it)"""
    from mlxl3_b200.runtime import DeviceBuffer
    buf = DeviceBuffer(array.nbytes + 64)
    buf.upload(array, offset=shift * array.itemsize)
    return buf, buf.ptr + shift * array.itemsize


def out(gpu, shape, dtype, shift=SHIFT):
    from mlxl3_b200.runtime import DeviceBuffer
    size = np.dtype(dtype).itemsize
    buf = DeviceBuffer(int(np.prod(shape)) * size + 64)
    buf.fill(0xFF)
    return buf, buf.ptr + shift * size, lambda: buf.download(shape, dtype, offset=shift * size)


@pytest.mark.parametrize("kind", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("rows", [1, 2, 3, 8, 9, 70])
def test_linear_and_group_rows_at_any_element(gpu, rows, kind):
    rng = np.random.default_rng(rows)
    n_in, widths, k = 384, (256, 128), 3
    code = {"f16": gpu.F16, "bf16": gpu.BF16, "f32": gpu.F32}[kind]
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    x = {"f16": x.astype(np.float16), "bf16": to_bf16_bits(x), "f32": x}[kind]
    value = (lambda a: (a.astype(np.uint32) << 16).view(np.float32)) if kind == "bf16" else (lambda a: a)
    layers = []
    for n in widths:
        t, suh, svh = random_layer(rng, n_in, n, k, signs=False)
        layers.append(gpu.Exl3Linear(t, suh, svh, (rng.standard_normal(n) * 0.1).astype(np.float16), k, 0))
    group, layer = gpu.Exl3Group(layers), layers[0]
    want = [l.forward(x, code) for l in layers]
    ws = gpu.new_workspace(max(group.workspace_bytes(rows), layer.workspace_bytes(rows)))
    keep, d_x = at(gpu, x)
    for shift in (0, SHIFT):
        same = shift == 0 or rows <= 8
        y, d_y, read = out(gpu, (rows, widths[0]), x.dtype, shift)
        layer.forward_device(d_x, code, rows, d_y, ws)
        got = read()
        assert np.array_equal(got, want[0]) if same else True
        _check_out(value(got), value(want[0]), 2e-2 if kind == "bf16" else 1e-2)
        y, d_y, read = out(gpu, (rows, widths[0]), x.dtype, shift)
        layer.forward_static_device(d_x, code, rows, d_y)
        _check_out(value(read()), value(want[0]), 2e-2 if kind == "bf16" else 1e-2)
        ys = [out(gpu, (rows, n), x.dtype, shift) for n in widths]
        group.forward_device(d_x, code, rows, [y[1] for y in ys], ws)
        for y, w in zip(ys, want):
            _check_out(value(y[2]()), value(w), 2e-2 if kind == "bf16" else 1e-2)
    assert gpu.workspace_status(ws) == 0 and gpu.static_status() == 0
    for bad in (d_x + 1, 2 + (d_x & ~3) if kind == "f32" else d_x + 1):
        with pytest.raises(gpu.B200Exl3Error, match="aligned to their elements"):
            layer.forward_device(bad, code, rows, ys[0][1], ws)
        with pytest.raises(gpu.B200Exl3Error, match="aligned to their elements"):
            layer.forward_device(d_x, code, rows, bad, ws)
        with pytest.raises(gpu.B200Exl3Error, match="aligned to their elements"):
            group.forward_device(d_x, code, rows, [ys[0][1], bad], ws)
        with pytest.raises(gpu.B200Exl3Error, match="aligned to their elements"):
            layer.forward_static_device(bad, code, rows, ys[0][1])
    group.close()


@pytest.mark.parametrize("per_row", [False, True])
def test_rotations_at_any_element(gpu, per_row):
    from ctypes import c_void_p

    from mlxl3_b200 import _lib
    rng = np.random.default_rng(5)
    rows, n = 5, 384
    x, scales = rng.standard_normal((rows, n)).astype(np.float16), rng.uniform(0.5, 1.5, (rows if per_row else 1, n)).astype(np.float16)
    bias, sums = rng.standard_normal(n).astype(np.float16), rng.standard_normal((2, rows, n)).astype(np.float32)
    results = []
    for shift in (0, SHIFT):
        kx, d_x = at(gpu, x, shift)
        ks, d_s = at(gpu, scales, shift)
        kb, d_b = at(gpu, bias, shift)
        kp, d_p = at(gpu, sums, 0)
        h, d_h, read_h = out(gpu, (rows, n), np.float16, 0)
        y, d_y, read_y = out(gpu, (rows, n), np.float16, shift)
        _lib.call("b200exl3_prepare", c_void_p(d_x), gpu.F16, c_void_p(d_s), scales.shape[0], rows, n, c_void_p(d_h), None)
        _lib.call("b200exl3_finish", c_void_p(d_p), 2, c_void_p(d_s), scales.shape[0], c_void_p(d_b), rows, n, gpu.F16, c_void_p(d_y), None)
        results.append((read_h(), read_y()))
    for a, b in zip(*results):
        assert np.array_equal(bits(a), bits(b))


@pytest.mark.parametrize("rows", [2, 40])
def test_expert_block_input_at_any_element(gpu, rows):
    from mlxl3_b200.runtime import DeviceBuffer
    rng = np.random.default_rng(rows)
    experts, top_k, n_in, hidden, k = 8, 2, 256, 128, 4
    moe = gpu.Exl3SwitchGlu(*make_bank(rng, experts, n_in, hidden, k), top_k, k, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    selected, scores = routes(rng, rows, experts, top_k)
    want = moe.forward(x, selected, scores)
    keep, d_x = at(gpu, x)
    d_sel, d_sc, d_y = DeviceBuffer.from_numpy(selected), DeviceBuffer.from_numpy(scores), DeviceBuffer(want.nbytes)
    ws = gpu.new_workspace(moe.workspace_bytes(rows))
    moe.forward_device(d_x, gpu.F32, rows, d_sel.ptr, d_sc.ptr, gpu.F16, d_y.ptr, ws)
    assert np.array_equal(bits(d_y.download(want.shape, np.float16)), bits(want))
    for args in ((d_x + 2, d_sel.ptr, d_sc.ptr), (d_x, d_sel.ptr + 2, d_sc.ptr), (d_x, d_sel.ptr, d_sc.ptr + 1)):
        with pytest.raises(gpu.B200Exl3Error, match="aligned to their elements"):
            moe.forward_device(args[0], gpu.F32, rows, args[1], args[2], gpu.F16, d_y.ptr, ws)
    moe.close()


def test_calls_that_need_wider_places_say_so(gpu):
    """Raw products are stored four floats at a time; fused operators read four or eight values at a time."""
    from ctypes import c_void_p

    from mlxl3_b200 import _lib
    from mlxl3_b200.linear import Prologue
    rng = np.random.default_rng(2)
    n, k = 256, 4
    t, suh, svh = random_layer(rng, n, n, k)
    layer = gpu.Exl3Linear(t, suh, svh, None, k, 0)
    x = rng.standard_normal((1, n)).astype(np.float16)
    keep, d_x = at(gpu, x, 0)
    ws = gpu.new_workspace(layer.workspace_bytes(1))
    y, d_y, read = out(gpu, (2, n), np.float32, 0)
    w, d_w = at(gpu, np.ones(n, np.float16), 0)
    with pytest.raises(gpu.B200Exl3Error, match="must be 16-byte aligned"):
        _lib.call("b200exl3_linear_forward_raw", c_void_p(layer.handle), c_void_p(d_x), 1, c_void_p(d_y + 8), c_void_p(ws.ptr), ws.nbytes, None)
    with pytest.raises(gpu.B200Exl3Error, match="must be 16-byte aligned"):
        layer.forward_partial_device(d_x, gpu.F16, 1, d_y + 4, ws)
    with pytest.raises(gpu.B200Exl3Error, match="must be 16-byte aligned"):
        layer.forward_fused_device(Prologue.rms_norm(d_w, 1e-5), d_x + 8, 1, d_y, ws)
    with pytest.raises(gpu.B200Exl3Error, match="must be 8-byte aligned"):
        layer.forward_fused_device(Prologue.swiglu(d_w), d_x + 4, 1, d_y, ws)
    # rows on 8 bytes are enough for the SwiGLU prologue, as before
    k8, d_x8 = at(gpu, x, 4)
    layer.forward_fused_device(Prologue.swiglu(d_w), d_x8, 1, d_y, ws)
    got = read().reshape(-1).view(np.float16)[:n].copy()
    layer.forward_fused_device(Prologue.swiglu(d_w), d_x, 1, d_y, ws)
    assert np.array_equal(bits(got), bits(read().reshape(-1).view(np.float16)[:n]))
    layer.close()
