"""Edges of the many-row product and of the array interface: row counts around its token tiles (16, 64, 256), shapes whose
items are shared by several CTAs, held whole by one, or fewer than the CTAs, groups in one launch, and the scratch pool."""
import threading

import numpy as np
import pytest

import oracle
from tests.gpu_util import bits, gpu, random_layer, to_bf16_bits, from_bf16_bits  # noqa: F401

pytestmark = pytest.mark.gpu


def _close(got, want, rel=1e-2):
    g, w = got.astype(np.float32), want.astype(np.float32)
    assert np.isfinite(g).all() and g.shape == w.shape
    assert (np.abs(g - w) <= rel * np.abs(w).max(axis=1, keepdims=True)).all()


@pytest.mark.parametrize("n_in,n_out,k", [(128, 128, 3), (384, 640, 2), (1152, 128, 6), (256, 4864, 7)])
@pytest.mark.parametrize("rows", [9, 16, 49, 64, 65, 256, 257, 500])
def test_row_counts_around_the_tiles(gpu, n_in, n_out, k, rows):
    rng = np.random.default_rng(n_in + n_out + rows)
    trellis, suh, svh = random_layer(rng, n_in, n_out, k)
    bias = (rng.standard_normal(n_out) * 0.1).astype(np.float16)
    layer = gpu.Exl3Linear(trellis, suh, svh, bias, k, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    pick = np.unique([0, 1, rows // 2, rows - 2, rows - 1])
    got = layer.forward(x)
    assert got.dtype == np.float32 and gpu.workspace_status(layer._workspace) == 0
    _close(got[pick], oracle.linear_forward(trellis, k, 0, suh, svh, bias, x[pick].astype(np.float16)))
    assert np.array_equal(got.view(np.uint32), layer.forward(x).view(np.uint32))         # same sums in the same order
    got16 = from_bf16_bits(layer.forward(to_bf16_bits(x), gpu.BF16))
    _close(got16[pick], oracle.linear_forward(trellis, k, 0, suh, svh, bias, from_bf16_bits(to_bf16_bits(x))[pick].astype(np.float16)), rel=2e-2)
    layer.close()


@pytest.mark.parametrize("rows", [3, 9, 70, 300])
def test_group_members_in_one_launch(gpu, rows):
    rng = np.random.default_rng(rows)
    n_in, widths, k = 512, (384, 128, 256), 3
    parts = [random_layer(rng, n_in, w, k, signs=False) for w in widths]
    group = gpu.Exl3Group([gpu.Exl3Linear(*p, None, k, 1) for p in parts])
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    pick = np.unique([0, rows // 2, rows - 1])
    for got, p in zip(group.forward(x), parts):
        _close(got[pick], oracle.linear_forward(p[0], k, 1, p[1], p[2], None, x[pick]))
    group.close()


def test_forced_splits_give_the_same_result(gpu):
    rng = np.random.default_rng(3)
    trellis, suh, svh = random_layer(rng, 2048, 256, 4)
    x = rng.standard_normal((40, 2048)).astype(np.float16)
    want = oracle.linear_forward(trellis, 4, 0, suh, svh, None, x)
    try:
        for splits in (1, 2, 4):
            gpu.set_option("qmm_splits", splits)
            layer = gpu.Exl3Linear(trellis, suh, svh, None, 4, 0)
            _close(layer.forward(x), want)
            layer.close()
    finally:
        gpu.set_option("qmm_splits", 0)


def test_array_calls_from_several_threads_share_the_pool(gpu):
    rng = np.random.default_rng(8)
    trellis, suh, svh = random_layer(rng, 256, 384, 4)
    xs = [rng.standard_normal((n, 256)).astype(np.float16) for n in (1, 5, 17, 90)]
    want = [oracle.linear_forward(trellis, 4, 0, suh, svh, None, x) for x in xs]
    failures = []

    def work(x, w):
        try:
            gpu.init(0)
            layer, stream = gpu.Exl3Linear(trellis, suh, svh, None, 4, 0), gpu.Stream()
            first = layer.forward(x, stream=stream)
            for _ in range(20):
                assert np.array_equal(bits(layer.forward(x, stream=stream)), bits(first))
            _close(first, w)
        except Exception as e:                                   # noqa: BLE001 -- reported by the main thread
            failures.append(e)
    threads = [threading.Thread(target=work, args=a) for a in zip(xs, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


@pytest.mark.parametrize("k", [5, 7, 8])
@pytest.mark.parametrize("rows", [48, 260])
def test_long_runs_of_wide_weights(gpu, k, rows):
    """Every CTA's run goes round the ring of packed stages many times and through several items."""
    rng = np.random.default_rng(k * rows)
    trellis, suh, svh = random_layer(rng, 2048, 3200, k)
    layer = gpu.Exl3Linear(trellis, suh, svh, None, k, 0)
    x = rng.standard_normal((rows, 2048)).astype(np.float16)
    got = layer.forward(x)
    for _ in range(10):
        assert np.array_equal(bits(layer.forward(x)), bits(got))
    pick = np.unique([0, rows // 2, rows - 1])
    _close(got[pick], oracle.linear_forward(trellis, k, 0, suh, svh, None, x[pick]))
    layer.close()


@pytest.mark.parametrize("n_in,n_out,k,rows", [(128, 81920, 3, 16), (256, 51200, 4, 48), (384, 30720, 6, 33), (640, 2176, 4, 64)])
def test_many_items_on_a_cta(gpu, n_in, n_out, k, rows):
    """Tiles of up to 64 tokens: a CTA's items follow each other while the one before is still being finished; items of one to
    five stages, fewer than are in flight."""
    rng = np.random.default_rng(n_in + rows)
    trellis, suh, svh = random_layer(rng, n_in, n_out, k)
    layer = gpu.Exl3Linear(trellis, suh, svh, None, k, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    got = layer.forward(x)
    for _ in range(5):
        assert np.array_equal(bits(layer.forward(x)), bits(got))
    assert gpu.workspace_status(layer._workspace) == 0
    pick = np.unique([0, 15, rows // 2, rows - 1])
    _close(got[pick], oracle.linear_forward(trellis, k, 0, suh, svh, None, x[pick]))
    layer.close()


@pytest.mark.parametrize("splits", [1, 3, 8])
@pytest.mark.parametrize("n_in,n_out,k,rows", [(128, 256, 4, 9), (1152, 384, 3, 17), (1024, 128, 8, 64), (2176, 640, 5, 33), (4224, 256, 2, 16), (256, 25600, 6, 48)])
def test_items_with_ctas_of_their_own(gpu, splits, n_in, n_out, k, rows):
    """Tiles of up to 64 tokens without finishing warps: whole items, items shared by CTAs that do not get equal stages, and more CTAs
    than a wave holds."""
    rng = np.random.default_rng(n_in + rows + splits)
    trellis, suh, svh = random_layer(rng, n_in, n_out, k)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    gpu.set_option("qmm_splits", splits)
    try:
        layer = gpu.Exl3Linear(trellis, suh, svh, None, k, 0)
        got = layer.forward(x)
        for _ in range(5):
            assert np.array_equal(bits(layer.forward(x)), bits(got))
        assert gpu.workspace_status(layer._workspace) == 0
        layer.close()
    finally:
        gpu.set_option("qmm_splits", 0)
    _close(got, oracle.linear_forward(trellis, k, 0, suh, svh, None, x))
