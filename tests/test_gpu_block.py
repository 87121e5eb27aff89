"""The few-row kernel with a cluster of CTAs per column block: every cluster size, inputs that do not divide evenly among CTAs and
warps, warps without rows, rows that begin inside a 128-input block, groups, rotated rows from outside, the row counts it takes."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import bits, gpu, random_layer  # noqa: F401

pytestmark = pytest.mark.gpu


def _close(got, want, rel=1e-2):                             # the bar of the layer tests: fp16 outputs after an fp16 rotation
    g, w = got.astype(np.float32), want.astype(np.float32)
    assert np.isfinite(g).all() and (np.abs(g - w) <= rel * np.abs(w).max(axis=1, keepdims=True)).all()


@pytest.mark.parametrize("cluster", [0, 1, 2, 3, 5, 8])
@pytest.mark.parametrize("n_in,n_out,k,cb", [(128, 128, 3, 0), (384, 640, 8, 1), (2176, 256, 5, 2), (4224, 1408, 4, 0)])
def test_cluster_sizes(gpu, cluster, n_in, n_out, k, cb):
    rng = np.random.default_rng(n_in + cluster)
    trellis, suh, svh = random_layer(rng, n_in, n_out, k, signs=False)
    bias = (rng.standard_normal(n_out) * 0.1).astype(np.float16)
    x = rng.standard_normal((8, n_in)).astype(np.float16)
    layer = gpu.Exl3Linear(trellis, suh, svh, bias, k, cb, exact_weights=cb != 2)
    want = oracle.linear_forward(trellis, k, cb, suh, svh, bias, x)
    gpu.set_option("block_cluster", cluster)
    try:
        batch = layer.forward(x)
        _close(batch, want)
        assert np.array_equal(bits(layer.forward_raw(oracle.prepare(x, suh)).astype(np.float16)),
                              bits(layer.forward_raw(oracle.prepare(x, suh)).astype(np.float16)))
        # the same sums from rotated rows, and for every row of a batch on its own
        assert np.array_equal(bits(batch), bits(oracle.finish(layer.forward_raw(oracle.prepare(x, suh)), svh, bias)))
        for rows in (1, 2, 3, 7):
            assert np.array_equal(bits(layer.forward(x[:rows])), bits(batch[:rows]))
    finally:
        gpu.set_option("block_cluster", 0)
    assert gpu.workspace_status(layer._workspace) == 0
    layer.close()


@pytest.mark.parametrize("rows", [1, 8])
def test_group_and_types_against_the_other_kernel(gpu, rows):
    rng = np.random.default_rng(rows)
    n_in, widths, k = 1152, (384, 128, 128), 6
    group = gpu.Exl3Group([gpu.Exl3Linear(*random_layer(rng, n_in, w, k, signs=False), None, k, 1) for w in widths])
    for dtype in (np.float16, np.float32):
        x = rng.standard_normal((rows, n_in)).astype(dtype)
        got = group.forward(x)
        gpu.set_option("block_cluster", -1)
        try:
            for a, b in zip(got, group.forward(x)):          # other order of the fp32 sums, then one fp16 rounding
                _close(a, b, rel=2e-3)
        finally:
            gpu.set_option("block_cluster", 0)
    group.close()


@pytest.mark.parametrize("experts,top_k,n_in,hidden,rows", [(6, 3, 512, 1152, 1), (9, 8, 256, 128, 2), (12, 2, 1024, 384, 5), (4, 1, 128, 256, 9)])
def test_expert_block_with_and_without_its_glue(gpu, experts, top_k, n_in, hidden, rows):
    """The glue behind the gate and up products and the sum over the slots behind the down product: same bits as launches of
    their own, whether a wave of clusters holds the products or not."""
    from tests.test_gpu_moe import check, make_bank, routes
    rng = np.random.default_rng(experts + rows)
    bank = make_bank(rng, experts, n_in, hidden, 4)
    moe = gpu.Exl3SwitchGlu(*bank, top_k, 4, 0)
    x = rng.standard_normal((rows, n_in)).astype(np.float16)
    selected, scores = routes(rng, rows, experts, top_k)
    selected[0, 0] = np.uint32(2 ** 31 + 5)                  # past the bank: counts as the last expert
    got = moe.forward(x, selected, scores)
    gpu.set_option("moe_fused", 0)
    try:
        assert np.array_equal(bits(got), bits(moe.forward(x, selected, scores)))
    finally:
        gpu.set_option("moe_fused", 1)
    selected[0, 0] = experts - 1
    check(got, oracle.switch_glu_forward(*bank, top_k, 4, 0, x, selected, scores), rms=4e-3)
    assert gpu.workspace_status(moe._workspace) == 0
    moe.close()


def test_the_device_holds_the_clusters_that_plans_count_on(gpu):
    """A wave of clusters is a constant of the plans, so that sums have one order on every GPU; a board that holds fewer would run
    full layers in two waves."""
    from tests.test_block_plan import RESIDENT
    from tests.test_plan_invariants import query
    held = query("clusters", 128, 128, 4, 1)
    assert len(held) == len(RESIDENT) and all(h >= r for h, r in zip(held, RESIDENT)), held
