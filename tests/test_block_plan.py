"""When a layer of up to 8 rows gets a cluster of CTAs per column block (no GPU needed): one wave of clusters that a B200 holds (of
single CTAs two), shared
memory for one CTA per SM, the same partition for every row count."""
import pytest

from tests.test_plan_invariants import query

RESIDENT = (148, 74, 45, 33, 26, 22, 15, 15)


@pytest.mark.parametrize("k", [1, 3, 4, 8])
@pytest.mark.parametrize("n_in", [128, 512, 2176, 4096, 14336, 28672])
@pytest.mark.parametrize("n_out", [128, 1408, 4096, 6144, 14336, 18944, 28672])
def test_plan(k, n_in, n_out):
    plans = [query("block", n_in, n_out, k, rows) for rows in (1, 2, 3, 8)]
    assert len({(p[0], p[1], p[2]) for p in plans}) == 1      # the row count does not change how the sums are cut
    for rows, (use, cluster, grid, warps, smem, warp_smem, xs_stride, stage) in zip((1, 2, 3, 8), plans):
        if not use:
            assert (n_in, n_out) not in ((4096, 4096), (4096, 6144), (14336, 4096), (2176, 1408), (512, 14336))
            continue
        blocks = n_out // 128
        assert grid == blocks * cluster and cluster <= n_in // 16
        assert blocks <= (2 if cluster == 1 else 1) * RESIDENT[cluster - 1]
        assert 112 * 1024 < smem <= 200 * 1024
        # inputs of a CTA, rounded out to whole 128-input blocks at both ends
        rows_of_cta = -(-(n_in // 16) // cluster)
        assert xs_stride >= min(n_in, (rows_of_cta + 14) // 8 * 128) + 8
        assert warp_smem >= rows * 132 * 4 and stage >= warps * warp_smem + rows * xs_stride * 2
        assert smem >= stage + -(-rows // cluster) * cluster * 512
    assert query("block", n_in, n_out, k, 9)[0] == 0
