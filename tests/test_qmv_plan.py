"""The grid of the fused few-row kernel (no GPU needed): whole CTAs per column block or the full grid, never more than two per
SM, at most a row per warp too many, the same for every batch of up to eight rows that fits two CTAs per SM."""
import pytest

from tests.test_plan_invariants import query


@pytest.mark.parametrize("n_in", [128, 512, 2176, 4096, 14336])
@pytest.mark.parametrize("n_out", [128, 1408, 4096, 37888, 102400])
def test_grid(n_in, n_out):
    blocks, rows_of_block = n_out // 128, n_in // 16
    full = min(296, max(1, blocks * rows_of_block // 8))
    grids = {query("qmv", n_in, n_out, 4, rows)[0] for rows in (1, 2, 3, 8)}
    assert len(grids) == 1
    grid = grids.pop()
    assert grid == full or (grid % blocks == 0 and grid <= full and grid * 8 <= blocks * rows_of_block)
