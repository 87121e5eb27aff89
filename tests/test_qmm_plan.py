"""The many-row product's plan over a small exhaustive domain (no GPU needed): tiles are whole sixteens of at most 256 tokens
that cover a pass, every CTA has at least one 128-input stage, shared tiles have room for their parts."""
import pytest

from tests.test_plan_invariants import query


@pytest.mark.parametrize("n_in", [128, 384, 4096, 25600])
@pytest.mark.parametrize("n_out", [128, 1408, 4096, 28672])
def test_tiles_and_parts(n_in, n_out):
    for rows in (9, 16, 63, 64, 65, 200, 256, 257, 1999, 16384):
        tile, splits, pass_rows, part_bytes = query("qmm", n_in, n_out, 4, rows)[4:]
        assert 16 <= tile <= 256 and tile % 16 == 0 and 1 <= pass_rows <= rows
        tiles = -(-pass_rows // tile)
        items, stages = tiles * n_out // 128, n_in // 128
        assert 0 <= splits <= stages and items <= 4095
        grid = items * splits if splits else min(148, items * stages)
        assert items * stages * grid < 2 ** 32
        parts = 0 if splits == 1 else (grid + items if items < grid else 2 * grid)
        assert part_bytes >= parts * tile * 128 * 4
