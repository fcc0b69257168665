"""The tilings the autotuner times: among them the engine's own choice of slabs
and, whatever the block widths, the default width in one slab, which (0, 1) does
not ask for."""
import pytest

from amss_b200 import autotune
from amss_b200.hierarchy import box_in_box, single_block


@pytest.mark.parametrize("H", [single_block(n, -6.0, 6.0, 3) for n in (10, 32, 64, 130)]
                         + [box_in_box(40, 10.0, [(1.2, 0.3, -0.4)], 3, box_cells=32, seed=4, block_min=14, block_max=28)])
def test_candidates(H):
    for lev in range(len(H.levels)):
        c = autotune.candidates(H, lev)
        assert len(set(c)) == len(c)
        assert (0, 1, 0) in c and (autotune.WIDEST, 1, 0) in c
        assert all((w == 0 or 8 <= w <= autotune.WIDEST) and 1 <= z <= 4 and o == 0 for w, z, o in c)
