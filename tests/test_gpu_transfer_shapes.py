"""The prolongation and restriction kernels over the box widths where their
division into lanes changes: pieces of up to 4, up to 10 and more coarse cells
along x (segments of 10, 16 and 32 lanes), boxes of several pieces, pieces and
row groups with remainders.  Patches cut into blocks of 8 to 12 cells, of 18 to
30 cells, and not at all give boxes of those widths; each cell is computed by
the same operations in the same order whatever the cut, so the assembled patch
data agree bit for bit, as in test_gpu_split.py."""
import numpy as np
import pytest

from amss_b200.hierarchy import box_in_box

from test_gpu_split import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [32, 38])
def test_transfers_do_not_depend_on_the_box_widths(cells):
    got = []
    for lo, hi in ((200, 200), (18, 30), (8, 12)):
        H = box_in_box(44, 11.0, [(1.2, 0.3, -0.4)], 3, box_cells=cells, seed=3, block_min=lo, block_max=hi)
        got.append(_run(H, steps=1))
    for key in got[0]:
        assert np.array_equal(got[0][key], got[1][key]), key
        assert np.array_equal(got[0][key], got[2][key]), key
