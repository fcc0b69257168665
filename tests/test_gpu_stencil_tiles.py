"""The stencil pass at the edges of its tiles: one tile exactly as wide (38) and
as high (18) as tiles get, one cell more, several tiles with remainders, the
narrowest block, odd heights (a thread owns two rows), few and many planes, and
the same with mirrored planes (octant), where every stencil reads across the
symmetry planes.

Against the fused kernel form, which evaluates every stencil point by point
from global memory.  Two steps; the forms differ by the rounding of the mixed
derivatives, of the KO quotients and of FMA contraction: 1e-12 of a field's
maximum in FP64, 1e-6 in the mixed form, the bars of test_gpu_engine_step.py."""
import numpy as np
import pytest

import amss_b200

from helpers import generic_state, relerr

pytestmark = pytest.mark.gpu


def _run(kernel, precision, symmetry, ex, h, st, bbox, tiling=None):
    e = amss_b200.Engine(precision=precision, kernel=kernel, symmetry=symmetry, eps=0.1)
    b = e.add_block(0, ex, bbox, bbox)
    e.commit()
    if tiling:
        e.set_level_tiling(0, *tiling)
    e.set_state(b, st)
    for _ in range(2):
        e.step(0, 0.25 * h)
    assert e.sync() == 0
    out = e.get_state(b)
    e.close()
    return out


@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("symmetry", [0, 2])
@pytest.mark.parametrize("ex", [(8, 7, 7), (38, 18, 9), (39, 19, 8), (77, 37, 12), (20, 36, 41)])
def test_tiles_match_the_fused_form(ex, symmetry, precision, bar):
    h = 0.2   # no power of two: the KO quotients round
    lo = [0.0] * 3 if symmetry == 2 else [-0.5 * n * h for n in ex]
    bbox = tuple(lo) + tuple(lo[d] + ex[d] * h for d in range(3))
    X = [lo[d] + (np.arange(ex[d]) + 0.5) * h for d in range(3)]
    st = generic_state(*X, seed=5, amp=0.5)
    ref = _run("fused", precision, symmetry, ex, h, st, bbox)
    got = _run("split", precision, symmetry, ex, h, st, bbox)
    for f in range(24):
        assert relerr(got[f], ref[f]) <= bar, f
    # slabs and tile widths change nothing
    again = _run("split", precision, symmetry, ex, h, st, bbox, tiling=(11, 2))
    assert np.array_equal(again, got)
