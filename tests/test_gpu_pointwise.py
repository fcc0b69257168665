"""The staged pointwise pass and its tile order of the stencil terms, at the
sizes where they can go wrong: blocks whose point count leaves 1, 31, 33 and
127 points in the last 128-point tile, whole tiles, and levels of several
blocks (whose tiles start mid-list) with owned-cell and final-substep regions,
whose tiles do not follow the arrays.

Against the fused kernel form, which evaluates the same formulas from global
memory without stencil terms or staging.  The two differ by the rounding of the
mixed derivatives (tensor product against cross stencil) and FMA contraction,
a few units in the last place of terms up to 1/dx^2 times the field, times dt:
1e-12 of a field's maximum in FP64, 1e-6 in the mixed form, the bars of
test_gpu_engine_step.py."""
import numpy as np
import pytest

import amss_b200
from amss_b200.hierarchy import box_in_box
import amr as OA

from helpers import generic_state, relerr

pytestmark = pytest.mark.gpu


def _steps(kernel, precision, blocks, n=2):
    e = amss_b200.Engine(precision=precision, kernel=kernel, eps=0.1)
    ids = []
    for ex, lo, h, _ in blocks:
        bbox = tuple(lo) + tuple(lo[d] + ex[d] * h for d in range(3))
        ids.append(e.add_block(0, ex, bbox, bbox))
    e.commit()
    for b, (_, _, _, st) in zip(ids, blocks):
        e.set_state(b, st)
    for _ in range(n):
        e.step(0, 0.25 * blocks[0][2])
    assert e.sync() == 0
    out = [e.get_state(b) for b in ids]
    e.close()
    return out


def _block(ex, lo, h, seed):
    X = [lo[d] + (np.arange(ex[d]) + 0.5) * h for d in range(3)]
    return ex, lo, h, generic_state(*X, seed=seed, amp=0.5)


# points mod 128: 0, 1, 31, 33, 127, 89
@pytest.mark.parametrize("precision,bar", [("fp64", 1e-12), ("mixed", 1e-6)])
@pytest.mark.parametrize("ex", [(8, 8, 8), (81, 7, 7), (79, 7, 7), (113, 7, 7), (47, 7, 7), (9, 9, 9)])
def test_tile_remainders(ex, precision, bar):
    blocks = [_block(ex, (-1.0, -0.7, -0.9), 0.2, 3)]
    got, ref = _steps("split", precision, blocks), _steps("fused", precision, blocks)
    for f in range(24):
        assert relerr(got[0][f], ref[0][f]) <= bar, f


def test_region_tiles():
    H = box_in_box(40, 10.0, [(1.2, 0.3, -0.4)], 3, box_cells=32, seed=4, block_min=14, block_max=28)
    init = OA.initial_state(H, [1.0], [[1.2, 0.3, -0.4]], noise=1e-8)
    out = []
    for kernel in ("split", "fused"):
        e = amss_b200.Engine.from_hierarchy(H, precision="fp64", eps=0.1, kernel=kernel)
        assert e.final_region(1)[0] == 2   # the level takes final-substep regions
        for i, st in enumerate(init):
            e.set_state(i, st)
        e.coarse_step(0.25 * H.h0)
        assert e.sync() == 0
        out.append([e.get_state(i) for i in range(len(H.blocks))])
        e.close()
    # trK's maximum after one step is small against the terms its right-hand
    # side cancels: 1e-11, as test_gpu_fullsize.py's bar for trK allows.  The
    # metric is stored as its offset d from 1 (here |d| <= 1e-4) and enforce_ga
    # rounds 1 + d, its product with det^(-1/3) and the difference to 1 at each
    # of the finest level's 16 substeps: 4 roundings of values near 1 each, that
    # is 64 * 2^-53 = 7.1e-15 absolute, whatever the size of d
    for a, b in zip(*out):
        for f in range(24):
            bar = (1e-11 if f == 1 else 1e-12) * np.abs(b[f]).max() + (7.2e-15 if 2 <= f <= 7 else 0.0)
            assert np.abs(a[f] - b[f]).max() <= bar, f
