"""The Z4c forms of the staged pointwise pass and of the stencil pass at the
edges of their tiles: blocks that leave 1, 31, 33 and 127 points in the last
128-point tile, tiles exactly as wide (38) and as high (18) as they get and one
cell more, odd heights, few and many planes, and the same with mirrored planes.
Z4c has rows (Theta's), slot sizes and line shifts of its own there, and no fused
form to compare with: the reference is the oracle's RK4 step.

One step at a spacing of 0.2.  FP64: 1e-12 of a field's maximum, the bar of
test_gpu_z4c.py.  Mixed: a stage's FP32 metric d is off by 2^-24 of itself.  The
second derivatives in a Ricci component weigh that by up to
(3 * 16/3 + 3 * 2 * 9/4) / dx^2 = 740 and one half, A~ takes it times
alpha chi <= 0.6 and dt = 0.05, and here d is at most about twice A~'s maximum:
2^-24 * 370 * 0.03 * 2 = 1.3e-6 of A~, the largest of any field.  Bar 2e-6.
"""
import ctypes

import numpy as np
import pytest

import amss_b200
import oracle as O
from amr import _ptrs

from helpers import generic_state, relerr

pytestmark = pytest.mark.gpu
H = 0.2


def _block(ex, symmetry):
    lo = [0.0] * 3 if symmetry == 2 else [-0.5 * n * H for n in ex]
    bbox = tuple(lo) + tuple(lo[d] + ex[d] * H for d in range(3))
    X = [lo[d] + (np.arange(ex[d]) + 0.5) * H for d in range(3)]
    z, y, x = np.meshgrid(X[2], X[1], X[0], indexing="ij")
    theta = 0.05 * np.sin(0.7 * x + 0.2) * np.cos(0.5 * y) * np.sin(0.9 * z + 0.4)
    return bbox, X, np.concatenate([generic_state(*X, seed=5, amp=0.5), theta[None]])


def _oracle_step(ex, symmetry, bbox, X, state, dt):
    u, a, b, K, new = (np.zeros_like(state) for _ in range(5))
    u[:] = state
    box = np.array(bbox)
    for sub, (src, out) in enumerate([(u, a), (a, b), (b, a), (a, new)]):
        err = O.lib().oracle_evolve_substep(
            (ctypes.c_int * 3)(*ex), *[O._p(v) for v in X], O._p(box), _ptrs(u), _ptrs(src), _ptrs(out), _ptrs(K),
            ctypes.c_int(sub), ctypes.c_double(dt), ctypes.c_double(0.1), ctypes.c_double(1e-5 - 1.0),
            ctypes.c_int(symmetry), ctypes.c_int(0), ctypes.c_int(25))
        assert err == 0
    return new


def _step(ex, symmetry, precision, bbox, state, dt, tiling=None):
    e = amss_b200.Engine(precision=precision, symmetry=symmetry, eps=0.1, formulation="z4c")
    b = e.add_block(0, ex, bbox, bbox)
    e.commit()
    if tiling:
        e.set_level_tiling(0, *tiling)
    e.set_state(b, state)
    e.step(0, dt)
    assert e.sync() == 0
    out = e.get_state(b)
    e.close()
    return out


@pytest.mark.parametrize("symmetry", [0, 2])
# points mod 128: 0, 1, 31, 33, 127; then the stencil pass's tiles
@pytest.mark.parametrize("ex", [(8, 8, 8), (81, 7, 7), (79, 7, 7), (113, 7, 7), (47, 7, 7),
                                (38, 18, 9), (39, 19, 8), (77, 37, 12), (20, 36, 41)])
def test_z4c_tiles_match_the_oracle(ex, symmetry):
    bbox, X, state = _block(ex, symmetry)
    dt = 0.25 * H
    ref = _oracle_step(ex, symmetry, bbox, X, state, dt)
    for precision, bar in (("fp64", 1e-12), ("mixed", 2e-6)):
        got = _step(ex, symmetry, precision, bbox, state, dt)
        for f in range(25):
            assert relerr(got[f], ref[f]) <= bar, (precision, f)
        # slabs and tile widths change nothing
        assert np.array_equal(_step(ex, symmetry, precision, bbox, state, dt, tiling=(11, 2)), got)
