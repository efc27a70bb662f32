"""The g(r) histogram's counts equal the oracle's FP64 binning (ObservableCorrelation.cc:191-207) where the FP32
distance cannot decide: distances on bin edges, positions far outside the box, bins finer than FP32 resolves, grids
that start inside or end short of the pairs; and at the edges of the particle tiles."""
import numpy as np
import pytest

import oracle as O
import pimcplusplus_b200 as P

from helpers import random_walk_path

pytestmark = pytest.mark.gpu


def check(path, box, start, end, points):
    slices, n = path.shape[:2]
    o = O.System(n, slices, box, 0.1, 1.0, 0)
    o.set_path(path)
    d = P.PathData(n, slices, box, 0.1, 1.0)
    d.set_path(path)
    d.gofr_setup(start, end, points)
    d.gofr_accumulate()
    hist, _, count = d.gofr_get()
    ref = o.gofr_accumulate(start, end if end > 0 else box[0], points)
    assert count == 1
    assert np.array_equal(hist, ref)
    d.close()


@pytest.mark.parametrize("n", [2, 15, 16, 17, 31, 33, 63, 64, 65, 129, 200])
def test_tiles(n):
    box = np.array([9.0, 10.0, 12.5])
    for slices in (2, 4):
        check(random_walk_path(n, slices, box, 0.5, n, far=0.2), box, 0.0, 0.0, 101)
    check(random_walk_path(n, 40, box, 0.5, n), box, 0.0, 5.0, 50)


@pytest.mark.parametrize("start,end,points", [(0.0, 0.0, 2), (0.0, 20.0, 101), (1.7, 4.2, 33), (0.0, 6.0, 12289),
                                              (3.0, 3.001, 12289), (0.0, 1e-3, 9), (9.9, 30.0, 500)])
def test_grids(start, end, points):
    box = np.array([10.0, 10.0, 10.0])
    check(random_walk_path(70, 5, box, 0.7, points, far=0.3), box, start, end, points)


@pytest.mark.parametrize("cells", [8, 10])
def test_distances_on_bin_edges(cells):
    """Lattice sites: every axis distance is a multiple of the bin width, many at exactly half the box."""
    box = np.array([10.0, 10.0, 10.0])
    ijk = np.stack(np.meshgrid(*[np.arange(5)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)
    path = np.repeat((ijk * (box / cells))[None], 3, axis=0)
    check(path, box, 0.0, 10.0, cells + 1)
    check(path, box, 0.0, 10.0, 4 * cells + 1)
    check(path + 3 * box, box, 0.0, 0.0, 101)


def test_far_positions_and_box_sizes():
    for side in (1e-17, 1e-3, 1e5, 1e18):
        box = np.array([1.0, 1.1, 1.3]) * side
        check(random_walk_path(40, 3, box, 0.3 * side, 3), box, 0.0, 0.0, 64)
    box = np.array([10.0, 10.0, 10.0])
    path = random_walk_path(40, 3, box, 0.3, 4)
    path[:, ::3] += 1e9 * box
    path[1, 5] -= 2e6 * box
    check(path, box, 0.0, 0.0, 201)
