"""ShortRangeClass::d_dBeta and the energy terms of the pair walk (csrc/pair_path.cu) against the oracle, where
its rules switch: particle tiles, link chunks, the cut at half a box between two slices, and the lists of pairs
within a short table's range (taken from 256 particles and 5e7 range / side (pair, link)s on for tables that end
below 0.3 box sides)."""
import math

import numpy as np
import pytest

import oracle as O
import pimcplusplus_b200 as P
from pimcplusplus_b200 import workloads as W

from helpers import random_walk_path, rel_err

pytestmark = pytest.mark.gpu

TAU, LEVELS = 0.01, 4
# FP64 sums of the same terms in another order, at most 1e6 of them of one sign's size: the repository's bound for sums
TOL = 1e-12


def david_tables(end, npts, cols, seed, last_zero=True):
    """V, u_00 and off-diagonal columns per level; the potential of tau table 0 differs from the others'."""
    rng = np.random.default_rng(seed)
    r = np.linspace(1.2, end, npts)
    u = np.zeros((LEVELS, npts, cols))
    du = np.zeros_like(u)
    for lev in range(LEVELS):
        u[lev, :, 0] = W.lj(np.maximum(r, 2.0)) * (1.0 + 0.1 * lev)
        u[lev, :, 1] = TAU * 2 ** lev * u[lev, :, 0]
        for c in range(2, cols):
            u[lev, :, c] = 1e-3 * rng.random() * np.exp(-r)
        du[lev] = 0.7 * u[lev] + 0.01 * np.sin(r)[:, None]
    if last_zero:
        u[:, -1] = du[:, -1] = 0.0
    return r[0], end, u, du


def pair(n, slices, box, end, npts=120, cols=2, terms=0, tau_pos=0, step=0.4, far=0.05, last_zero=True):
    box = np.asarray(box, dtype=np.float64)
    path = random_walk_path(n, slices, box, step, n + slices, far=far)
    start, end, u, du = david_tables(end, npts, cols, n, last_zero)
    o = Oracle(n, box, W.HE4_LAMBDA, O.PairAction.david_arrays(start, end, u, du, tau_pos, terms), path)
    d = P.PathData(n, slices, box, TAU, W.HE4_LAMBDA, 0)
    d.pa_david(P.GRID_LINEAR, start, end, u, du, tau_pos, terms)
    d.set_path(path)
    return o, d


class Oracle:
    """The oracle link by link, the links added exactly: its own running sum over a path of 3e6 like terms (a table
    whose end is not zero) is off by more than the bound."""

    def __init__(self, n, box, lam, pa, path):
        self.n, self.box, self.lam, self.pa, self.path = n, box, lam, pa, path

    def system(self, rows):
        o = O.System(self.n, len(rows), self.box, TAU, self.lam, 0)
        o.set_pa(self.pa)
        o.set_path(rows)
        return o

    def energy(self):
        m = len(self.path) - 1
        links = [self.system(self.path[s:s + 2]).energy() for s in range(m)]
        e = {k: math.fsum(x[k] for x in links) for k in ("kinetic", "du_short", "v_short")}
        e["total"] = (e["kinetic"] + e["du_short"]) / m
        return e

    def shortrange_dbeta(self, s1, s2, level):
        o, skip = self.system(self.path), 1 << level
        return math.fsum(o.shortrange_dbeta(s, s + skip, level) for s in range(s1, s2, skip))


def check(o, d, ranges=()):
    ref = o.energy()
    if math.isfinite(ref["kinetic"]):
        got = d.energy()
    else:  # the kinetic estimator's Gaussian underflows on the longest links (light particles), as the oracle's
        with pytest.raises(P.PimcError) as e:
            d.energy()
        assert e.value.status == 3
        got = ref
    for k in ("kinetic", "du_short", "v_short", "total"):
        assert got is ref or rel_err(got[k], ref[k], max(abs(ref[k]), 1.0)) < TOL, (k, got[k], ref[k])
    for s1, s2, level in ranges:
        a, b = o.shortrange_dbeta(s1, s2, level), d.d_dbeta(P.ACTION_SHORTRANGE, s1, s2, level)
        assert rel_err(b, a, max(abs(a), 1.0)) < TOL, (s1, s2, level, b, a)
    d.close()


@pytest.mark.parametrize("n", [2, 15, 16, 17, 33, 63, 64, 65, 130])
@pytest.mark.parametrize("slices", [2, 10, 18])
def test_tiles_and_chunks(n, slices):
    o, d = pair(n, slices, [9.0, 10.0, 11.0], 4.5)
    check(o, d, [(0, slices - 1, 0)] + ([(1, 9, 3), (2, 8, 1), (3, 4, 0), (5, 5, 0)] if slices > 9 else []))


@pytest.mark.parametrize("end", [3.0, 5.9, 6.1, 14.0])  # 0.15, 0.295 and 0.305 of the box (lists / none), and 0.7
@pytest.mark.parametrize("last_zero", [True, False])
def test_range(end, last_zero):
    for n, slices in ((255, 4), (256, 4), (300, 70)):  # lists from 256 on; three chunks of links
        o, d = pair(n, slices, [20.0] * 3, end, last_zero=last_zero, step=0.3)
        check(o, d, [(1, slices - 1, 0)])


@pytest.mark.parametrize("n", [512, 513, 577, 1090])  # eight tiles, a ninth, a ragged row of groups, three rows
@pytest.mark.parametrize("end", [2.0, 5.9])  # a group's pairs in one list, and in several
def test_groups_of_tiles(n, end):
    o, d = pair(n, 4, [20.0, 20.5, 21.0], end, step=0.3)
    check(o, d, [(0, 3, 0)])


@pytest.mark.parametrize("terms", [1, 2])
@pytest.mark.parametrize("n,end", [(40, 5.0), (280, 3.2)])
def test_offdiagonal_terms(n, end, terms):
    o, d = pair(n, 20, [11.0, 11.5, 12.0], end, cols=7, terms=terms, tau_pos=1)
    check(o, d, [(0, 16, 2)])


def test_long_steps_take_the_following_image():
    """Links longer than half the box: DistDisp's second displacement is not the slice's own minimum image."""
    for n, end in ((50, 12.0), (260, 2.9)):
        o, d = pair(n, 12, [10.0] * 3, end, step=4.0, far=0.3)
        check(o, d, [(0, 8, 1)])


@pytest.mark.parametrize("n", [5, 32, 70])
def test_tricubic_and_coulomb(n):
    box = np.array([12.0, 12.0, 12.0])
    for slices, step in ((2, 0.3), (11, 0.3), (11, 4.0)):
        path = random_walk_path(n, slices, box, step, n, far=0.1)
        qg, yg, tg, umat, dumat, pg, pot = W.tricubic_tables(box[0], TAU, LEVELS, nq=25, ny=8, nt=9, pot_n=200)
        o = Oracle(n, box, W.HE4_LAMBDA, O.PairAction.tricubic(qg, yg, tg, TAU, umat, dumat, pg, pot), path)
        d = P.PathData(n, slices, box, TAU, W.HE4_LAMBDA, 0)
        d.pa_tricubic(qg, yg, tg, TAU, umat, dumat, pg, pot)
        d.set_path(path)
        check(o, d, [(0, slices - 1, 0)] + ([(1, 9, 2)] if slices > 9 else []))
        o = Oracle(n, box, 1.0, O.PairAction.classical_coulomb(TAU, LEVELS, 2.0), path)
        d = P.PathData(n, slices, box, TAU, 1.0, 0)
        d.pa_coulomb(2.0, LEVELS)
        d.set_path(path)
        check(o, d, [(0, slices - 1, 0)])


@pytest.mark.parametrize("n,end", [(20, 4.0), (300, 2.9)])
def test_non_finite_positions_are_reported(n, end):
    for bad in (np.nan, np.inf):
        o, d = pair(n, 40, [10.0] * 3, end)
        path = d.get_path()
        path[17, n - 3, 1] = bad
        d.set_path(path)
        for call in (d.energy, lambda: d.d_dbeta(P.ACTION_SHORTRANGE, 0, 39, 0)):
            with pytest.raises(P.PimcError) as e:
                call()
            assert e.value.status == 3
        d.close()


@pytest.mark.parametrize("n,end", [(20, 4.0), (300, 2.9)])
@pytest.mark.parametrize("rows", [[17], [16, 17, 18], list(range(40))])
def test_overflowing_distances_are_reported(n, end, rows):
    """Positions whose squared distance overflows: no pair of theirs has a length, so no sum of theirs is a number."""
    o, d = pair(n, 40, [10.0] * 3, end, last_zero=False)
    path = d.get_path()
    path[rows, n - 3, 1] = 1e200
    d.set_path(path)
    for call in (d.energy, lambda: d.d_dbeta(P.ACTION_SHORTRANGE, 0, 39, 0)):
        with pytest.raises(P.PimcError) as e:
            call()
        assert e.value.status == 3
    d.close()


@pytest.mark.parametrize("n", [5, 32, 70])
def test_coulomb_long_steps_with_the_potential(n):
    """Links longer than half the box in the walk that carries V: heavier zero-point motion than in
    test_tricubic_and_coulomb keeps the kinetic estimator finite there, so d_dBeta and V are compared."""
    box = np.array([12.0, 12.0, 12.0])
    path = random_walk_path(n, 11, box, 4.0, n, far=0.1)
    o = Oracle(n, box, W.HE4_LAMBDA, O.PairAction.classical_coulomb(TAU, LEVELS, 2.0), path)
    assert math.isfinite(o.energy()["kinetic"])
    d = P.PathData(n, 11, box, TAU, W.HE4_LAMBDA, 0)
    d.pa_coulomb(2.0, LEVELS)
    d.set_path(path)
    check(o, d, [(0, 10, 0), (1, 9, 2)])


class EndApart(Oracle):
    """The oracle on tables less their end value, which every pair of every link adds and is multiplied out here: a
    spline through y - c is the spline through y, less c.  Its running sum over a link's 1e5 like end values is off by
    more than the bound."""

    def __init__(self, n, box, end, npts, path):
        start, end, u, du = david_tables(end, npts, 2, n, last_zero=False)
        self.v, self.du = u[0, -1, 0], u[0, -1, 0] + du[0, -1, 1]
        super().__init__(n, box, W.HE4_LAMBDA, O.PairAction.david_arrays(start, end, u - u[:, -1:], du - du[:, -1:], 0, 0),
                         path)

    def energy(self):
        e, m, pairs = super().energy(), len(self.path) - 1, self.n * (self.n - 1) // 2
        e["du_short"] += m * pairs * self.du
        e["v_short"] += m * pairs * self.v
        e["total"] = (e["kinetic"] + e["du_short"]) / m
        return e

    def shortrange_dbeta(self, s1, s2, level):
        return super().shortrange_dbeta(s1, s2, level) + (s2 - s1 >> level) * (self.n * (self.n - 1) // 2) * self.du


# Lists are taken from 5e7 range / side (pair, link)s on.  The cases above that were short of that go the general way
# now; these reach the lists again, with the same edges: tiles, groups of tiles, chunks of links, ragged ends.
@pytest.mark.parametrize("n,slices,end", [
    (512, 39, 2.0), (512, 40, 2.0),  # 4.97e6 and 5.10e6 at 0.1 sides: either side of the line
    (513, 41, 2.0), (577, 33, 2.0), (1090, 10, 2.0),  # a ninth tile, a ragged row of groups, three rows
    (1090, 27, 5.9), (300, 331, 5.9),  # groups whose pairs fill several lists; eleven chunks of links, the last of ten
    (256, 470, 5.9)])
@pytest.mark.parametrize("last_zero", [True, False])
def test_lists(n, slices, end, last_zero):
    box = np.array([20.0, 20.5, 21.0])
    o, d = pair(n, slices, box, end, step=0.3, last_zero=last_zero)
    if not last_zero:
        o = EndApart(n, box, end, 120, o.path)
    check(o, d, [(0, slices - 1, 0), (1, slices - 1, 0)])


@pytest.mark.parametrize("end", [2.0, 5.9])  # above the line at 0.1 sides, below it at 0.295
def test_lists_one_link(end):
    """Fifty rows of tiles.  With a table that ends at zero: the oracle's running sum over 5e6 like terms is off by
    more than the bound."""
    o, d = pair(3170, 2, [20.0, 20.5, 21.0], end, step=0.3)
    check(o, d, [(0, 1, 0)])


@pytest.mark.parametrize("terms", [1, 2])
def test_lists_offdiagonal_terms(terms):
    o, d = pair(280, 400, [11.0, 11.5, 12.0], 3.2, cols=7, terms=terms, tau_pos=1)
    check(o, d, [(0, 399, 0)])


def test_lists_long_steps():
    o, d = pair(260, 450, [10.0] * 3, 2.9, step=4.0, far=0.3)
    check(o, d, [(0, 448, 0)])


@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e200])
@pytest.mark.parametrize("rows", [[170], [16, 17, 18], list(range(330))])
def test_lists_report_non_finite_pairs(bad, rows):
    o, d = pair(300, 330, [10.0] * 3, 2.9, last_zero=False)
    path = d.get_path()
    path[rows, 297, 1] = bad
    d.set_path(path)
    for call in (d.energy, lambda: d.d_dbeta(P.ACTION_SHORTRANGE, 0, 329, 0)):
        with pytest.raises(P.PimcError) as e:
            call()
        assert e.value.status == 3
    d.close()
