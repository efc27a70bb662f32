"""Device moves at the library's own launch shape (cluster_ctas = 0, threads_per_cta = 0): the accept trace and the
path against the oracle's replay on both sides of each line of the rule (work = (N - 1) 2^L: 200, 1200, 4000), for
both schedules, and for so many windows that the clusters are halved."""
import numpy as np
import pytest

import oracle as O
import pimcplusplus_b200 as P
from pimcplusplus_b200 import workloads as W

from helpers import lj_case, tricubic_case
from test_gpu_coulomb import compare, jellium_moves
from test_gpu_parity import compare_traces, compare_window_traces, run_trace_pair

pytestmark = pytest.mark.gpu


def system(tmp_path, n, m, levels, seed):
    cfg, tau, box, dm = lj_case(tmp_path, n=n, m=m, levels=levels)
    path = W.lattice_path(n, m + 1, box, np.random.default_rng(seed))
    o = O.System(n, m + 1, box, tau, W.HE4_LAMBDA, 0)
    o.set_pa(O.PairAction.from_dm(dm, tau, 0))
    o.set_path(path)
    d = P.PathData(n, m + 1, box, tau, W.HE4_LAMBDA, 0)
    d.set_path(path)
    d.pa_david_from_dm(dm, 0)
    return o, d


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
@pytest.mark.parametrize("n", [2, 25, 27, 150, 152, 500, 502])
def test_sequential(tmp_path, n, precision):
    o, d = system(tmp_path, n, 16, 3, n)
    ref, got, stats = run_trace_pair(o, d, 3, 5, 12, 31 + n, precision=precision)
    compare_traces(ref, got, stats)
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("n,m,levels", [(30, 64, 1), (502, 64, 1), (152, 64, 2), (502, 16, 3), (9, 40, 3), (60, 64, 5)])
def test_windows(tmp_path, n, m, levels):
    o, d = system(tmp_path, n, m, levels, n)
    o.bisection_config(levels, 4)
    o.rng_seed(7 + n)
    ref = o.run_windows(6)
    bb = P.BisectionBlock(d, levels, 4, schedule=P.WINDOWS)
    bb.seed(7 + n)
    assert bb.windows == min(m >> levels, 64) and bb.occupancy() >= bb.windows
    got, stats = bb.MakeMoves(6)
    compare_window_traces(ref, got, stats)
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
@pytest.mark.parametrize("n", [25, 27, 150, 152, 500, 502])
def test_tricubic(n, precision):
    cfg, tau, box, (qg, yg, tg, umat, dumat, pg, pot) = tricubic_case(n=n, m=16)
    path = W.lattice_path(n, 17, box, np.random.default_rng(n))
    o = O.System(n, 17, box, tau, W.HE4_LAMBDA, 0)
    o.set_pa(O.PairAction.tricubic(qg, yg, tg, tau, umat, dumat, pg, pot))
    o.set_path(path)
    d = P.PathData(n, 17, box, tau, W.HE4_LAMBDA, 0)
    d.pa_tricubic(qg, yg, tg, tau, umat, dumat, pg, pot)
    d.set_path(path)
    ref, got, stats = run_trace_pair(o, d, 3, 5, 12, 43 + n, precision=precision)
    compare_traces(ref, got, stats)
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("precision", [P.FP64, P.MIXED])
@pytest.mark.parametrize("kcut", [0.5, 0.65, 1.30, 1.38, 1.94, 1.98])
def test_jellium_counts_its_k_vectors(kcut, precision):
    """Work 88 + 18 a k-vector with 3, 9, 61, 73, 194 and 218 of them: 142, 250, 1186, 1402, 3580, 4012."""
    o, d, m, levels = jellium_moves(n=12, kcut=kcut)
    o.bisection_config(3, 4, use_longrange=True)
    o.rng_seed(5)
    ref = o.run_bisection(20)
    bb = P.BisectionBlock(d, 3, 4, use_longrange=True, precision=precision)
    bb.seed(5)
    got, stats = bb.MakeMoves(20)
    compare(ref, got, stats)
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    rk = o.rhok(0)
    assert np.max(np.abs(d.get_rhok(P.OLDMODE) - rk)) < 1e-9 * np.max(np.abs(rk))
    d.close()
