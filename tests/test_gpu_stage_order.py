"""The device moves at every count of warps, where the order of a stage's warps matters: which warps evaluate, sum the
kinetic links, sample and speculate changes at 4 and at 6 warps, and with concurrent proposals.  Each case's accept
trace and path equal the oracle's; the tolerances are test_gpu_parity's."""
import numpy as np
import pytest

import oracle as O
import pimcplusplus_b200 as P
from pimcplusplus_b200 import workloads as W

from helpers import lj_case
from test_gpu_parity import compare_traces, run_trace_pair
from test_gpu_proposals import _c5_pair, _compare

pytestmark = pytest.mark.gpu

WARPS = [2, 3, 4, 5, 6, 7, 8, 12, 15, 16]


def system(tmp_path, n, m=16, levels=3, seed=5):
    cfg, tau, box, dm = lj_case(tmp_path, n=n, m=m, levels=levels)
    path = W.lattice_path(n, m + 1, box, np.random.default_rng(seed))
    o = O.System(n, m + 1, box, tau, W.HE4_LAMBDA, 0)
    o.set_pa(O.PairAction.from_dm(dm, tau, 0))
    o.set_path(path)
    d = P.PathData(n, m + 1, box, tau, W.HE4_LAMBDA, 0)
    d.set_path(path)
    d.pa_david_from_dm(dm, 0)
    return o, d


@pytest.mark.parametrize("cluster", [1, 3])
@pytest.mark.parametrize("warps", WARPS)
@pytest.mark.parametrize("n", [2, 40])
def test_stream_table_refills(tmp_path, n, warps, cluster):
    """Many moves, so many refills of the table of the stream; below 4 warps, and where two atoms leave the same one to
    be drawn again after an accepted move, the next move is not speculated and its draws start behind the refill."""
    o, d = system(tmp_path, n)
    ref, got, stats = run_trace_pair(o, d, 3, 5, 80, 23 + warps, cluster_ctas=cluster, threads_per_cta=32 * warps)
    compare_traces(ref, got, stats)
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("warps", [2, 4, 6, 8])
def test_stream_table_refills_proposals(tmp_path, warps):
    o, d, L = _c5_pair(tmp_path, 64, 128, 17)
    o.bisection_config(L, 20)
    o.rng_seed(19)
    bb = P.BisectionBlock(d, L, 20, schedule=P.PROPOSALS, cluster_ctas=4, threads_per_cta=32 * warps)
    bb.seed(19)
    got, stats = bb.MakeMoves(3)
    live, acc = _compare(list(o.run_proposals(3, 4)), got)
    assert stats["moves"] == len(live) and stats["status"] == 0 and stats["redone"] > 0
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()
