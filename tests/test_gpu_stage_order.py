"""The device moves at every count of warps, where the order of a stage's warps matters: which warps evaluate, sum the
kinetic links, sample and speculate changes at 4 and at 6 warps, and with concurrent proposals.  Each case's accept
trace and path equal the oracle's; the tolerances are test_gpu_parity's."""
import numpy as np
import pytest

import oracle as O
import pimcplusplus_b200 as P
from pimcplusplus_b200 import workloads as W

from helpers import lj_case
from test_gpu_batch import make_chains, oracle_run
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


@pytest.mark.parametrize("cluster", [1, 3])
@pytest.mark.parametrize("warps", WARPS)
def test_every_stage_reevaluated(tmp_path, warps, cluster):
    """The relative guard re-evaluates stage after stage in FP64; warps without a part in that pass it by."""
    o, d = system(tmp_path, 40)
    ref, got, stats = run_trace_pair(o, d, 3, 4, 60, 11, precision=P.MIXED, guard=P.GUARD_RELATIVE,
                                     cluster_ctas=cluster, threads_per_cta=32 * warps)
    compare_traces(ref, got, stats)
    assert stats["reevaluated"] > 0.5 * stats["stages_attempted"]
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("warps", [2, 4, 6, 8])
def test_every_stage_reevaluated_proposals(tmp_path, warps):
    o, d, L = _c5_pair(tmp_path, 64, 128, 17)
    o.bisection_config(L, 3)
    o.rng_seed(19)
    bb = P.BisectionBlock(d, L, 3, schedule=P.PROPOSALS, cluster_ctas=4, threads_per_cta=32 * warps,
                          precision=P.MIXED, guard=P.GUARD_RELATIVE)
    bb.seed(19)
    got, stats = bb.MakeMoves(4)
    ref = list(o.run_proposals(4, 4))
    live = [(r, g) for r, g in zip(ref, got) if r.slice1 >= 0]
    assert len(ref) == len(got) and stats["moves"] == len(live) and stats["status"] == 0
    for i, (r, g) in enumerate(live):
        assert (r.slice1, r.ptcl, r.accepted, r.stages_passed) == (
            int(g["slice1"]), int(g["ptcl"]), int(g["accepted"]), int(g["stages_passed"])), i
    assert stats["reevaluated"] > 0
    assert np.max(np.abs(d.get_path(P.OLDMODE) - o.get_path(0))) < 1e-9
    d.close()


@pytest.mark.parametrize("threads,max_split", [(64, 0), (128, 0), (160, 0), (192, 0), (256, 2), (512, 1), (512, 2)])
def test_every_stage_reevaluated_batch(threads, max_split):
    chains = make_chains()
    b = P.BatchChains(chains, precision=P.MIXED, threads_per_cta=threads, ctas=5, max_split=max_split)
    b.set_guard(P.GUARD_RELATIVE)
    trace, stats = b.run(20, trace=True)
    assert stats["status"] == 0 and stats["reevaluated"] > 0.5 * stats["stages_attempted"]
    for i, c in enumerate(chains):
        ref, ref_path, _ = oracle_run(c, 20)
        for k, r in enumerate(ref):
            g = trace[i][k]
            assert (r.slice1, r.ptcl, r.accepted, r.stages_passed) == (
                int(g["slice1"]), int(g["ptcl"]), int(g["accepted"]), int(g["stages_passed"])), (i, k)
        assert np.max(np.abs(b.path(i) - ref_path)) < 1e-9, i
    b.close()
