"""rho_k of every slice (PathClass::CalcRho_ks_Fast, PathClass.cc:616-647) against the plain sum over
particles of e^{ik.r}, at the edges of the kernel's split: particles per block of a cluster (one below,
at and above a share), shares of more than one batch of phase tables, and k-vectors per thread."""
import numpy as np
import pytest

import pimcplusplus_b200 as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,slices,side,kcut", [
    (2, 2, 7.0, 1.0),       # no split, fewer k-vectors than a warp
    (15, 3, 9.0, 2.0), (16, 3, 9.0, 2.0), (17, 3, 9.0, 2.0),    # one block / two blocks per slice
    (63, 5, 11.0, 2.5), (64, 5, 11.0, 2.5), (65, 5, 11.0, 2.5),  # four / eight blocks per slice
    (129, 600, 8.0, 2.0),   # slices alone fill the GPU: one block per slice, two batches
    (1500, 2, 20.0, 1.3),   # eight blocks, several batches each
    (40, 4, 12.0, 3.2),     # two k-vectors per thread
    (40, 4, 12.0, 4.1),     # four
    (21, 3, (4.0, 60.0, 5.0), 3.0),  # uneven box: long table in one dimension
])
def test_rhok_full_against_direct_sum(n, slices, side, kcut):
    box = np.array(side if isinstance(side, tuple) else [side] * 3)
    rng = np.random.default_rng(n * 1000 + slices)
    path = (rng.random((slices, n, 3)) - 0.5) * box * 2.5  # some positions outside the box
    d = P.PathData(n, slices, box, 0.1, 1.0)
    nk = d.setup_kvecs(kcut)
    assert 0 < nk <= 1024
    d.set_path(path)
    d.calc_rhok()
    got = d.get_rhok(P.OLDMODE)
    k = d.kvecs()
    phase = path @ k.T
    ref = np.sum(np.exp(1j * phase), axis=1)
    # a term: the phase's rounding (argument times 2^-53, here and in the reference), the powers of
    # e^{i k_d x_d} (one complex product each, 3 * 2^-53), and the sum over n terms of magnitude 1
    kmax = np.max(np.ceil(1.1 * kcut * box / (2 * np.pi)))
    tol = n * (4 * np.max(np.abs(phase)) + 12 * kmax + n) * 2.0 ** -53
    assert np.max(np.abs(got - ref)) <= tol
    assert np.array_equal(got, d.get_rhok(P.NEWMODE))
    d.close()
