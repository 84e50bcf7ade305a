"""FP64 bricks of 3x3x3 and 7x7x5 nodes (basis solves whose vectors are stored in
FP32): grids of one brick, with remainders in every direction, of more bricks than
SMs, and two whose fine level takes bricks of 7x7x5, with remainders and without.

Tolerance: the basis vectors of both modes solve the same FP64 systems to rtol
1e-13; the first row of the mixed one is that of the plain path rounded to FP32,
2^-24 of a value, and each solve may differ by one iteration at the threshold.
The shift lies below the first eigenfrequency of every grid: with one above it
P0 = K - om^2 M is indefinite and the solves are refused.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
M6 = (1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)


@pytest.mark.parametrize("n,nlvls", [((2, 2, 2), 2), ((6, 2, 4), 2), ((8, 4, 4), 3), ((28, 16, 12), 3),
                                     ((44, 24, 24), 3), ((48, 24, 24), 4)])
def test_small_bricks(gpu, n, nlvls):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    x = 0.3 + 0.1 * np.random.default_rng(sum(n)).random(np.prod(n))
    rows, its = [], []
    for mixed in (True, False):
        le = LinearElasticity(*n, nlvls=nlvls, ncp=1, tsc=2, t1=0.08, objective=3, loadsignal=1, dalpha=1e-3,
                              dbeta=1e-3, mixed=mixed, rtol=1e-13, reduction=True, basis=2, omega0=1e-4)
        s0 = le.stats()
        le.CompleteInitialState(x, *M6)
        s1 = le.stats()
        rows.append(np.asarray(le.reduced_system()[0])[0])
        its.append((s1["cg_iterations"] - s0["cg_iterations"], s1["solves"] - s0["solves"]))
    assert np.abs(rows[0] - rows[1]).max() <= 2.0 ** -23 * np.abs(rows[1]).max()
    assert its[0][1] == its[1][1] and abs(its[0][0] - its[1][0]) <= its[1][1]
