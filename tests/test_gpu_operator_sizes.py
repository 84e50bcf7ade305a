"""The FP64 operator kernel (columns of elements marched along z) at sizes where
its patches and runs change: one element, patches with a remainder along x and
y, runs of one layer, equal and unequal element edges; and the Kronecker
preconditioner's lines shorter than its band.

Tolerance: a node sums at most 8 element products of 24 terms in FP64: 1e-13 of
the largest value, as in the parity test.  The preconditioned solve is checked
by the state it leaves: rtol 1e-12 of a mass-dominated operator, 1e-10.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
M6 = (1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)


def _rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("h", [(1.0, 1.0, 1.0), (0.5, 1.25, 2.0)])
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (15, 7, 2), (16, 8, 4), (31, 3, 5), (33, 12, 2), (7, 40, 6)])
def test_fp64_operator_sizes(gpu, n, h):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    rng = np.random.default_rng(sum(n))
    x = 0.1 + 0.8 * rng.random(np.prod(n))
    le = LinearElasticity(*n, nlvls=1, ncp=1, tsc=2, t1=0.02, mixed=False, h=h)
    le.CompleteInitialState(x, *M6)
    ref = O.LinearElasticity(*n, ncp=1, tsc=2, t1=0.02, hx=h[0], hy=h[1], hz=h[2])
    ref.CompleteInitialState(x)
    v = rng.standard_normal(le.ndof)
    for a, b in zip(le.apply_km(v), ref.apply_KM(v)):
        assert _rel(a, b) < 1e-13


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [(3, 2, 2), (18, 15, 16), (25, 7, 34)])
def test_kronecker_line_ends(gpu, n, mixed):
    # lines of 3 to 35 nodes against a band of 17 taps
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    kw = dict(ncp=1, tsc=3, t1=0.03, objective=3, loadsignal=1, dalpha=0.0, dbeta=1e-3)
    x = 0.12 + 0.04 * np.random.default_rng(5).random(np.prod(n))
    le = LinearElasticity(*n, nlvls=1, mixed=mixed, rtol=1e-12, sens_fp32=False, **kw)
    le.CompleteInitialState(x, *M6)
    le.GenerateCheckPoints()
    df = np.zeros(x.size)
    fx = le.ComputeObjectiveSensitivities(df)
    assert le.stats()["step_precond"] == 1
    rc, fx_r, df_r = O.LinearElasticity(*n, **kw).objective_sensitivities(x)
    assert rc == 0
    assert abs(fx - fx_r) <= 1e-10 * abs(fx_r) and _rel(df, df_r) < 1e-9
