"""More smoothing steps than the Chebyshev table has rows (64): the V-cycle goes on
with the last row, and the solves converge to the oracle's result.

Tolerance: the solve's (rtol 1e-11, condition number up to 1e5): 1e-6.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mixed", [True, False])
@pytest.mark.parametrize("smooth,coarse_smooth,coarse_dense_max", [(70, 12, None), (3, 90, 0), (200, 12, None)])
def test_more_steps_than_the_table(gpu, mixed, smooth, coarse_smooth, coarse_dense_max):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    n, kw = (16, 8, 8), dict(ncp=1, tsc=3, t1=3.0, objective=3, loadsignal=0, dalpha=0.0, dbeta=1e-3)
    x = 0.2 + 0.6 * np.random.default_rng(2).random(np.prod(n))
    le = LinearElasticity(*n, nlvls=3, mixed=mixed, rtol=1e-11, sens_fp32=False, smooth=smooth, mass_precond=0,
                          coarse_smooth=coarse_smooth, coarse_dense_max=coarse_dense_max, adaptive_kappa=0.0, **kw)
    le.CompleteInitialState(x, 1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)
    le.GenerateCheckPoints()
    df = np.zeros(x.size)
    fx = le.ComputeObjectiveSensitivities(df)
    rc, fx_r, df_r = O.LinearElasticity(*n, **kw).objective_sensitivities(x)
    assert rc == 0 and fx_r != 0.0
    assert abs(fx - fx_r) <= 1e-6 * abs(fx_r)
    assert np.abs(df - df_r).max() <= 1e-6 * np.abs(df_r).max()
