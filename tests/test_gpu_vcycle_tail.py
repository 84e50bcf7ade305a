"""The V-cycle's last smoothed level and coarse solve as one cluster: levels of 1
to 16 bricks (1, 2, 3, 8, 9 and 12: full and partly idle clusters), 18 (the separate
kernels), one to three smoothing steps.

Tolerance: the solve converges on the FP64 residual (rtol 1e-11); with a condition
number of up to 1e5 (density contrast 64, 36 elements) the sensitivities are
within 1e-6 of the oracle's whatever the preconditioner does.  That it is the
V-cycle is checked by the iterations: those of the FP64 V-cycle, two more for each
replacement of the residual, at which the recurrence starts anew, and one a solve.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
M6 = (1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)


@pytest.mark.parametrize("n,nlvls,smooth", [((4, 4, 4), 3, 3), ((16, 8, 8), 3, 1), ((24, 24, 24), 3, 2),
                                            ((28, 28, 12), 3, 3), ((36, 16, 16), 3, 3), ((28, 12, 12), 3, 2),
                                            ((28, 16, 28), 3, 3)])
def test_vcycle_tail(gpu, n, nlvls, smooth):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    kw = dict(ncp=1, tsc=3, t1=3.0, objective=3, loadsignal=1, dalpha=0.0, dbeta=1e-3)
    x = 0.2 + 0.6 * np.random.default_rng(sum(n)).random(np.prod(n))
    its = []
    for mixed in (True, False):
        le = LinearElasticity(*n, nlvls=nlvls, mixed=mixed, rtol=1e-11, sens_fp32=False, smooth=smooth,
                              mass_precond=0, adaptive_kappa=0.0, **kw)
        le.CompleteInitialState(x, *M6)
        le.GenerateCheckPoints()
        df = np.zeros(x.size)
        fx = le.ComputeObjectiveSensitivities(df)
        st = le.stats()
        assert st["step_precond"] == 0
        its.append((st["cg_iterations"], 2 * st["replacements"] + st["solves"]))
        if mixed:
            rc, fx_r, df_r = O.LinearElasticity(*n, **kw).objective_sensitivities(x)
            assert rc == 0
            assert abs(fx - fx_r) <= 1e-6 * abs(fx_r)
            assert np.abs(df - df_r).max() <= 1e-6 * np.abs(df_r).max()
    assert its[0][0] <= its[1][0] + its[0][1]
