"""The cases of test_gpu_vcycle_tail.py under a load that acts at its time steps (the
sine of that file is zero at whole times), and V-cycles without extra smoothing steps
(smooth = 0: the first step from zero, the coarse correction, no step after it).

Tolerances: as there.  With smooth = 0 the iterations of the FP32 V-cycle are held to
those of the FP64 one and one more a solve: a cycle without its coarse correction, all
that is left to it, needs two more a solve.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
M6 = (1e-9, 1.0, 1e-3, 1.0, 3.0, 1.0)


@pytest.mark.parametrize("n,nlvls,smooth", [((4, 4, 4), 3, 3), ((16, 8, 8), 3, 1), ((24, 24, 24), 3, 2),
                                            ((28, 28, 12), 3, 3), ((36, 16, 16), 3, 3), ((28, 12, 12), 3, 2),
                                            ((28, 16, 28), 3, 3), ((16, 8, 8), 3, 0), ((24, 24, 24), 3, 0)])
def test_vcycle_tail_under_load(gpu, n, nlvls, smooth):
    from topopt_in_petsc_transient_gb300 import LinearElasticity
    kw = dict(ncp=1, tsc=3, t1=3.0, objective=3, loadsignal=0, dalpha=0.0, dbeta=1e-3)
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
        assert st["step_precond"] == 0 and st["cg_iterations"] > 0
        its.append((st["cg_iterations"], st["solves"] + (2 * st["replacements"] if smooth else 0)))
        if mixed:
            rc, fx_r, df_r = O.LinearElasticity(*n, **kw).objective_sensitivities(x)
            assert rc == 0 and fx_r != 0.0
            assert abs(fx - fx_r) <= 1e-6 * abs(fx_r)
            assert np.abs(df - df_r).max() <= 1e-6 * np.abs(df_r).max()
    assert its[0][0] <= its[1][0] + its[0][1], its
