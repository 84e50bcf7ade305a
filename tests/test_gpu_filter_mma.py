"""The cooperative kernels of the PDE filter and of MMA at the sizes where their
layouts change: fewer nodes than a patch, patches with a remainder, two nodes
along an axis, one and two right-hand sides, element boxes with unequal edges;
design vectors below, at and above one CTA, one and two constraints.

Tolerances.  Filter: solves to rtol 1e-13 of a system whose Jacobi-scaled
condition number stays below 1e2 for these radii, against an oracle at 1e-14:
1e-10 of the largest value leaves a factor of ten.  MMA: the update and the
oracle differ by the rounding of sums of at most 1e3 terms and of a Newton
iteration that ends at the same step: 1e-10 of the largest value, as in the
parity test.
"""
import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("n,h,rmin", [((1, 1, 1), (1.0, 1.0, 1.0), 2.0), ((31, 9, 1), (1.0, 1.0, 1.0), 2.0),
                                      ((1, 40, 13), (1.0, 0.5, 2.0), 1.5), ((64, 8, 5), (0.7, 1.3, 1.0), 3.0),
                                      ((70, 17, 19), (1.0, 1.0, 1.0), 1.2)])
def test_filter_solve_sizes(gpu, n, h, rmin):
    from topopt_in_petsc_transient_gb300 import Filter
    rng = np.random.default_rng(sum(n))
    x = rng.random(np.prod(n))
    f = Filter(*n, 2, rmin, h=h, rtol=1e-13)
    xt_r, xp_r = O.filter_project(*n, x, rmin, True, 4.0, 0.3, h=h)
    xt, xp = np.zeros_like(x), np.zeros_like(x)
    f.FilterProject(x, xt, xp, True, 4.0, 0.3)
    assert _rel(xt, xt_r) < 1e-10 and _rel(xp, xp_r) < 1e-10
    # 1 + m right-hand sides in batches of two, in place; the all-zero one is done at once
    df, dg = rng.standard_normal(x.size), np.concatenate([np.full(x.size, 1.0 / x.size), np.zeros(x.size)])
    df_r, dg_r = O.filter_gradients(*n, xt_r, df.copy(), dg[:x.size].copy(), rmin, True, 4.0, 0.3, h=h)
    f.Gradients(x, xt, df, 2, dg, True, 4.0, 0.3)
    assert _rel(df, df_r) < 1e-10 and _rel(dg[:x.size], dg_r) < 1e-10
    assert not dg[x.size:].any()


def test_filter_accepts_tolerances_below_rounding(gpu):
    from topopt_in_petsc_transient_gb300 import PDEFilt
    n = (16, 8, 8)
    x = np.random.default_rng(3).random(np.prod(n))
    out = np.zeros_like(x)
    PDEFilt(*n, 2.0, rtol=1e-18).FilterProject(x, out)
    assert _rel(out, O.pde_filter(*n, x, 2.0)) < 1e-10


@pytest.mark.parametrize("n,m", [(1, 1), (255, 1), (256, 2), (257, 1), (1000, 2)])
def test_mma_update_sizes(gpu, n, m):
    from topopt_in_petsc_transient_gb300 import MMA
    rng = np.random.default_rng(n + m)
    c = rng.random(n)
    x = np.full(n, 0.5)
    mo, mg = O.MMA(n, m, x), MMA(n, m)
    mo.SetAsymptotes(0.1, 0.6, 1.05)
    mg.SetAsymptotes(0.1, 0.6, 1.05)
    xo, xg = x.copy(), torch.tensor(x, device="cuda")
    lo, hi = torch.zeros_like(xg), torch.zeros_like(xg)
    for it in range(5):  # the asymptotes move from the third update on
        df = 2 * (xo - c) * (1 + 0.1 * it)
        g = np.array([xo.mean() - 0.4, 0.2 - xo.mean()][:m])
        dg = np.concatenate([np.full(n, 1.0 / n), np.full(n, -1.0 / n)][:m])
        lo_r, hi_r = O.MMA.SetOuterMovelimit(0.0, 1.0, 0.2, xo)
        xprev = xo.copy()
        mo.Update(xo, df, g, dg, lo_r, hi_r)
        dfd, dgd, xold = (torch.tensor(v, device="cuda") for v in (df, dg, xprev))
        torch.cuda.synchronize()
        mg.SetOuterMovelimit(0.0, 1.0, 0.2, xg, lo, hi)
        mg.Update(xg, dfd, g, dgd, lo, hi)
        assert _rel(xg.cpu().numpy(), xo) < 1e-10, it
        assert abs(mg.DesignChange(xg, xold) - np.abs(xo - xprev).max()) < 1e-10
        assert torch.equal(xold, xg)
