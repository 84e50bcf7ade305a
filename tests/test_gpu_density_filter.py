"""The density and sensitivity filters over the widths of their stencils: each
marched half-width (2, 3, 4), the general one (5), meshes thinner than the
stencil, patches with a remainder, unequal element edges, odd column counts.

Tolerance: an output is a sum of at most 11^3 positive-weighted terms with
quotients and one projection: 1e-12 of the largest value, as in the parity test.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300)


@pytest.mark.parametrize("ftype", [0, 1])
@pytest.mark.parametrize("n,R,h", [((1, 1, 1), 2.5, (1.0, 1.0, 1.0)), ((70, 3, 2), 2.1, (1.0, 1.0, 1.0)),
                                   ((3, 41, 9), 3.4, (1.0, 1.0, 1.0)), ((2, 150, 3), 4.9, (1.0, 1.0, 1.0)),
                                   ((33, 17, 12), 2.5, (1.0, 2.0, 0.6)), ((9, 8, 7), 5.5, (1.0, 1.0, 1.0)),
                                   ((6, 5, 4), 1.5, (1.0, 1.0, 1.0))])
def test_density_filter_widths(gpu, ftype, n, R, h):
    from topopt_in_petsc_transient_gb300 import Filter
    nel = int(np.prod(n))
    rng = np.random.default_rng(nel)
    x = 0.05 + 0.9 * rng.random(nel)
    f = Filter(*n, ftype, R, h=h)
    for proj in (False, True):
        xt, xp = np.zeros(nel), np.zeros(nel)
        f.FilterProject(x, xt, xp, proj, 4.0, 0.5)
        xt_r, xp_r = O.dens_filter_project(*n, ftype, x, R, proj, 4.0, 0.5, h=h)
        assert _rel(xt, xt_r) < 1e-12 and _rel(xp, xp_r) < 1e-12
        df, dg = rng.standard_normal(nel), rng.standard_normal(2 * nel)
        df1, dg1 = df.copy(), dg.copy()
        f.Gradients(x, xt, df1, 2, dg1, proj, 4.0, 0.5)
        for c in range(2):
            df_r, dg_r = O.dens_filter_gradients(*n, ftype, x, xt_r, df, dg[c * nel:(c + 1) * nel], R, proj, 4.0, 0.5,
                                                 h=h)
            assert _rel(dg1[c * nel:(c + 1) * nel], dg_r) < 1e-12
        assert _rel(df1, df_r) < 1e-12
