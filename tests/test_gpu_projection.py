"""The smoothed Heaviside projection at the ends of its range: void and solid
densities are kept exactly, by every filter, and the result stays in [0, 1]; with
eta = 0 and with a small beta it is as accurate as its hyperbolic tangents.

Tolerance of the values: two tangents to 2.2e-16, their sum and a quotient on each
side: 2e-15, relative where eta = 0 leaves one tangent.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = (24, 12, 10)
NEL = 24 * 12 * 10
PARAMS = [(b, e) for b in (0.1, 1.0, 2.0, 3.0, 4.0, 6.0, 8.0, 16.0, 48.0) for e in (0.0, 0.2, 0.3, 0.5, 0.7, 1.0)]


@pytest.mark.parametrize("n", [N, (5, 33, 2)])
@pytest.mark.parametrize("R,h", [(2.5, (1.0, 1.0, 1.0)), (3.4, (1.0, 1.0, 1.0)), (4.9, (1.0, 1.0, 1.0)),
                                 (5.5, (1.0, 1.0, 1.0)), (0.3, (0.1, 0.1, 0.1)), (2.3, (1.0, 0.7, 0.5))])
def test_solid_density_is_kept(gpu, n, R, h):
    """H 1 / (H 1) is 1 to the bit when both are the same sum."""
    from topopt_in_petsc_transient_gb300 import Filter
    nel = int(np.prod(n))
    xt, xp = np.zeros(nel), np.zeros(nel)
    Filter(*n, 1, R, h=h).FilterProject(np.ones(nel), xt, xp, False, 1.0, 0.5)
    assert (xt == 1.0).all()


def _project(f, x, beta, eta):
    xt, xp = np.zeros(NEL), np.zeros(NEL)
    f.FilterProject(x, xt, xp, True, beta, eta)
    return xt, xp


@pytest.mark.parametrize("ftype,R", [(0, 2.5), (1, 0.9), (1, 2.5), (1, 3.4), (1, 4.9), (1, 5.5), (2, 2.0)])
def test_void_and_solid_are_kept(gpu, ftype, R):
    from topopt_in_petsc_transient_gb300 import Filter
    f = Filter(*N, ftype, R)
    half = np.zeros((N[2], N[1], N[0]))
    half[:, :, N[0] // 2:] = 1.0
    for beta, eta in PARAMS:
        xt, xp = _project(f, np.zeros(NEL), beta, eta)
        assert not xt.any() and not xp.any(), (beta, eta)
        assert not _project(f, -np.zeros(NEL), beta, eta)[1].any(), (beta, eta)
        if ftype != 2:  # (the PDE filter's solid is 1 to its solve's tolerance)
            xt, xp = _project(f, np.ones(NEL), beta, eta)
            assert (xt == 1.0).all() and (xp == 1.0).all(), (beta, eta)
        xt, xp = _project(f, half.ravel(), beta, eta)
        assert xp.min() >= 0.0 and xp.max() <= 1.0, (beta, eta)
        assert not xp[xt == 0.0].any() and (xp[xt == 1.0] == 1.0).all(), (beta, eta)


@pytest.mark.parametrize("beta,eta", [(1.0, 0.0), (4.0, 0.0), (1e-3, 0.5), (1e-6, 0.3), (0.1, 0.5), (64.0, 0.5)])
def test_accuracy_of_the_projection(gpu, beta, eta):
    from topopt_in_petsc_transient_gb300 import Filter
    x = np.concatenate([np.logspace(-12, 0, NEL // 2), np.linspace(0, 1, NEL - NEL // 2)])
    _, xp = _project(Filter(*N, 1, 0.9), x, beta, eta)
    ref = (np.tanh(beta * eta) + np.tanh(beta * (x - eta))) / (np.tanh(beta * eta) + np.tanh(beta * (1.0 - eta)))
    assert (np.abs(xp - ref) <= 2e-15 * (ref if eta == 0.0 else 1.0)).all()


def test_fractional_penalty_on_projected_void(gpu):
    from topopt_in_petsc_transient_gb300 import Filter, LinearElasticity
    n = (8, 4, 4)
    x = np.zeros((4, 4, 8))
    x[:, :, :5] = 1.0
    f = Filter(*n, 1, 1.5)
    for beta, eta in PARAMS:
        xt, xp = np.zeros(128), np.zeros(128)
        f.FilterProject(x.ravel(), xt, xp, True, beta, eta)
        le = LinearElasticity(*n, nlvls=2, mixed=False, ncp=1, tsc=2, t1=0.5, objective=3, loadsignal=1, dalpha=0.0,
                              dbeta=1e-3)
        le.CompleteInitialState(xp, 1e-3, 1.0, 1e-3, 1.0, 2.5, 1.0)
        le.GenerateCheckPoints()
        df = np.zeros(128)
        assert np.isfinite(le.ComputeObjectiveSensitivities(df)) and np.isfinite(df).all(), (beta, eta)
