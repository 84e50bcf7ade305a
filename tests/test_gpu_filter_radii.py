"""The PDE filter for radii of tens to thousands of elements and tolerances near
FP64's rounding, where FP32 corrections cannot finish the solve: solved as by CG in
FP64, for random and uniform fields, one and two right-hand sides.

Tolerance: with K / V >= M / V >= 1/216 (a third to a sixth an axis), a residual of
rtol |b| leaves the solution within 216 rtol |b|, and the rounding of K's rows, whose
entries are of the size of rho = R^2 / h^2 and sum to that of M, within a relative
64 eps rho; against the same system solved in the eigenvectors of its 1-D factors.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exact(n, rmin, x):
    R2, Q, W = rmin * rmin / 12.0, [], []
    for e in n:
        K, M = np.zeros((e + 1, e + 1)), np.zeros((e + 1, e + 1))
        for i in range(e):
            K[i:i + 2, i:i + 2] += [[1, -1], [-1, 1]]
            M[i:i + 2, i:i + 2] += np.array([[2, 1], [1, 2]]) / 6.0
        Li = np.linalg.inv(np.linalg.cholesky(M))
        w, q = np.linalg.eigh(Li @ K @ Li.T)
        w[0] = 0.0  # the constant
        Q.append(Li.T @ q)
        W.append(w)
    den = 1.0 + R2 * (W[2][:, None, None] + W[1][None, :, None] + W[0][None, None, :])
    x = x.reshape(n[2], n[1], n[0])
    corners = [(slice(a, a + n[2]), slice(b, b + n[1]), slice(c, c + n[0])) for a in (0, 1) for b in (0, 1) for c in (0, 1)]
    rhs = np.zeros((n[2] + 1, n[1] + 1, n[0] + 1))
    for c in corners:
        rhs[c] += 0.125 * x
    u = np.einsum("ck,bj,ai,kji->cba", Q[2].T, Q[1].T, Q[0].T, rhs, optimize=True) / den
    u = np.einsum("kc,jb,ia,cba->kji", Q[2], Q[1], Q[0], u, optimize=True)
    return sum(0.125 * u[c] for c in corners).ravel(), np.sqrt((rhs * rhs).sum())


def _check(out, n, rmin, rtol, x):
    ref, b = _exact(n, rmin, x)
    tol = 216 * rtol * b + 64 * 2.2e-16 * (1 + rmin * rmin / 12.0) * np.abs(ref).max()
    assert np.abs(out - ref).max() <= tol


@pytest.mark.parametrize("n,rmin,rtol,uniform", [
    ((48, 24, 24), 16.0, 1e-10, False), ((48, 24, 24), 128.0, 1e-13, False), ((48, 24, 24), 256.0, 1e-12, False),
    ((48, 24, 24), 256.0, 1e-13, False), ((48, 24, 24), 2048.0, 1e-10, False), ((96, 48, 48), 1000.0, 1e-10, False),
    ((32, 16, 16), 2048.0, 1e-10, True), ((16, 8, 8), 1e5, 1e-10, True), ((1, 1, 1), 1e4, 1e-10, False),
    ((17, 1, 40), 512.0, 1e-12, False)])
def test_large_radii(gpu, n, rmin, rtol, uniform):
    from topopt_in_petsc_transient_gb300 import Filter, PDEFilt
    nel = int(np.prod(n))
    x = np.full(nel, 0.3) if uniform else np.random.default_rng(nel).random(nel)
    out = np.zeros(nel)
    PDEFilt(*n, rmin, rtol=rtol).FilterProject(x, out)
    _check(out, n, rmin, rtol, x)
    # two right-hand sides, and a third of zeros
    f = Filter(*n, 2, rmin, rtol=rtol)
    df, dg = -x ** 4, np.concatenate([np.full(nel, 1.0 / nel), np.zeros(nel)])
    df1, dg1 = df.copy(), dg.copy()
    f.Gradients(x, x, df1, 2, dg1, False, 1.0, 0.5)
    _check(df1, n, rmin, rtol, df)
    _check(dg1[:nel], n, rmin, rtol, dg[:nel])
    assert not dg1[nel:].any()


def test_iteration_limit_counts_fp64_iterations(gpu):
    from topopt_in_petsc_transient_gb300 import PDEFilt, _lib
    n, x, out = (48, 24, 24), np.random.default_rng(1).random(48 * 24 * 24), np.zeros(48 * 24 * 24)
    PDEFilt(*n, 32.0, maxit=150).FilterProject(x, out)  # CG in FP64 takes 127
    _check(out, n, 32.0, 1e-10, x)
    with pytest.raises(_lib.TopoError):
        PDEFilt(*n, 32.0, maxit=60).FilterProject(x, out)


@pytest.mark.parametrize("h,scale", [(1.0, 1.0), (1e-3, 1e155), (1e-3, 1e-140), (1e3, 1e-160), (1e3, 1e140)])
def test_range_of_fields(gpu, h, scale):
    """|b| with the element volume in T, V |T x|, is from 1e-150 to 1e148 here."""
    from topopt_in_petsc_transient_gb300 import PDEFilt
    n, x = (16, 8, 8), np.random.default_rng(5).random(16 * 8 * 8)
    out = np.zeros(x.size)
    PDEFilt(*n, 2.0 * h, h=(h, h, h)).FilterProject(scale * x, out)
    _check(out / scale, n, 2.0, 1e-10, x)


@pytest.mark.parametrize("scale", [1e-157, 1e-161, 1e-165])
def test_fields_that_underflow_end(gpu, scale):
    """Sums of squares below FP64's range: an error or a result, and the filter works on."""
    from topopt_in_petsc_transient_gb300 import PDEFilt, _lib
    n, x = (16, 8, 8), np.random.default_rng(5).random(16 * 8 * 8)
    f, out = PDEFilt(*n, 2.0), np.zeros(x.size)
    try:
        f.FilterProject(scale * x, out)
    except _lib.TopoError:
        pass
    f.FilterProject(x, out)
    _check(out, n, 2.0, 1e-10, x)
