"""The filters and the smoothed Heaviside projection at the ends of their range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = (24, 12, 10)
NEL = 24 * 12 * 10


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
