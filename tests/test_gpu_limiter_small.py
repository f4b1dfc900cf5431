"""The TVB limiter with M = 0 on a field whose disturbance has decayed to the
smallest numbers of the precision, as ahead of a front in a component that is
zero in the far field: the limited increments are subnormal, and their ratio
theta = min(1, neg / pos) is a quotient of subnormals.  Limited modes stay
finite and no larger than the increments they are made of, in the limiter's own
kernel and inside the resident steps."""
import numpy as np
import pytest

from rkdg_heter_calculate_b200 import CUDARkdgSolver, meshgen

pytestmark = pytest.mark.gpu

FAR = (1.4, 4.2, 0.0, 8.8)


@pytest.mark.parametrize("precision,size", [("fp64", 1e-310), ("fp32", 1e-40), ("fp32c", 1e-40)])
@pytest.mark.parametrize("order", [1, 2])
def test_limiter_on_subnormal_increments(precision, size, order):
    mesh = meshgen.periodic_structured(20, 20, jitter=0.15, seed=4)
    nb = 3 if order == 1 else 6
    rng = np.random.default_rng(5)
    U = np.zeros((4, nb, mesh.ntri))
    U[:, 0, :] = np.array(FAR)[:, None]
    U[2] = size * rng.uniform(-1.0, 1.0, (nb, mesh.ntri))  # rho v: means and modes
    s = CUDARkdgSolver(mesh, order=order, nq=3 if order == 1 else 6, ng=2 if order == 1 else 3, flux="llf",
                       precision=precision, limiter="tvb", tvb_m=0.0, cfl=0.1, farfield=FAR)
    s.setFreedom(U, basis="native")
    s.limit()
    V = s.copyFreedomToHost(basis="native")
    assert np.isfinite(V).all()
    np.testing.assert_array_equal(V[:, 0][:2], U[:, 0][:2])
    assert np.abs(V[2]).max() < 100 * size and np.abs(V[2, 1:3]).max() > 0
    s.advance(5)
    assert np.isfinite(s.copyFreedomToHost(basis="native")).all()
    s.close()
