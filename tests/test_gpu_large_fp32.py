"""FP32 stage kernels on more tiles than the device holds at once, where a
CTA prefetches the tile a device of CTAs ahead: one step against FP64 from the
same state, on a tile count with a ragged end.  The tolerance is the FP32
form's own (1e-5 relative), as in the parity tests."""
import numpy as np
import pytest

from helpers import rel_err
from rkdg_heter_calculate_b200 import CUDARkdgSolver, meshgen, vortex

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,flux,limiter", [(2, "hllc", None), (2, "llf", None), (1, "llf", None),
                                                (1, "llf", "tvb")])
def test_fp32_beyond_one_wave_of_tiles(order, flux, limiter):
    n = 401  # 321,602 triangles, 2,513 tiles
    mesh = meshgen.periodic_structured(n, n, jitter=0.15, seed=4)
    nb = 3 if order == 1 else 6
    U = vortex.project_native(mesh, lambda X, Y: vortex.exact(X, Y, 0.0, 5.0, 1.4, 1.0, 1.0), nb, n=3)
    kw = dict(order=order, flux=flux, limiter=limiter, cfl=0.2, farfield=(1.0, 1.0, 1.0, 3.5))
    kw.update(dict(nq=3, ng=2) if order == 1 else dict(nq=6, ng=3))
    out = {}
    for precision in ("fp64", "fp32", "fp32c"):
        s = CUDARkdgSolver(mesh, precision=precision, **kw)
        s.setFreedom(U, basis="native")
        for _ in range(2):
            s.step()
        out[precision] = s.copyFreedomToHost(basis="native")
        s.close()
    assert np.isfinite(out["fp64"]).all()
    assert rel_err(out["fp32"], out["fp64"]) < 1e-5
    assert rel_err(out["fp32c"], out["fp64"]) < 1e-5
