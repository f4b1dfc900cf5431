"""Batched independent solves: each solve in a mixed P1/P2 batch of uneven
meshes equals the same solve run alone (bit for bit, FP32 and FP64), lands
on its own final time, and matches the oracle."""
import math

import numpy as np
import pytest

from helpers import rel_err
from oracle import oracle
from rkdg_heter_calculate_b200 import CUDARkdgSolver, meshgen, vortex
from rkdg_heter_calculate_b200.batch import Batch

pytestmark = pytest.mark.gpu


def cases():
    specs = [  # (mesh, order, beta, theta)
        (meshgen.periodic_delaunay(20, seed=11), 2, 5.0, 0.3),
        (meshgen.periodic_structured(14, 14, jitter=0.2, seed=12), 1, 3.0, 1.2),
        (meshgen.periodic_delaunay(12, seed=13), 2, 2.0, 4.0),
        (meshgen.periodic_delaunay(9, seed=14), 1, 1.5, 2.5),
    ]
    out = []
    for m, order, beta, th in specs:
        ui, vi = math.sqrt(2) * math.cos(th), math.sqrt(2) * math.sin(th)
        nb = 3 if order == 1 else 6
        U = vortex.project_native(m, lambda X, Y: vortex.exact(X, Y, 0.0, beta, 1.4, ui, vi), nb)
        far = (1.0, ui, vi, 2.5 + 0.5 * (ui * ui + vi * vi))
        out.append((m, order, U, far))
    return out


def solo(m, order, U, far, precision, steps, t_final=0.0):
    kw = dict(order=2, nq=6, ng=3) if order == 2 else dict(order=1, nq=3, ng=2)
    s = CUDARkdgSolver(m, flux="hllc", rk=3, precision=precision, cfl=0.2, farfield=far, **kw)
    s.setFreedom(U, basis="native")
    t, n = s.advance(steps, t_final=t_final)
    out = s.copyFreedomToHost(basis="native")
    s.close()
    return out, t, n


@pytest.mark.parametrize("precision,shape", [("fp32", (0, 0)), ("fp32c", (0, 0)), ("fp64", (0, 0)),
                                             ("fp32", (0, 2)), ("fp32c", (3, 2)), ("fp64", (0, 2))])
def test_batch_equals_solo_runs(precision, shape):
    """Every launch shape: one launch per stage in solve order (0, 0), and
    the P2 and P1 tiles as two concurrent launches of the single-order
    kernels, one CTA per tile (0, 2) or three persistent CTAs each (3, 2)."""
    cs = cases()
    b = Batch([c[0] for c in cs], [c[1] for c in cs], precision=precision, flux="hllc", cfl=0.2,
              farfields=[c[3] for c in cs])
    b.set_shape(*shape)
    for i, c in enumerate(cs):
        b.set_state(i, c[2])
    t, n = b.advance(12)
    assert (n == 12).all()
    for i, c in enumerate(cs):
        ref, ts, ns = solo(*c, precision, 12)
        np.testing.assert_array_equal(b.state(i), ref, err_msg=f"solve {i}")
        assert t[i] == ts
    b.close()


def test_batch_final_times_and_autotune():
    cs = cases()
    b = Batch([c[0] for c in cs], [c[1] for c in cs], precision="fp32", flux="hllc", cfl=0.2,
              farfields=[c[3] for c in cs])
    for i, c in enumerate(cs):
        b.set_state(i, c[2])
    ctas, order, tile = b.autotune()
    assert ctas >= 0 and order in (0, 1, 2) and tile in (128, 256)
    # a solve alone runs 128-element tiles: bit-for-bit equality holds at the same tile size
    b.set_tile(128)
    tf = np.array([0.05, 0.11, 0.02, 0.3])
    t, n = b.advance(100000, t_final=tf)
    np.testing.assert_array_equal(t, tf)
    for i, c in enumerate(cs):
        ref, ts, ns = solo(*c, "fp32", 100000, t_final=tf[i])
        assert ts == tf[i] and ns == n[i]
        np.testing.assert_array_equal(b.state(i), ref)
    b.close()


@pytest.mark.parametrize("tile", [128, 256])
def test_batch_fp64_matches_oracle(tile):
    cs = cases()
    b = Batch([c[0] for c in cs], [c[1] for c in cs], precision="fp64", flux="hllc", cfl=0.2,
              farfields=[c[3] for c in cs])
    b.set_tile(tile)
    for i, c in enumerate(cs):
        b.set_state(i, c[2])
    b.advance(6)
    for i in (1, 2):
        m, order, U, far = cs[i]
        kw = dict(order=2, nq=6, ng=3) if order == 2 else dict(order=1, nq=3, ng=2)
        o = oracle.Oracle(m, flux=oracle.HLLC, rk=3, cfl=0.2, farfield=far, **kw)
        # native -> reference basis through a single-solve context
        s = CUDARkdgSolver(m, flux="hllc", rk=3, cfl=0.2, farfield=far, **kw)
        s.setFreedom(U, basis="native")
        o.set_state(s.copyFreedomToHost(basis="reference"))
        for _ in range(6):
            o.step()
        s.setFreedom(b.state(i), basis="native")
        assert rel_err(s.copyFreedomToHost(basis="reference"), o.state()) < 1e-11
        s.close()
    b.close()


def test_stage_timing_has_the_launch_form_of_the_steps():
    """In tile order 2 a step's two chains of launches run side by side over all
    the steps of a graph; what the autotuner times must do so too.  Joined
    after every launch, the stages of this pack sum to 1.06 of a step, as two
    chains to 0.92."""
    import time

    sizes = [60 + 10 * i for i in range(16)]
    orders = [2 if i % 2 else 1 for i in range(16)]
    far = (1.0, 1.0, 1.0, 3.5)
    b = Batch([meshgen.periodic_structured(n, n, jitter=0.15, seed=n) for n in sizes], orders, precision="fp32c",
              flux="hllc", cfl=0.2, farfields=[far] * 16)
    b.set_shape(0, 2)
    for i, n in enumerate(sizes):
        U = np.zeros((4, 6 if orders[i] == 2 else 3, 2 * n * n))
        U[:, 0] = np.array(far)[:, None]
        b.set_state(i, U)
    b.advance(96)
    step = math.inf
    for _ in range(8):
        t0 = time.perf_counter()
        b.advance(96)
        step = min(step, (time.perf_counter() - t0) / 96 * 1e3)
    stages = sum(min(b.time_stage(k, 20) for _ in range(8)) for k in range(3))
    b.close()
    assert stages < step, (stages, step)
