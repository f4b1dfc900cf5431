"""Whole steps in one launch (csrc/resident.cuh) against the same steps through
the stage kernels: a context made as one partition that owns the whole mesh
keeps the stage kernels and the caller's order, so with reorder=False both run
the same tiles and must give the same bits, whatever the method.  Sizes: one
tile, a ragged second one, the most tiles that run with 256 threads each (and
one more), several launches' worth of steps (64 per launch), landing on a final
time, and the residual history, which needs a launch per step."""
import numpy as np
import pytest

from rkdg_heter_calculate_b200 import CUDARkdgSolver, meshgen, vortex

pytestmark = pytest.mark.gpu

FAR = (1.0, 1.0, 1.0, 3.5)


def ordered(mesh):
    return meshgen.permute(mesh, meshgen.locality_order(mesh))


def start(mesh, nb, far, kind):
    if kind == "vortex":
        return vortex.project_native(mesh, lambda X, Y: vortex.exact(X, Y, 0.0, 5.0, 1.4, 1.0, 1.0), nb, n=3)
    U = np.zeros((4, nb, mesh.ntri))  # a jump that the limiter acts on
    c = mesh.coords().mean(axis=1)
    scale = np.where(c[:, 0] < np.median(c[:, 0]), 1.0, 1.6)
    for v in range(4):
        U[v, 0] = far[v] * scale
    return U


def both(mesh, U, far, steps, t_final=0.0, **kw):
    out = []
    for whole in (None, mesh.ntri):
        s = CUDARkdgSolver(mesh, farfield=far, reorder=False, n_owned=whole, **kw)
        s.setFreedom(U, basis="native")
        reached = s.advance(steps, t_final=t_final)
        monitored = s.step()
        out.append((s.copyFreedomToHost(basis="native"), reached, s.time(), monitored[0], tuple(monitored[1])))
        s.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    assert np.isfinite(out[0][0]).all()
    assert out[0][1:] == out[1][1:]
    return out[0]


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32c"])
@pytest.mark.parametrize("order,nq,flux,limiter,rk", [(2, 7, "llf", None, 3), (2, 6, "hllc", None, 3),
                                                      (1, 3, "llf", None, 2), (1, 3, "hllc", "tvb", 3),
                                                      (2, 6, "llf", "tvb", 3)])
def test_resident_equals_stage_kernels(precision, order, nq, flux, limiter, rk):
    kw = dict(order=order, nq=nq, ng=2 if order == 1 else 3, flux=flux, limiter=limiter, rk=rk, precision=precision,
              cfl=0.15)
    nb = 3 if order == 1 else 6
    for n, steps in ((8, 3), (9, 70), (25, 20)):  # 128, 162 and 1250 triangles
        mesh = ordered(meshgen.periodic_structured(n, n, jitter=0.15, seed=n))
        both(mesh, start(mesh, nb, FAR, "vortex"), FAR, steps, **kw)
    # boundaries of every kind; a jump in the state where the limiter is on
    mesh = ordered(meshgen.channel(40, 16))
    far = (1.4, 4.2, 0.0, 8.8)
    both(mesh, start(mesh, nb, far, "jump"), far, 10, **kw)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n", [97, 98, 137])  # 148, 151 and 294 tiles
def test_resident_at_the_edges_of_its_forms(precision, n):
    mesh = ordered(meshgen.periodic_structured(n, n, jitter=0.15, seed=3))
    both(mesh, start(mesh, 6, FAR, "vortex"), FAR, 5, order=2, nq=6, ng=3, flux="hllc", precision=precision, cfl=0.2)


def test_resident_final_time_and_history(tmp_path):
    mesh = ordered(meshgen.periodic_structured(20, 20, jitter=0.15, seed=2))
    U = start(mesh, 6, FAR, "vortex")
    kw = dict(order=2, nq=6, ng=3, flux="hllc", precision="fp64", cfl=0.2)
    _, (t, steps), _, _, _ = both(mesh, U, FAR, 1000, t_final=0.25, **kw)
    assert t == 0.25 and 64 < steps < 1000
    text = []
    for whole in (None, mesh.ntri):
        path = tmp_path / f"history_{whole}"
        s = CUDARkdgSolver(mesh, farfield=FAR, reorder=False, n_owned=whole, **kw)
        s.setFreedom(U, basis="native")
        s.setResidualLog(str(path))
        s.advance(7)
        s.setResidualLog(None)
        text.append(path.read_text())
        s.close()
    assert text[0] == text[1] and len(text[0].splitlines()) == 8


def test_resident_reports_a_non_physical_state():
    from rkdg_heter_calculate_b200.capi import RkdgError

    mesh = ordered(meshgen.periodic_structured(20, 20, jitter=0.15, seed=2))
    U = start(mesh, 6, FAR, "vortex")
    U[3, 0, 17] = -1.0
    s = CUDARkdgSolver(mesh, farfield=FAR, order=2, nq=6, ng=3, flux="hllc", cfl=0.2)
    s.setFreedom(U, basis="native")
    with pytest.raises(RkdgError) as e:
        s.advance(5)
    assert e.value.code == 4
    s.close()


def test_resident_solves_in_several_threads():
    """Launches that each fill the device, from contexts in several host
    threads: each gets the device as a whole, one after the other, and gives
    the bits it gives alone."""
    import threading

    kw = dict(order=2, nq=6, ng=3, flux="hllc", precision="fp64", cfl=0.2, farfield=FAR)
    mesh = meshgen.periodic_structured(136, 136, jitter=0.15, seed=3)
    U = start(mesh, 6, FAR, "vortex")

    def solve(out, i):
        s = CUDARkdgSolver(mesh, **kw)
        s.setFreedom(U, basis="native")
        for _ in range(4):
            s.advance(70)
        out[i] = s.copyFreedomToHost(basis="native")
        s.close()

    alone, together = [None], [None] * 4
    solve(alone, 0)
    threads = [threading.Thread(target=solve, args=(together, i)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for out in together:
        np.testing.assert_array_equal(out, alone[0])


@pytest.mark.parametrize("n", [40, 97])  # 25 and 148 tiles
def test_resident_reports_a_bad_first_time_step(n):
    """Every tile stops at the first step's dt; whichever block comes first or
    last, that is a state error, not a wait that ran out."""
    from rkdg_heter_calculate_b200.capi import RkdgError

    mesh = ordered(meshgen.periodic_structured(n, n, jitter=0.15, seed=2))
    s = CUDARkdgSolver(mesh, farfield=FAR, order=2, nq=6, ng=3, flux="hllc", cfl=0.2)
    s.setFreedom(start(mesh, 6, FAR, "vortex"), basis="native")
    for _ in range(50):
        with pytest.raises(RkdgError) as e:
            s.step(float("inf"))
        assert e.value.code == 4
    s.close()


def test_exchange_buffers_are_made_at_the_first_step():
    """A context that only forms residuals does not pay for them; a mesh far too
    large to be resident never does."""
    for n, resident in ((20, True), (400, False)):
        mesh = meshgen.periodic_structured(n, n, jitter=0.15, seed=2)
        s = CUDARkdgSolver(mesh, farfield=FAR, order=2, nq=6, ng=3, flux="hllc", precision="fp32", cfl=0.2)
        s.initRKDG()
        before = s.sizes()[2]
        s.residual(basis="native")
        staged = s.sizes()[2]
        s.advance(3)
        after = s.sizes()[2]
        assert staged - before == 0  # (the staging array came with the state)
        assert after > staged if resident else after == staged
        s.close()


def in_threads(solvers, steps, calls, out=None):
    """Each solver's advance(steps), calls times, in a thread of its own; seconds."""
    import threading
    import time

    gate = threading.Barrier(len(solvers) + 1)

    def go(s):
        gate.wait()
        for _ in range(calls):
            s.advance(steps)

    threads = [threading.Thread(target=go, args=(s,)) for s in solvers]
    for t in threads:
        t.start()
    gate.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    return time.perf_counter() - t0


@pytest.mark.parametrize("precision,order,flux,limiter", [("fp32", 1, "llf", None), ("fp32c", 2, "hllc", None),
                                                          ("fp64", 1, "llf", "tvb"), ("fp64", 2, "hllc", None)])
def test_solves_beyond_one_device(precision, order, flux, limiter):
    """More solves in flight than the device holds whole: each call takes the
    form that there is room for (256 threads per tile, 128, the stage kernels),
    changing from call to call, and the bits stay those of the solve alone."""
    kw = dict(order=order, nq=6 if order == 2 else 3, ng=3 if order == 2 else 2, flux=flux, limiter=limiter,
              precision=precision, cfl=0.1, farfield=FAR)
    mesh = meshgen.periodic_structured(100, 100, jitter=0.15, seed=3)
    U = start(mesh, 6 if order == 2 else 3, FAR, "vortex")
    solvers = [CUDARkdgSolver(mesh, **kw) for _ in range(8)]
    for s in solvers:
        s.setFreedom(U, basis="native")
    in_threads(solvers[:1], 7, 6)
    in_threads(solvers[1:], 7, 6)
    ref = solvers[0].copyFreedomToHost(basis="native")
    for s in solvers[1:]:
        np.testing.assert_array_equal(s.copyFreedomToHost(basis="native"), ref)
        assert s.time() == solvers[0].time()
        s.close()
    solvers[0].close()


@pytest.mark.parametrize("precision,order,flux", [("fp32", 1, "llf"), ("fp32", 2, "hllc")])
def test_solves_in_several_threads_share_the_device(precision, order, flux):
    """Eight threads with a solve each that alone takes half the device or more:
    queued behind one another they took 8.3 and 9.2 times as long as one, through
    the stage kernels, which fill the device together, 4.0 and 3.4 times."""
    kw = dict(order=order, nq=6 if order == 2 else 3, ng=3 if order == 2 else 2, flux=flux, precision=precision,
              cfl=0.1, farfield=FAR)
    mesh = meshgen.periodic_structured(100, 100, jitter=0.15, seed=3)
    solvers = [CUDARkdgSolver(mesh, **kw) for _ in range(8)]
    for s in solvers:
        s.initRKDG()
    in_threads(solvers, 100, 2)
    one = min(in_threads(solvers[:1], 100, 10) for _ in range(3))
    eight = min(in_threads(solvers, 100, 10) for _ in range(3))
    for s in solvers:
        s.close()
    assert eight < 6.5 * one, (eight, one)


@pytest.mark.parametrize("precision", ["fp64", "fp32", "fp32c"])
@pytest.mark.parametrize("order,nq,flux,limiter,rk", [(1, 3, "hllc", "tvb", 3), (1, 3, "llf", "tvb", 2),
                                                      (2, 7, "llf", None, 3), (2, 6, "llf", "tvb", 3),
                                                      (2, 6, "hllc", "tvb", 3), (1, 3, "llf", None, 3)])
def test_resident_with_128_threads_per_tile(precision, order, nq, flux, limiter, rk):
    """Meshes that the device holds only with 128 threads per tile: beyond one
    (FP64) and two (FP32) tiles of 256 threads per SM."""
    kw = dict(order=order, nq=nq, ng=2 if order == 1 else 3, flux=flux, limiter=limiter, rk=rk, precision=precision,
              cfl=0.15)
    for nx, ny in ((160, 60), (190, 99)) if precision == "fp64" else ((200, 96), (270, 139)):
        mesh = ordered(meshgen.channel(nx, ny))  # 150, 294; 300 and 587 tiles
        both(mesh, start(mesh, 3 if order == 1 else 6, (1.4, 4.2, 0.0, 8.8), "jump"), (1.4, 4.2, 0.0, 8.8), 4, **kw)


def test_a_small_solve_beside_a_large_one_leaves_it_the_device():
    """While a resident launch waits for its neighbours' tiles it keeps its
    places: looping beside it, a solve of 33,800 triangles made one of 500,000
    take 3.7 times as long as its stage launches do (then 1.2 times as long as
    alone).  Its bits stay."""
    import threading

    kw = dict(order=2, nq=6, ng=3, flux="hllc", cfl=0.1, farfield=FAR)
    mesh = meshgen.periodic_structured(130, 130, jitter=0.15, seed=3)
    small = CUDARkdgSolver(mesh, precision="fp64", **kw)
    large = CUDARkdgSolver(meshgen.periodic_structured(500, 500, jitter=0.15, seed=3), precision="fp32", **kw)
    large.initRKDG()
    U = start(mesh, 6, FAR, "vortex")
    small.setFreedom(U, basis="native")
    small.advance(50)
    ref = small.copyFreedomToHost(basis="native")
    large.advance(64)
    alone = min(in_threads([large], 64, 10) for _ in range(2))
    stop, same = threading.Event(), []

    def loop():
        while not stop.is_set():
            small.setFreedom(U, basis="native")
            small.advance(50)
            same.append(np.array_equal(small.copyFreedomToHost(basis="native"), ref))

    t = threading.Thread(target=loop)
    t.start()
    beside = min(in_threads([large], 64, 10) for _ in range(2))
    stop.set()
    t.join()
    small.close()
    large.close()
    assert all(same) and len(same) > 1
    assert beside < 2.2 * alone, (beside, alone)
