"""Failure paths on the GPU, made on the host: no GPU fault, trap or hang.

* A bounded device wait that gives up: the tile product's waits for a tile
  copy get a poll limit of 0 (fem_batch_set_wait_limit), so every wait gives
  up at once while the copy itself completes; the blocks drain their copies
  and fem_batch_synchronize reports FEM_E_TIMEOUT once. The batch then steps
  normally again, and as a fresh batch does.
* NaN injected through the state setters (a NaN initial velocity): the CG
  residual turns NaN and the solid, the batch and the server report
  FEM_E_NAN (ILSS_CG.h:42-46 -- the reference has no such check; its loop
  test is false for NaN and it returns silently).
"""
import dataclasses

import numpy as np
import pytest

from risdsdgcfem_thesis_gb300 import scenes

pytestmark = pytest.mark.gpu


def _meshes():
    rng = np.random.default_rng(11)
    return [scenes.random_block(rng, idx=i, dims=d) for i, d in enumerate([(6, 5, 4), (9, 4, 5), (5, 5, 5)])]


def test_tile_copy_wait_gives_up_and_reports_timeout(fem_lib):
    sc = _meshes()
    b = fem_lib.Batch(sc, fem_lib.FEM_PRECISION_MIXED, reorder=False)
    fresh = fem_lib.Batch(sc, fem_lib.FEM_PRECISION_MIXED, reorder=False)
    x0 = [b.state(i) for i in range(len(sc))]
    b.set_wait_limit(0)
    with pytest.raises(fem_lib.FemError) as e:
        b.step(1)
    assert e.value.code == fem_lib.FEM_E_TIMEOUT and "gave up" in str(e.value)
    # reported once (the word is cleared); the aborted step's own statistics
    # are left as they were (its CG loop stopped half way)
    assert fem_lib.load().fem_batch_synchronize(b.h) != fem_lib.FEM_E_TIMEOUT
    # back to the default limit, from the initial states: the same step as a
    # batch that never timed out
    b.set_wait_limit(None)
    for i, (x, v) in enumerate(x0):
        b.set_state(i, x, v)
    b.step(2)
    fresh.step(2)
    for i in range(len(sc)):
        xa, va = b.state(i)
        xb, vb = fresh.state(i)
        assert np.isfinite(xa).all() and np.isfinite(va).all()
        assert np.array_equal(xa, xb) and np.array_equal(va, vb), i
        assert b.stats(i)["cg_iterations"] == fresh.stats(i)["cg_iterations"]


def _nan_velocity(sc):
    """NaN on every node (a single node could sit on the fixed face, whose
    rows the constraint projection zeroes)."""
    return np.full_like(sc.rest, np.nan)


def test_nan_velocity_is_reported_by_the_solid(fem_lib):
    sc = scenes.cantilever_160()
    s = fem_lib.Solid(sc)
    s.set_state(v=_nan_velocity(sc))
    with pytest.raises(fem_lib.FemError) as e:
        s.step(1)
    assert e.value.code == fem_lib.FEM_E_NAN


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nan_velocity_is_reported_by_the_batch(fem_lib, precision):
    prec = fem_lib.FEM_PRECISION_FP64 if precision == "fp64" else fem_lib.FEM_PRECISION_MIXED
    sc = _meshes()
    b = fem_lib.Batch(sc, prec, reorder=False)
    b.set_state(1, v=_nan_velocity(sc[1]))
    with pytest.raises(fem_lib.FemError) as e:
        b.step(1)
    assert e.value.code == fem_lib.FEM_E_NAN and "mesh 1" in str(e.value)
    # the other meshes stepped as they do alone
    alone = fem_lib.Batch([sc[0]], prec, reorder=False)
    alone.step(1)
    assert np.array_equal(b.state(0)[0], alone.state(0)[0])


def test_nan_velocity_is_reported_by_the_server(fem_lib):
    sc = _meshes()
    srv = fem_lib.Server(fem_lib.FEM_PRECISION_MIXED)
    ids = [srv.add(s) for s in sc]
    assert srv.admit() == len(sc)
    srv.set_state(ids[2], v=_nan_velocity(sc[2]))
    for i in ids:
        srv.submit(i, tag=100 + i)
    done = {c["scene"]: c for c in srv.drain()}
    assert done[ids[2]]["status"] == fem_lib.FEM_E_NAN
    assert done[ids[0]]["status"] == fem_lib.FEM_OK and done[ids[1]]["status"] == fem_lib.FEM_OK


def _same_after_recovery(fem_lib, b, fresh, x0, step):
    b.set_wait_limit(None)
    for i, (x, v) in enumerate(x0):
        b.set_state(i, x, v)
    step(b)
    step(fresh)
    for i in range(len(x0)):
        for p, q in zip(b.state(i), fresh.state(i)):
            assert np.isfinite(p).all() and np.array_equal(p, q), i


@pytest.mark.parametrize("integrator", [0, 1])
@pytest.mark.parametrize("solver", [0, 1])
def test_host_driven_loops_end_when_a_wait_gives_up(fem_lib, integrator, solver):
    """Without a step graph the host drives the solver's and the Newton loop:
    both end when the device reports that a wait gave up."""
    sc = _meshes()
    for s in sc:
        s.integrator, s.ls_solver = integrator, solver
    b, fresh = (fem_lib.Batch(sc, fem_lib.FEM_PRECISION_MIXED, use_graph=False) for _ in range(2))
    x0 = [b.state(i) for i in range(len(sc))]
    b.set_wait_limit(0)
    with pytest.raises(fem_lib.FemError) as e:
        b.step(2)
    assert e.value.code == fem_lib.FEM_E_TIMEOUT
    assert fem_lib.load().fem_batch_synchronize(b.h) != fem_lib.FEM_E_TIMEOUT
    _same_after_recovery(fem_lib, b, fresh, x0, lambda s: s.step(2))


def test_lock_step_reports_a_wait_that_gives_up(fem_lib):
    sc = _meshes()
    b, fresh = (fem_lib.Batch(sc, fem_lib.FEM_PRECISION_MIXED) for _ in range(2))
    x0 = [b.state(i) for i in range(len(sc))]
    b.set_wait_limit(0)
    b.nr_phase("init", 1 / 60)
    b.nr_phase("prestep", 1 / 60)
    with pytest.raises(fem_lib.FemError) as e:
        b.nr_phase("midstep", 1 / 60)
    assert e.value.code == fem_lib.FEM_E_TIMEOUT
    _same_after_recovery(fem_lib, b, fresh, x0, lambda s: s.multi_step(1 / 60))


@pytest.mark.parametrize("dims", [(10, 10, 6), (17, 16, 15)], ids=["cluster", "clusters"])
@pytest.mark.parametrize("solver", [0, 1])
@pytest.mark.parametrize("integrator", [0, 1])
def test_resident_solve_gives_up_and_reports_timeout(fem_lib, dims, solver, integrator):
    """A solve whose waits give up reports it once, however many steps the
    call makes and whatever the later solves do, and no step is made from it;
    then the solid steps as a fresh one."""
    rest, tets, _ = scenes.grid_mesh(*dims, 0.1, 0.01, 5)
    sc = scenes.Scene(name="block", rest=rest, tets=tets, ls_solver=solver, integrator=integrator)
    sc.init_vel = 0.1 * np.random.default_rng(5).standard_normal(rest.shape)
    s, fresh = fem_lib.Solid(sc), fem_lib.Solid(sc)
    x0, v0 = s.state()
    s.step(1)
    s.set_state(x0, v0)
    s.set_wait_limit(0)
    with pytest.raises(fem_lib.FemError) as e:
        s.step(3)
    assert e.value.code == fem_lib.FEM_E_TIMEOUT
    assert all(np.array_equal(a, b) for a, b in zip(s.state(), (x0, v0)))
    if integrator == 0:  # unread while the later solves are whole
        assert fem_lib.load().fem_solid_step_async(s.h, 1) == fem_lib.FEM_OK
        s.set_wait_limit(None)
        with pytest.raises(fem_lib.FemError) as e:
            s.step(2)
        assert e.value.code == fem_lib.FEM_E_TIMEOUT
        assert all(np.array_equal(a, b) for a, b in zip(s.state(), (x0, v0)))
    s.set_wait_limit(None)
    s.step(2)
    fresh.step(2)
    assert s.stats()["cg_iterations"] == fresh.stats()["cg_iterations"]
    for a, b in zip(s.state(), fresh.state()):
        assert np.isfinite(a).all() and np.array_equal(a, b)


def test_lock_step_solve_gives_up_and_reports_timeout(fem_lib):
    rest, tets, _ = scenes.grid_mesh(10, 10, 6, 0.1, 0.01, 5)
    sc = scenes.Scene(name="block", rest=rest, tets=tets)
    sc.init_vel = 0.1 * np.random.default_rng(5).standard_normal(rest.shape)
    s, fresh = fem_lib.Solid(sc), fem_lib.Solid(sc)
    s.set_wait_limit(0)
    s.nr_phase("init", 1 / 60)
    s.nr_phase("prestep", 1 / 60)
    with pytest.raises(fem_lib.FemError) as e:
        s.nr_phase("midstep", 1 / 60)
    assert e.value.code == fem_lib.FEM_E_TIMEOUT
    s.set_wait_limit(None)
    for a in (s, fresh):
        fem_lib.multi_step([a], 1 / 60)
    for a, b in zip(s.state(), fresh.state()):
        assert np.array_equal(a, b)


def test_step_graph_after_a_newton_step_that_failed(fem_lib):
    """A Newton step that ends at a NaN right-hand side leaves work on the
    solid's second stream; a step graph captured next does not wait for it."""
    sc = scenes.cantilever_160()
    fresh = fem_lib.Solid(sc)
    sc = dataclasses.replace(sc, integrator=1)
    s = fem_lib.Solid(sc)
    x0, v0 = s.state()
    s.set_state(v=_nan_velocity(sc))
    with pytest.raises(fem_lib.FemError) as e:
        s.step(1)
    assert e.value.code == fem_lib.FEM_E_NAN
    s.set_state(x0, v0)
    p = s.get_params()
    p.integrator = 0
    s.set_params(p)
    s.step(2)
    fresh.step(2)
    for a, b in zip(s.state(), fresh.state()):
        assert np.isfinite(a).all() and np.array_equal(a, b)
