"""The FP64 solid's solvers as loops of kernels, on the element products and
on the assembled stiffness: solids whose rows do not fit the shared memory of
the GPU's SMs (test_rows_plan.py), which solve there otherwise."""
import ctypes
import dataclasses

import numpy as np
import pytest

from risdsdgcfem_thesis_gb300 import scenes
from test_fx_element import _block, _fan

pytestmark = pytest.mark.gpu

SHAPES = {
    "block": (lambda: _block((30, 30, 30)), 1e-12),
    "flat": (lambda: _block((100, 30, 6)), 1e-12),
    "graded": (lambda: _block((30, 30, 30), (1, 1, 0.1)), 1e-12),
    "part-graded": (lambda: _block((30, 30, 30), (1, 1, 0.4)), 1e-12),
    "stiff": (lambda: _block((30, 30, 30), poisson=0.499), 1e-12),
    # ten times thinner wedges and ten times longer sums than the fan of 100 in test_fx_element.py
    "fan1000": (lambda: _fan(1000), 1e-10),
}


@pytest.fixture(scope="module")
def reference(oracle):
    """The oracle's velocities after one step of two iterations, per shape,
    solver and integrator."""
    made = {}

    def get(shape, solver, integrator):
        key = (shape, solver, integrator)
        if key not in made:
            sc = SHAPES[shape][0]()
            rng = np.random.default_rng(4)
            sc = dataclasses.replace(sc, ls_solver=solver, integrator=integrator, max_iter=2, nr_max_iter=1,
                                     init_vel=0.1 * rng.standard_normal(sc.rest.shape),
                                     knc_nodes=np.array([0, len(sc.rest) - 1], np.uint32))
            sc.knc_targets = sc.rest[sc.knc_nodes].copy()
            o = oracle.Solid(sc, "port")
            o.step()
            made[key] = sc, o.state()[1]
        return made[key]

    return get


@pytest.mark.parametrize("integrator", [0, 1], ids=["graph", "host"])
@pytest.mark.parametrize("assembled", [False, True], ids=["elements", "assembled"])
@pytest.mark.parametrize("solver", [0, 1], ids=["cg", "minres"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_solver_loop_matches_the_oracle(fem_lib, reference, shape, solver, assembled, integrator):
    """As test_solve_on_resident_rows_matches_the_oracle: two iterations, from
    a step graph (QIE) and driven from the host (FIE, one Newton iteration),
    where the kernels that ran are read back."""
    sc, v = reference(shape, solver, integrator)
    s = fem_lib.Solid(sc, compute_energy=False)
    s.set_assembled(assembled)
    if integrator:
        fem_lib.profile_enable(True)  # from zero
    try:
        s.step(1)
    finally:
        fem_lib.profile_enable(False)
    if integrator:
        rows, elem, assembly, node_q = [fem_lib.profile_read(n)[1] for n in
                                        ("cg_rows_fp64", "elem_spmv_fp64", "bsr_assemble_fp64", "node_q_fp64")]
        assert rows == 0 and (elem == 0) == assembled and (assembly > 0) == assembled and (node_q > 0) == (solver == 0)
    assert s.stats()["cg_iterations"] == 2
    assert np.linalg.norm(s.state()[1] - v) <= SHAPES[shape][1] * np.linalg.norm(v)


@pytest.mark.parametrize("solver", [0, 1], ids=["cg", "minres"])
def test_assembled_stiffness_switched_between_steps(fem_lib, solver):
    """Steps on the element products and on the assembled stiffness in turn,
    which each agree with the oracle's to 1e-12, stay within ten times that
    of steps on the element products alone over four steps."""
    sc = _block((30, 30, 30))
    sc = dataclasses.replace(sc, ls_solver=solver, max_iter=2,
                             init_vel=0.1 * np.random.default_rng(4).standard_normal(sc.rest.shape))
    a, b = (fem_lib.Solid(sc, compute_energy=False) for _ in range(2))
    for on in (False, True, False, True):
        b.set_assembled(on)
        a.step(1)
        b.step(1)
    for p, q in zip(a.state(), b.state()):
        assert np.linalg.norm(p - q) <= 1e-11 * np.linalg.norm(p)


@pytest.mark.parametrize("solver", [0, 1], ids=["cg", "minres"])
@pytest.mark.parametrize("form", ["cluster", "clusters", "elements", "assembled", "batch"])
def test_sums_that_overflow(fem_lib, oracle, form, solver):
    """Velocities near the square root of the largest double: where |r|^2 or
    d.q overflows, a solve ends or goes on as the reference's does (an infinite
    d.q makes alpha zero, not NaN). Bar as above, where the oracle is finite."""
    sc = _block({"cluster": (3, 2, 4), "clusters": (16, 16, 12), "batch": (9, 8, 7)}.get(form, (30, 30, 30)))
    v0 = np.random.default_rng(4).standard_normal(sc.rest.shape)
    for scale in 10.0 ** np.arange(148, 160):
        sc = dataclasses.replace(sc, ls_solver=solver, max_iter=3, init_vel=scale * v0)
        o = oracle.Solid(sc, "port")
        iters = o.step()["iters"]
        x, v = o.state()
        g = fem_lib.Batch([sc], fem_lib.FEM_PRECISION_FP64, compute_energy=False) if form == "batch" else \
            fem_lib.Solid(sc, compute_energy=False)
        if form in ("elements", "assembled"):
            g.set_assembled(form == "assembled")
        try:
            g.step(1)
        except fem_lib.FemError as e:
            assert e.code == fem_lib.FEM_E_NAN
        if form == "batch":
            (xg, vg), k = g.state(0), g.stats(0)["cg_iterations"]
        else:
            st = fem_lib.FemStepStats()
            fem_lib.load().fem_solid_synchronize(g.h, ctypes.byref(st))
            (xg, vg), k = g.state(), st.cg_iterations
        assert k == iters, (scale, k, iters)
        ok = np.isfinite(v)
        assert np.array_equal(np.isfinite(vg), ok) and np.array_equal(np.isfinite(xg), np.isfinite(x)), scale
        if ok.all():
            assert np.abs((vg - v) / scale).max() <= 1e-12 * np.abs(v / scale).max(), scale
        g.close()


def _shuffled(dims):
    sc = _block(dims)
    p = np.random.default_rng(2).permutation(len(sc.rest)).astype(np.uint32)
    rest = np.empty_like(sc.rest)
    rest[p] = sc.rest
    return dataclasses.replace(sc, rest=rest, tets=p[sc.tets])


@pytest.mark.parametrize("solver", [0, 1], ids=["cg", "minres"])
@pytest.mark.parametrize("shape, bar", [(_shuffled((3, 2, 4)), 1e-12), (_shuffled((10, 10, 6)), 1e-12),
                                        (_shuffled((17, 16, 15)), 1e-12), (_fan(300), 1e-11), (_fan(342), 1e-11)],
                         ids=["120", "3000", "20400", "fan300", "fan342"])
def test_resident_rows_of_any_numbering(fem_lib, oracle, shape, bar, solver):
    """Meshes whose rows and rims are spread over the numbering, and hubs at the
    line up to which rows are made on the device (341 corners): as the solves in
    numbering order, 1e-12 after two iterations (fans of thinner wedges: 1e-11)."""
    rng = np.random.default_rng(4)
    sc = dataclasses.replace(shape, ls_solver=solver, max_iter=2, init_vel=0.1 * rng.standard_normal(shape.rest.shape))
    g, o = fem_lib.Solid(sc), oracle.Solid(sc, "port")
    g.step(1)
    assert o.step()["iters"] == g.stats()["cg_iterations"] == 2
    v = o.state()[1]
    assert np.linalg.norm(g.state()[1] - v) <= bar * np.linalg.norm(v)
