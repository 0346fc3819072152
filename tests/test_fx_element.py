"""The fixed-point element product of the FP64 path (risdsdgcfem_thesis_gb300/
csrc/fx.cuh): on the CPU against 128-bit products, next to the FP64 strain
form it takes the place of; on the GPU against the oracle at its edges.
"""
import ctypes as C
import os
import shutil
import subprocess
import threading

import numpy as np
import pytest

from risdsdgcfem_thesis_gb300 import scenes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SHIM = r"""
#include <float.h>
#include <math.h>
#include <stdint.h>
#define __device__
#define __forceinline__ inline
#include "fx.cuh"
#include "elem_math.cuh"
#if LDBL_MANT_DIG >= 113
typedef long double Q;
#else
typedef __float128 Q;
#endif
using namespace femgb;
extern "C" {
// One element's product in FP64 and in fixed point against 128 bits: squared
// relative errors (over the 12 outputs); returns 1 when the element takes
// FP64, 2 when the vector does.
int one(const double* R, const double* Di, double kl, double km, double grade, const double* d, double* e64, double* efx)
{
    FxL K[kFxK], D[9];
    int64_t out[12];
    int32_t x;
    if (!fx_grade_ok((float)grade, kl, km)) return 1;
    const int32_t scale = fx_bake(R, Di, kl, km, [&](int k, int64_t v) { K[k] = fx_split(v); });
    if (scale == kFxFp64) return 1;
    if (!fx_differences(d, D, x)) return 2;
    x += scale + fx_product([&](int k) { return K[k]; }, D, out);
    if (!fx_stamp(out, x)) return 2;
    Q Rq[9], Dq[9], dq[12], oq[12], n = 0, a = 0, b = 0;
    for (int i = 0; i < 9; i++) Rq[i] = R[i], Dq[i] = Di[i];
    for (int i = 0; i < 12; i++) dq[i] = d[i];
    elem_RKRt<Q, Q>(Rq, Dq, (Q)kl + 2 * (Q)km, (Q)kl, (Q)km, dq, oq);
    double o[12];
    elem_RKRt<double, double>(R, Di, kl + 2 * km, kl, km, d, o);
    for (int i = 0; i < 12; i++) {
        const int c = i - i % 3;
        FxSum s{{0, 0, 0}, 0};
        fx_add(s, out[c], out[c + 1], out[c + 2], 5);  // as a node of 32 corners adds it
        const Q f = fx_sum_value(s.acc[i - c], s.E, 5);
        n += oq[i] * oq[i];
        a += ((Q)o[i] - oq[i]) * ((Q)o[i] - oq[i]);
        b += (f - oq[i]) * (f - oq[i]);
    }
    *e64 = n > 0 ? (double)(a / n) : 0.0;
    *efx = n > 0 ? (double)(b / n) : (double)b;
    return 0;
}
double through_double(double v) { return fx_to_double(fx_align<62>(v, fx_exp(v)), fx_exp(v) - 1022 - 62); }
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    d = tmp_path_factory.mktemp("fx")
    (d / "shim.cpp").write_text(SHIM)
    so = d / "shim.so"
    subprocess.run([gxx, "-O2", "-std=gnu++17", "-Wno-unknown-pragmas", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                    os.path.join(ROOT, "risdsdgcfem_thesis_gb300", "csrc"), str(d / "shim.cpp"), "-o", str(so)],
                   check=True)
    lib = C.CDLL(str(so))
    p = C.POINTER(C.c_double)
    lib.one.argtypes = [p, p, C.c_double, C.c_double, C.c_double, p, p, p]
    lib.through_double.argtypes = [C.c_double]
    lib.through_double.restype = C.c_double
    return lib


def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _elements(nu, rng):
    """Elements of a jittered block of the library's scenes, with rotations a
    little off orthonormal: (R, Dm^-1, V lambda, V mu, grade, rest)."""
    rest, tets, _ = scenes.grid_mesh(5, 4, 3, 0.01, 0.001, int(rng.integers(1 << 30)))
    p = rest[tets]
    Dm = (p[:, 1:] - p[:, :1]).transpose(0, 2, 1)
    Di = np.linalg.inv(Dm)
    vol = np.linalg.det(Dm) / 6.0
    lam, mu = 1e5 * nu / ((1 + nu) * (1 - 2 * nu)), 0.5e5 / (1 + nu)
    for e in range(len(tets)):
        Q, _ = np.linalg.qr(rng.standard_normal((3, 3)))
        yield (np.ascontiguousarray(Q * (1 + 1e-4 * rng.standard_normal((3, 3)))), np.ascontiguousarray(Di[e]),
               vol[e] * lam, vol[e] * mu, np.abs(Dm[e]).max() * np.abs(Di[e]).max(), p[e])


def _run(shim, el, d):
    R, Di, kl, km, grade, _ = el
    a, b = np.zeros(1), np.zeros(1)
    d = np.ascontiguousarray(d, dtype=np.float64)
    rc = shim.one(_ptr(R), _ptr(Di), kl, km, grade, _ptr(d), _ptr(a), _ptr(b))
    return rc, a[0], b[0]


@pytest.mark.parametrize("nu", [-0.2, 0.0, 0.3, 0.45])
@pytest.mark.parametrize("field", ["random", "affine", "drifting"])
def test_error_is_no_larger_than_fp64s(shim, nu, field):
    """Root mean square relative error over a block's elements, against 128
    bits: at most the FP64 strain form's."""
    rng = np.random.default_rng(7)
    s64 = sfx = 0.0
    n = 0
    for el in _elements(nu, rng):
        if field == "random":
            d = rng.standard_normal((4, 3)) * 10.0 ** rng.uniform(-6, 2)
        else:
            d = el[5] @ rng.standard_normal((3, 3)) + (0.01 if field == "affine" else 1.0) * rng.standard_normal(3)
        rc, a, b = _run(shim, el, d)
        assert rc == 0
        s64, sfx, n = s64 + a, sfx + b, n + 1
    assert n == 300 and sfx <= s64, (np.sqrt(sfx / n), np.sqrt(s64 / n))


@pytest.mark.parametrize("nu", [-2.0, -1.2, 0.50001, 0.51, 0.55, 0.6, 1.0])
def test_indefinite_materials_take_fp64(shim, nu):
    """Outside (-1, 0.5) the element matrix is not positive semidefinite, and
    its largest entry need not be on the diagonal that scales it."""
    rng = np.random.default_rng(7)
    assert all(_run(shim, el, rng.standard_normal((4, 3)))[0] == 1 for el in _elements(nu, rng))


def test_edges_of_the_number_format(shim):
    rng = np.random.default_rng(3)
    el = next(_elements(0.3, rng))
    base = rng.standard_normal((4, 3))
    assert _run(shim, el, np.zeros((4, 3))) == (0, 0.0, 0.0)
    assert _run(shim, el, np.ones((4, 3)))[0] == 0  # equal nodal vectors: no force
    assert _run(shim, el, np.ones((4, 3)))[2] == 0.0
    for scale in (1e-280, 1e280):  # the exponents are carried, not the magnitudes
        rc, a, b = _run(shim, el, base * scale)
        assert rc == 0 and b <= max(a, 1e-31)
    far = base.copy()
    far[0, 0] = 1e300  # one component far above the others
    assert _run(shim, el, far)[0] == 0
    for bad in (np.nan, np.inf):
        v = base.copy()
        v[2, 1] = bad
        assert _run(shim, el, v)[0] == 2
    long_row = (el[0] * 1.2, *el[1:])
    assert _run(shim, long_row, base)[0] == 1
    graded = (*el[:4], 3.5, el[5])
    assert _run(shim, graded, base)[0] == 1
    for v in (1.0, -1.0, 1.5, np.nextafter(1.0, 2), -3.25e-200, 7e200, 0.0, np.nextafter(2.0, 0)):
        assert shim.through_double(v) == v


def _fan(k):
    """k wedges around the edge (0, 1): two nodes with k corners each, thin
    elements that the fixed-point form leaves to FP64."""
    t = 2 * np.pi * np.arange(k) / k
    rest = np.concatenate([[[0, 0, 0], [0, 0, 1.0]], np.stack([np.cos(t), np.sin(t), 0.5 + 0 * t], 1)])
    tets = np.array([[0, 1, 2 + i, 2 + (i + 1) % k] for i in range(k)], np.uint32)
    p = rest[tets]
    bad = np.linalg.det(p[:, 1:] - p[:, :1]) < 0
    tets[bad] = tets[bad][:, [0, 2, 1, 3]]
    return scenes.Scene(name="fan", rest=rest, tets=tets)


def _block(dims, stretch=(1, 1, 1), poisson=0.3):
    rest, tets, _ = scenes.grid_mesh(*dims, 0.1, 0.01, 5)
    return scenes.Scene(name="block", rest=rest * np.asarray(stretch), tets=tets, poisson=poisson)


@pytest.mark.gpu
@pytest.mark.parametrize("scene", [_block((1, 1, 1)), _block((3, 2, 4)), _block((7, 9, 8)), _block((17, 16, 15)),
                                   _block((4, 4, 4), (1, 1, 0.1)), _block((4, 3, 4), (1, 1, 0.4)),
                                   _block((4, 4, 4), poisson=0.499), _fan(5), _fan(300)],
                         ids=["5", "120", "2520", "20400", "graded", "part-graded", "stiff", "fan5", "fan300"])
def test_products_match_the_oracle(fem_lib, oracle, scene):
    """df_x and A d on an evaluated state. The oracle's own FP64 products and
    sums (300 corners at a node of the fan) set the bar: 2e-13 of the largest
    entry."""
    rng = np.random.default_rng(1)
    g, o = fem_lib.Solid(scene), oracle.Solid(scene, "port")
    x = scene.rest + 0.02 * rng.standard_normal(scene.rest.shape) * np.ptp(scene.rest, axis=0).min() / 3
    g.begin_eval(x)
    o.begin_eval(x)
    for scale in (1.0, 1e-150, 1e150):
        d = scale * rng.standard_normal(scene.rest.shape)
        for a, b in ((g.df_x(d), o.df_x(d)), (g.apply_A(1.0, 1 / 3600, d), o.apply_A(1.0, 1 / 3600, d))):
            assert np.abs(a - b).max() <= 2e-13 * np.abs(b).max()
    d[scene.tets[0, 1], 2] = np.nan
    assert np.array_equal(np.isnan(g.df_x(d)).any(1), np.isnan(o.df_x(d)).any(1))


@pytest.mark.gpu
@pytest.mark.parametrize("nu", [-1.2, 0.55, 1.0])
def test_indefinite_materials_match_the_oracle(fem_lib, oracle, nu):
    """Elements whose matrix is not semidefinite run in FP64 in every form of
    the product: the hooks', the resident rows' and the FP64 batch's. Bars as
    in test_products_match_the_oracle (products) and
    test_batch_products_match_the_oracle (two CG iterations)."""
    rng = np.random.default_rng(8)
    scene = _block((4, 3, 4), poisson=nu)
    scene.init_vel = 0.1 * rng.standard_normal(scene.rest.shape)
    scene.max_iter = 2
    g, o, b = fem_lib.Solid(scene), oracle.Solid(scene, "port"), fem_lib.Batch([scene], precision=fem_lib.FEM_PRECISION_FP64)
    x = scene.rest + 0.005 * rng.standard_normal(scene.rest.shape)
    g.begin_eval(x)
    o.begin_eval(x)
    d = rng.standard_normal(scene.rest.shape)
    for p, q in ((g.df_x(d), o.df_x(d)), (g.apply_A(1.0, 1 / 3600, d), o.apply_A(1.0, 1 / 3600, d))):
        assert np.abs(p - q).max() <= 2e-13 * np.abs(q).max()
    g, o = fem_lib.Solid(scene), oracle.Solid(scene, "port")
    g.step(1)
    b.step(1)
    assert o.step()["iters"] == g.stats()["cg_iterations"] == b.stats(0)["cg_iterations"] == 2
    v = o.state()[1]
    for w in (g.state()[1], b.state(0)[1]):
        assert np.linalg.norm(w - v) <= 1e-12 * np.linalg.norm(v)


@pytest.mark.gpu
def test_batch_products_match_the_oracle(fem_lib, oracle):
    """FP64 batch of meshes whose tiles are in fixed point, partly or not at
    all, from one cell to several tiles: one step of two CG iterations, five
    products that each agree to 2e-13 as above, so 1e-12 for the velocity."""
    scs = [_block((1, 1, 1)), _block((3, 2, 4)), _block((7, 9, 8)), _block((4, 4, 4), (1, 1, 0.1)),
           _block((4, 3, 4), (1, 1, 0.4)), _block((4, 4, 4), poisson=0.499), _fan(5), _fan(100)]
    rng = np.random.default_rng(4)
    for sc in scs:
        sc.init_vel = 0.1 * rng.standard_normal(sc.rest.shape)
        sc.max_iter = 2
    b = fem_lib.Batch(scs, precision=fem_lib.FEM_PRECISION_FP64)
    b.step(1)
    for i, sc in enumerate(scs):
        o = oracle.Solid(sc, "port")
        assert o.step()["iters"] == b.stats(i)["cg_iterations"] == 2
        v = o.state()[1]
        assert np.linalg.norm(b.state(i)[1] - v) <= 1e-12 * np.linalg.norm(v)


@pytest.mark.gpu
@pytest.mark.parametrize("scene", [_block((1, 1, 1)), _block((2, 2, 1)), _block((5, 5, 5)), _block((11, 12, 11)),
                                   _block((4, 4, 4), (1, 1, 0.1)), _block((4, 3, 4), (1, 1, 0.4)),
                                   _block((4, 4, 4), poisson=0.499), _fan(5), _fan(100)],
                         ids=["5", "20", "625", "7260", "graded", "part-graded", "stiff", "fan5", "fan100"])
@pytest.mark.parametrize("solver", ["cg", "minres"])
def test_solve_on_resident_rows_matches_the_oracle(fem_lib, oracle, scene, solver):
    """The solid's solve from one block of nodes to all clusters, with fixed
    nodes: as the batch above, 1e-12 after two CG or MINRES iterations."""
    rng = np.random.default_rng(4)
    scene.ls_solver = fem_lib.FEM_LS_MINRES if solver == "minres" else fem_lib.FEM_LS_CG
    scene.init_vel = 0.1 * rng.standard_normal(scene.rest.shape)
    scene.knc_nodes = np.array([0, len(scene.rest) - 1], np.uint32)
    scene.knc_targets = scene.rest[scene.knc_nodes].copy()
    scene.max_iter = 2
    g, o = fem_lib.Solid(scene), oracle.Solid(scene, "port")
    g.step(1)
    assert o.step()["iters"] == g.stats()["cg_iterations"] == 2
    v = o.state()[1]
    assert np.linalg.norm(g.state()[1] - v) <= 1e-12 * np.linalg.norm(v)


@pytest.mark.gpu
def test_resident_solves_side_by_side(fem_lib):
    """Solids of one and of several clusters stepped from threads at once give
    the bits they give alone."""
    shapes = [((16, 16, 12), 0), ((14, 10, 10), 1), ((10, 10, 6), 0), ((8, 2, 2), 0)]

    def run(k, out):
        dims, solver = shapes[k]
        sc = _block(dims)
        sc.ls_solver = solver
        sc.init_vel = 0.1 * np.random.default_rng(k).standard_normal(sc.rest.shape)
        s = fem_lib.Solid(sc)
        for _ in range(20):
            s.step(1)
        out[k] = s.state()

    alone, together = [None] * 4, [None] * 4
    for k in range(4):
        run(k, alone)
    threads = [threading.Thread(target=run, args=(k, together)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(alone, together):
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


@pytest.mark.gpu
def test_solve_after_many_solves_without_iterations(fem_lib):
    """The words between the clusters carry 16 bits of the exchange's number.
    65,534 solves that end at their residual bring the number round to that
    of the last d.q: the next solve takes none of its sums."""
    sc = _block((17, 16, 15))
    v0 = 0.1 * np.random.default_rng(6).standard_normal(sc.rest.shape)
    fresh, s = (fem_lib.Solid(sc, compute_energy=False) for _ in range(2))
    s.set_state(v=v0)
    s.step(1)
    p = s.get_params()
    full, p.ls_max_iter = p.ls_max_iter, 0
    s.set_params(p)
    s.set_state(sc.rest, np.zeros_like(v0))
    s.step(65534)
    assert s.stats()["cg_iterations"] == 0
    p.ls_max_iter = full
    s.set_params(p)
    s.set_state(sc.rest, v0)
    fresh.set_state(v=v0)
    s.step(1)
    fresh.step(1)
    assert s.stats()["cg_iterations"] == fresh.stats()["cg_iterations"] > 0
    for a, b in zip(s.state(), fresh.state()):
        assert np.array_equal(a, b)
