"""The library's performance cases.

A case is one fixed step (or one round of element hooks) of the work a caller gives this
library, through its public entry points: the FP64 solid (the drop-in for the reference's
step), batches of meshes in FP64 and in mixed precision, and the step-request server. Every pass
starts from the same host state in pinned memory, so a pass is what a host program that owns the
positions does per frame: states up, one step, states down.

Meshes, materials and solver settings are those of the library's own scenes (`scenes.py`): blocks
of cubes of five jittered tets. Solids take the cantilever's material and iteration cap (h = 0.1 m,
E = 1e5, nu = 0.3, at most 200 iterations), solved to 1e-10 so that the rounding of a sum does not
show in the state (at the cantilever's 1e-8 it moves 160 tets by up to 6e-9), or the large block's
per-element material with the library's default solver settings (relative 1e-3, at most 20
iterations: an interactive caller); batches and the server take the batched workload's meshes
(h = 0.01 m, per-mesh E and nu, a random fixed face), in mixed precision with its tolerance (1e-6,
at most 500 iterations), in FP64 with the default settings. States are mid-motion: bent, noisy
and moving.
"""
import ctypes as C
import math

import numpy as np
import torch

from risdsdgcfem_thesis_gb300 import capi, scenes

# ---------------------------------------------------------------- the cases


def listed():
    return [
        # The smallest solid: the 160-tet cantilever, one interactive object. Latency counts.
        {"name": "solid_cantilever_160", "kind": "solid", "a": 8, "b": 2, "c": 2, "material": "uniform"},
        # A small object with odd extents, 3,060 tets.
        {"name": "solid_3k", "kind": "solid", "a": 17, "b": 9, "c": 4, "material": "uniform"},
        # A medium object, 20,480 tets.
        {"name": "solid_20k", "kind": "solid", "a": 16, "b": 16, "c": 16, "material": "uniform"},
        # The large block, 1,080,000 tets, per-element material, at interactive solver settings.
        {"name": "solid_block60", "kind": "solid", "a": 60, "b": 60, "c": 60, "material": "per_element"},
        # The assembled-stiffness option on 320,000 tets, solved to 1e-10.
        {"name": "solid_assembled_40", "kind": "solid_assembled", "a": 40, "b": 40, "c": 40, "material": "uniform"},
        # MINRES, the solver the reference's own scenes select, on 7,215 tets.
        {"name": "solid_minres_7k", "kind": "solid_minres", "a": 13, "b": 37, "c": 3, "material": "uniform"},
        # The Newton integrator (three Newton iterations, each its own solve), 2,700 tets.
        {"name": "solid_newton_2k7", "kind": "solid_newton", "a": 9, "b": 10, "c": 6, "material": "uniform"},
        # The element set's hooks for a caller with its own solver: evaluation, force, one
        # differential and one operator product on 40,000 tets.
        {"name": "hooks_40k", "kind": "hooks", "a": 20, "b": 20, "c": 20, "material": "uniform"},
        # 64 uneven meshes stepped together in FP64.
        {"name": "batch_fp64_64", "kind": "batch_fp64", "count": 64, "lo": 4, "hi": 20},
        # A few small scenes in mixed precision, a quarter each with CG, MINRES, the C_LCM
        # material and the DAPD rotation.
        {"name": "batch_mixed_small", "kind": "batch_methods", "count": 24, "lo": 3, "hi": 9},
        # The batched workload (uneven meshes, mixed precision) at 192 meshes, about 4.7 M tets.
        {"name": "batch_mixed_192", "kind": "batch_mixed", "count": 192, "lo": 4, "hi": 30},
        # 96 resident scenes of 200 to 40,000 tets, one step requested of each.
        {"name": "served_96", "kind": "served", "count": 96, "lo": 200, "hi": 40000},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _dims(rng, lo, hi):
    """Extents of a block of about log-uniform [lo, hi] tets, of an aspect of up to 3."""
    cubes = _log(rng, lo, hi) / 5.0
    r1, r2 = rng.uniform(0.6, 1.8), rng.uniform(0.6, 1.8)
    a = max(1, round((cubes * r1 * r2) ** (1.0 / 3.0)))
    b = max(1, round(a / r1))
    return a, b, max(1, round(cubes / (a * b)))


def draw(rng):
    kind = rng.choice(["solid", "solid", "solid", "solid", "solid_assembled", "solid_minres", "solid_newton",
                       "hooks", "batch_fp64", "batch_methods", "batch_mixed", "served"])
    case = {"kind": kind}
    if kind.startswith("batch"):
        most = {"batch_fp64": 64, "batch_methods": 48, "batch_mixed": 160}[kind]
        case["count"] = max(1, round(_log(rng, 1, most)))
        case["lo"] = rng.randint(2, 6)
        case["hi"] = case["lo"] + rng.randint(1, {"batch_fp64": 14, "batch_methods": 6, "batch_mixed": 24}[kind])
    elif kind == "served":
        case["count"] = max(2, round(_log(rng, 2, 96)))
        case["lo"], case["hi"] = 200, round(_log(rng, 1000, 40000))
    else:
        hi = {"solid": 600000, "solid_assembled": 300000, "solid_minres": 30000, "solid_newton": 20000,
              "hooks": 300000}[kind]
        case["a"], case["b"], case["c"] = _dims(rng, 9000 if kind == "solid_assembled" else 100, hi)
        case["material"] = "uniform" if kind == "solid_assembled" else rng.choice(["uniform", "per_element"])
    return case


# ---------------------------------------------------------------- inputs


def _solid_scene(case, rng):
    per_element = case["material"] == "per_element"
    a, b, c = case["a"], case["b"], case["c"]
    h = 0.01 if per_element else 0.1
    rest, tets, ijk = scenes.grid_mesh(a, b, c, h, 0.1 * h, int(rng.integers(0, 2**31)))
    fixed = np.nonzero(ijk[:, 0] == 0)[0].astype(np.uint32)
    sc = scenes.Scene(name="block_%dx%dx%d" % (a, b, c), rest=rest, tets=tets, young=1e5, poisson=0.3,
                      gravity=(0.0, 0.0, -9.81), rel_eps=1e-10, abs_eps=0.0, max_iter=200, knc_nodes=fixed,
                      knc_targets=rest[fixed].copy(), grid=(a, b, c), h=h)
    if per_element:  # the large block's material, the library's default solver settings
        sc.young_per_elem = np.exp(rng.uniform(math.log(5e4), math.log(5e5), size=tets.shape[0]))
        sc.poisson_per_elem = rng.uniform(0.25, 0.45, size=tets.shape[0])
        sc.rel_eps, sc.abs_eps, sc.max_iter = 1e-3, 1e-6, 20
    if case["kind"] == "solid_minres":
        sc.ls_solver = capi.FEM_LS_MINRES
    if case["kind"] == "solid_newton":
        sc.integrator = capi.FEM_INTEGRATOR_FIE_DX
    return sc


def _scenes(case, seed):
    """The case's scenes: sizes from the case, geometry, materials and fixed faces from the seed."""
    rng = np.random.default_rng([int(seed), 17])
    kind = case["kind"]
    if "count" in case:
        sizes = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    if kind.startswith("batch"):
        dims = sizes.integers(case["lo"], case["hi"] + 1, size=(case["count"], 3))
        scs = [scenes.random_block(rng, idx=i, dims=tuple(int(n) for n in d)) for i, d in enumerate(dims)]
    elif kind == "served":
        targets = np.exp(sizes.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))
        scs = [scenes.sized_block(rng, float(t), idx=i) for i, t in enumerate(targets)]
    else:
        scs = [_solid_scene(case, rng)]
    for i, sc in enumerate(scs):
        if kind == "batch_fp64":
            sc.rel_eps, sc.abs_eps, sc.max_iter = 1e-3, 1e-6, 20
        if kind == "batch_methods":
            if i % 4 == 1:
                sc.ls_solver = capi.FEM_LS_MINRES
            elif i % 4 == 2:
                sc.material = capi.FEM_MATERIAL_C_LCM
            elif i % 4 == 3:
                sc.rotation = capi.FEM_ROTATION_DAPD
    return scs, rng


def _moving(sc, rng):
    """A mid-motion state: bent and twisted away from the fixed face, with noise."""
    fixed = sc.rest[sc.knc_nodes]
    axis = int(np.argmin(fixed.max(0) - fixed.min(0)))
    s = np.abs(sc.rest[:, axis] - fixed[:, axis].mean())
    s = (s / max(s.max(), 1e-30))[:, None]
    size = float((sc.rest.max(0) - sc.rest.min(0)).max())
    phase = rng.uniform(0.0, 2.0 * math.pi, size=3)
    wave = np.sin(2.0 * sc.rest[:, [1, 2, 0]] / size + phase)
    x = sc.rest + 0.06 * size * s * s * (rng.uniform(-1.0, 1.0, size=3) + 0.3 * wave)
    x += 0.005 * sc.h * rng.standard_normal(x.shape)
    v = s * (rng.uniform(-0.5, 0.5, size=3) + 0.3 * wave) + 0.005 * rng.standard_normal(x.shape)
    x[sc.knc_nodes] = sc.knc_targets
    v[sc.knc_nodes] = 0.0
    return x, v


def _states(scs, rng):
    xv = [_moving(sc, rng) for sc in scs]
    return np.concatenate([x for x, _ in xv]), np.concatenate([v for _, v in xv])


def _probe(scs, rng):
    """A direction for the hooks' products, as a caller's own solver iterates on."""
    return rng.standard_normal(scs[0].rest.shape)


def _host(a=None, like=None):
    t = torch.empty(like.shape if a is None else a.shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    if a is not None:
        t.copy_(torch.from_numpy(a))
    return t


_dp = C.POINTER(C.c_double)


def _at(t, node=0):
    return C.cast(t.data_ptr() + 24 * node, _dp)


def prepare(case, seed):
    scs, rng = _scenes(case, seed)
    x, v = _states(scs, rng)
    kind = case["kind"]
    s = {"kind": kind, "x": _host(x), "v": _host(v), "scenes": scs}
    if kind == "hooks":
        s["d"] = _probe(scs, rng)
        s["solid"] = capi.Solid(scs[0])
        return s
    s["x_out"], s["v_out"] = _host(like=x), _host(like=v)
    if kind.startswith("solid"):
        s["solid"] = capi.Solid(scs[0])
        if kind == "solid_assembled":
            s["solid"].set_assembled(True)
    elif kind.startswith("batch"):
        s["batch"] = capi.Batch(scs, precision=capi.FEM_PRECISION_FP64 if kind == "batch_fp64"
                                else capi.FEM_PRECISION_MIXED)
    else:
        s["server"] = capi.Server()
        s["ids"] = [s["server"].add(sc) for sc in scs]
        s["server"].admit()
        s["at"] = np.concatenate([[0], np.cumsum([sc.num_nodes for sc in scs])]).tolist()
    return s


def run(s):
    kind = s["kind"]
    if kind == "hooks":  # the force seam of a caller that keeps its own solver
        solid, sc = s["solid"], s["scenes"][0]
        solid.begin_eval(s["x"].numpy())
        return {"f": solid.f_e(), "df": solid.df_x(s["d"]), "q": solid.apply_A(1.0, sc.dt * sc.dt, s["d"])}
    x, v, x_out, v_out = s["x"], s["v"], s["x_out"], s["v_out"]
    if kind.startswith("solid"):
        solid = s["solid"]
        capi.check(solid.lib.fem_solid_step_host(solid.h, _at(x), _at(v), 1, _at(x_out), _at(v_out), None))
    elif kind.startswith("batch"):
        b = s["batch"]
        capi.check(b.lib.fem_batch_step_host(b.h, _at(x), _at(v), 1, _at(x_out), _at(v_out)))
    else:
        srv, at = s["server"], s["at"]
        for i, k in enumerate(s["ids"]):
            capi.check(srv.lib.fem_server_set_state(srv.h, k, _at(x, at[i]), _at(v, at[i])))
            srv.submit(k, k)
        srv.drain()
        for i, k in enumerate(s["ids"]):
            capi.check(srv.lib.fem_server_get_state(srv.h, k, _at(x_out, at[i]), _at(v_out, at[i])))
    return {"x": x_out, "v": v_out}


# ---------------------------------------------------------------- work


def _iterations(case):
    """Solver iterations one step needs, about."""
    kind = case["kind"]
    if kind == "hooks":
        return 2
    if kind in ("batch_mixed", "batch_methods", "served"):
        return 150
    if kind == "batch_fp64" or case.get("material") == "per_element":
        return 20
    return 200 if kind == "solid_newton" else 65


def work(case):
    kind = case["kind"]
    if "a" in case:
        cubes = case["a"] * case["b"] * case["c"]
        nodes = (case["a"] + 1) * (case["b"] + 1) * (case["c"] + 1)
    elif kind == "served":
        lo, hi = case["lo"], case["hi"]
        cubes = case["count"] * (hi - lo) / math.log(hi / lo) / 5.0
        nodes = 1.2 * cubes
    else:
        mean = lambda f: sum(f(k) for k in range(case["lo"], case["hi"] + 1)) / (case["hi"] + 1 - case["lo"])  # noqa: E731
        cubes = case["count"] * mean(lambda k: k) ** 3
        nodes = case["count"] * mean(lambda k: k + 1) ** 3
    tets = 5.0 * cubes
    # per tet: ids, shape gradients, material (FP32 in mixed precision); per node: rest
    # positions, x and v in, x and v out. Per tet: about 400 operations for the rotation and the
    # force, 250 for a product, and 33 vector operations per node and iteration.
    per_tet = 16 + 12 * (4 if kind in ("batch_mixed", "batch_methods", "served") else 8)
    return {"bytes": per_tet * tets + 120.0 * nodes,
            "flops": 400.0 * tets + _iterations(case) * (250.0 * tets + 33.0 * nodes)}


# ---------------------------------------------------------------- the same in plain torch, 64 bits


def _mm(a, b):
    """Products of 3x3 matrices."""
    return (a[:, :, 0, None] * b[:, None, 0] + a[:, :, 1, None] * b[:, None, 1]) + a[:, :, 2, None] * b[:, None, 2]


def _t(a):
    return a.transpose(1, 2)


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _orthogonal(v):
    """A vector orthogonal to v: its smallest component's axis left out."""
    a = v.abs()
    z = torch.zeros_like(v[:, 0])
    drop_x = torch.stack([z, v[:, 2], -v[:, 1]], 1)
    drop_y = torch.stack([-v[:, 2], z, v[:, 0]], 1)
    drop_z = torch.stack([v[:, 1], -v[:, 0], z], 1)
    x_min = (a[:, 0] < a[:, 1]) & (a[:, 0] < a[:, 2])
    y_min = (a[:, 0] >= a[:, 1]) & (a[:, 1] < a[:, 2])
    return torch.where(x_min[:, None], drop_x, torch.where(y_min[:, None], drop_y, drop_z))


def _svd_rotation(F):
    """R = U V^T of the step's closed-form SVD (eigenvalues of F^T F by the trigonometric
    formula with a sine factor of 1, the flip to the better separated end, cofactor columns)."""
    A = _mm(_t(F), F)
    m = (A[:, 0, 0] + A[:, 1, 1] + A[:, 2, 2]) / 3.0
    eye = torch.eye(3, dtype=F.dtype, device=F.device)
    B = A - m[:, None, None] * eye
    p = (B * B).sum((1, 2)) / 6.0
    q = 0.5 * torch.linalg.det(B)
    phi = torch.atan2((p * p * p - q * q).clamp_min(0.0).sqrt(), q) / 3.0
    cs, sn = p.sqrt() * torch.cos(phi), p.sqrt() * torch.sin(phi)
    lam = torch.stack([m + 2.0 * cs, m - cs - sn, m - cs + sn], 1).sort(dim=1, descending=True).values
    flip = lam[:, 0] - lam[:, 1] < lam[:, 1] - lam[:, 2]
    first = torch.where(flip, lam[:, 2], lam[:, 0])
    last = torch.where(flip, lam[:, 0], lam[:, 2])
    M = A - first[:, None, None] * eye
    cof = torch.stack([torch.linalg.cross(M[:, 1], M[:, 2]), torch.linalg.cross(M[:, 2], M[:, 0]),
                       torch.linalg.cross(M[:, 0], M[:, 1])], 1)
    best = (cof * cof).sum(2).argmax(1)
    v1 = _unit(cof[torch.arange(F.shape[0], device=F.device), best])
    o0 = _unit(_orthogonal(v1))
    o1 = torch.linalg.cross(v1, o0)
    Ao0, Ao1 = (A * o0[:, None]).sum(2), (A * o1[:, None]).sum(2)
    r11, r21, r22 = (Ao0 * o0).sum(1) - last, (Ao1 * o0).sum(1), (Ao1 * o1).sum(1) - last
    w1, w2 = torch.stack([r22, -r21], 1), torch.stack([-r21, r11], 1)
    w = _unit(torch.where((w1.square().sum(1) > w2.square().sum(1))[:, None], w1, w2))
    v3 = o0 * w[:, :1] + o1 * w[:, 1:]
    v2 = torch.linalg.cross(v3, v1)
    f = flip[:, None]
    V = torch.stack([torch.where(f, v3, v1), v2, torch.where(f, -v1, v3)], 2)
    u0 = _unit((F * V[:, None, :, 0]).sum(2))
    n0 = _unit(_orthogonal(u0))
    n1 = torch.linalg.cross(u0, n0)
    t = _unit((F * V[:, None, :, 1]).sum(2))
    u1 = n0 * (n0 * t).sum(1, keepdim=True) + n1 * (n1 * t).sum(1, keepdim=True)
    U = torch.stack([u0, u1, torch.linalg.cross(u0, u1)], 2)
    return _mm(U, _t(V))


def _polar_rotation(F):
    """The polar factor by H <- (H + H^-T) / 2, at most ten times, per element until a pass
    moves it by at most 0.01 (squared norm)."""
    H = F.clone()
    live = torch.ones(F.shape[0], dtype=torch.bool, device=F.device)
    for _ in range(10):
        H1 = 0.5 * (H + torch.linalg.inv(H).transpose(1, 2))
        moved = (H1 - H).square().sum((1, 2))
        H = torch.where(live[:, None, None], H1, H)
        live = live & (moved > float(np.float32(0.01)))
    return H


class _Group:
    """Scenes of one solver, material and rotation as one system with per-scene scalars."""

    def __init__(self, scs):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t64 = lambda a: torch.as_tensor(np.asarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.sc = scs[0]
        self.M = len(scs)
        base = np.concatenate([[0], np.cumsum([s.num_nodes for s in scs])])
        self.N = int(base[-1])
        ids = np.concatenate([s.tets.astype(np.int64) + b for s, b in zip(scs, base)])
        self.ids = torch.as_tensor(ids, device=dev)
        self.flat = self.ids.reshape(-1)
        self.rest = t64(np.concatenate([s.rest for s in scs]))
        self.mesh = torch.as_tensor(np.repeat(np.arange(self.M), [s.num_nodes for s in scs]), device=dev)
        elem_mesh = np.repeat(np.arange(self.M), [s.num_tets for s in scs])
        per = lambda name, alt: t64(np.concatenate([  # noqa: E731
            getattr(s, name) if getattr(s, name) is not None else np.full(s.num_tets, getattr(s, alt)) for s in scs]))
        E, nu = per("young_per_elem", "young"), per("poisson_per_elem", "poisson")
        self.lam, self.mu = E * nu / ((1 + nu) * (1 - 2 * nu)), 0.5 * E / (1 + nu)
        D = self.edges(self.rest)
        self.vol = torch.linalg.det(D) / 6.0
        self.Di = torch.linalg.inv(D)
        total = torch.zeros(self.M, dtype=torch.float64, device=dev).index_add_(
            0, torch.as_tensor(elem_mesh, device=dev), self.vol)
        mass = total * t64([s.density for s in scs]) / t64([s.num_nodes for s in scs])
        self.mass = mass[self.mesh][:, None]
        self.g = t64([s.gravity for s in scs])[self.mesh]
        fixed = np.concatenate([s.knc_nodes.astype(np.int64) + b for s, b in zip(scs, base)])
        self.fixed = torch.as_tensor(fixed, device=dev)
        self.targets = t64(np.concatenate([s.knc_targets for s in scs]))
        self.rel2 = t64([s.rel_eps**2 for s in scs])
        self.abs2 = t64([s.abs_eps**2 for s in scs])
        self.cap = scs[0].max_iter
        self.dt = scs[0].dt

    def edges(self, x):
        p = x[self.ids]
        return (p[:, 1:] - p[:, :1]).transpose(1, 2)

    def evaluate(self, x):
        self.F = _mm(self.edges(x), self.Di)
        self.R = _polar_rotation(self.F) if self.sc.rotation else _svd_rotation(self.F)

    def nodal(self, P):
        """Element stresses to nodal sums: V P Dm^-T to nodes 1 to 3, minus their sum to 0."""
        h = _t(self.vol[:, None, None] * _mm(P, _t(self.Di)))
        h = torch.cat([-h.sum(1, keepdim=True), h], 1).reshape(-1, 3)
        return torch.zeros((self.N, 3), dtype=h.dtype, device=h.device).index_add_(0, self.flat, h)

    def warped(self, S):
        """R sigma(S) for a gradient S in the element frame."""
        eye = torch.eye(3, dtype=S.dtype, device=S.device)
        tr = S[:, 0, 0] + S[:, 1, 1] + S[:, 2, 2]
        sig = self.mu[:, None, None] * (S + _t(S)) + (self.lam * tr)[:, None, None] * eye
        return _mm(self.R, sig)

    def force(self, x):
        """Minus the elastic force: sum over the elements of K (u)."""
        eye = torch.eye(3, dtype=x.dtype, device=x.device)
        if self.sc.material:
            S = _mm(_t(self.R), self.F) - eye
            tr = S[:, 0, 0] + S[:, 1, 1] + S[:, 2, 2]
            return self.nodal(_mm(self.R, 2 * self.mu[:, None, None] * S + (self.lam * tr)[:, None, None] * eye))
        return self.nodal(self.warped(_mm(_t(self.R), _mm(self.edges(x), self.Di)) - eye))

    def K(self, d):
        H = _mm(self.edges(d), self.Di)
        if self.sc.material:
            tr = (self.R * H).sum((1, 2))
            return self.nodal(2 * self.mu[:, None, None] * H + (self.lam * tr)[:, None, None] * self.R)
        return self.nodal(self.warped(_mm(_t(self.R), H)))

    def A(self, fM, fK, d):
        q = fK * self.K(d) + fM * self.mass * d
        q[self.fixed] = 0.0
        return q

    def dot(self, a, b):
        s = (a * b).sum(1)
        if self.M == 1:
            return s.sum()[None]
        return torch.zeros(self.M, dtype=s.dtype, device=s.device).index_add_(0, self.mesh, s)

    def solve(self, fM, fK, b, y):
        return (self.minres if self.sc.ls_solver else self.cg)(fM, fK, b, y)

    def cg(self, fM, fK, b, y):
        r = b - self.A(fM, fK, y)
        r[self.fixed] = 0.0
        d = r.clone()
        new = self.dot(r, r)
        goal = torch.maximum(self.rel2 * new, self.abs2)
        at = lambda s: s[self.mesh][:, None]  # noqa: E731
        live = new > goal
        for _ in range(self.cap):
            if not bool(live.any()):
                break
            q = self.A(fM, fK, d)
            dq = self.dot(d, q)
            live = live & (dq.abs() >= self.abs2)
            alpha = torch.where(live, new / dq, torch.zeros_like(new))
            y = y + at(alpha) * d
            r = r - at(alpha) * q
            old, now = new, self.dot(r, r)
            new = torch.where(live, now, old)
            d = torch.where(at(live), r + at(new / old) * d, d)
            live = live & (new > goal)
        return y

    def minres(self, fM, fK, b, y):
        at = lambda s: s[self.mesh][:, None]  # noqa: E731
        r = b - self.A(fM, fK, y)
        r[self.fixed] = 0.0
        norm2 = self.dot(r, r)
        goal = torch.maximum(self.rel2 * self.dot(b, b), self.abs2)
        live = norm2 > goal
        beta = norm2.sqrt()
        first = beta.clone()
        v, v_old = r / at(beta), torch.zeros_like(r)
        p, p_old = torch.zeros_like(r), torch.zeros_like(r)
        one = torch.ones_like(beta)
        c, c_old, s, s_old, eta, beta_v = one, one, 0 * one, 0 * one, one, beta
        for _ in range(self.cap):
            if not bool(live.any()):
                break
            w = self.A(fM, fK, v) - at(beta_v) * v_old
            alpha = self.dot(w, v)
            w = w - at(alpha) * v
            beta_new = self.dot(w, w).sqrt()
            r2, r3 = s * alpha + c * c_old * beta_v, s_old * beta_v
            hat = c * alpha - c_old * s * beta_v
            r1 = (hat * hat + beta_new * beta_new).sqrt()
            c_old, s_old, c, s = c, s, hat / r1, beta_new / r1
            p_old, p = p, (v - at(r2) * p - at(r3) * p_old) / at(r1)
            y = torch.where(at(live), y + at(first * c * eta) * p, y)
            norm2 = torch.where(live, norm2 * s * s, norm2)
            eta = -s * eta
            live = live & (norm2 > goal)
            v_old, v, beta_v = v, w / at(beta_new), beta_new
        return y

    def step(self, x, v):
        dt = self.dt
        self.evaluate(x)
        if self.sc.integrator:
            xn, y = x, dt * v
            for k in range(self.sc.nr_max_iter):
                b = self.mass * self.g - self.force(x) + self.mass / dt * (v - (x - xn) / dt)
                b[self.fixed] = self.targets - x[self.fixed]
                if float(b.square().sum().sqrt()) < self.sc.nr_abs_eps:
                    break
                y = dt * v if k == 0 else torch.zeros_like(x)
                y[self.fixed] = b[self.fixed]
                x = x + self.solve(1.0 / dt / dt, 1.0, b, y)
                self.evaluate(x)
            return x, (x - xn) / dt
        b = dt * (self.mass * self.g - self.force(x)) + self.mass * v
        y = v.clone()
        vk = (self.targets - x[self.fixed]) / dt
        n = vk.norm(dim=1, keepdim=True)
        vk = torch.where(n > float(np.float32(0.001)), vk / n.clamp_min(1e-300) * n.clamp_max(50.0),
                         torch.zeros_like(vk))
        b[self.fixed] = vk
        y[self.fixed] = vk
        y = self.solve(1.0, dt * dt, b, y)
        return x + dt * y, y


def exact(case, seed):
    scs, rng = _scenes(case, seed)
    x, v = _states(scs, rng)
    if case["kind"] == "hooks":
        g = _Group(scs)
        x, d = torch.as_tensor(x, device=g.rest.device), torch.as_tensor(_probe(scs, rng), device=g.rest.device)
        g.evaluate(x)
        return {"f": (-g.force(x)).cpu(), "df": (-g.K(d)).cpu(), "q": g.A(1.0, g.dt * g.dt, d).cpu()}
    at = np.concatenate([[0], np.cumsum([s.num_nodes for s in scs])])
    groups = {}
    for i, sc in enumerate(scs):
        groups.setdefault((sc.ls_solver, sc.material, sc.rotation), []).append(i)
    xo, vo = np.empty_like(x), np.empty_like(v)
    for of in groups.values():
        g = _Group([scs[i] for i in of])
        pick = np.concatenate([np.arange(at[i], at[i + 1]) for i in of])
        xn, vn = g.step(torch.as_tensor(x[pick], device=g.rest.device), torch.as_tensor(v[pick], device=g.rest.device))
        xo[pick], vo[pick] = xn.cpu().numpy(), vn.cpu().numpy()
    return {"x": torch.from_numpy(xo), "v": torch.from_numpy(vo)}
