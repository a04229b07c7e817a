"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one call (or one training iteration) through the public entry points of
``parallel_admm_b200``: substeps of the benchmark's scene families from host positions and
velocities (``Handle.step_host``, the boundary's per-step host synchronisation), the collision
detector on its own (``BVHB200.detect``), the global step on its own, the learned step's network
(set-up of a new scene, and training), the converged solve that makes its training data, and the
allocation-free Jacobi solve on a caller's device buffers.

Scenes are those of ``parallel_admm_b200.scene`` (bench.py and the tests use the same ones) at the
sizes of the configurations and below; the seed makes the state: a rotation or a wave of the
bodies, the gap to the collider and the velocities.  The lanes per matrix row are pinned (an
option of the description) so that all handles of a case sum in the same order; everything else is
the default.  Substeps start from the same positions and velocities in every pass, the dual
variables stay warm from pass to pass.
"""
import ctypes
import functools
import math
import os

import numpy as np
import torch

from parallel_admm_b200 import backend as B
from parallel_admm_b200 import gnn
from parallel_admm_b200 import scene as S

WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(gnn.__file__)), "weights")
MODELS = {"batch": "learned_step.npz", "cube": "learned_step_cube.npz", "sheets": "learned_step_sheets.npz",
          "cloth": "learned_step_sheets.npz"}


def listed():
    return [
        # the interactive size: the 32 x 32 cloth swinging down onto the box, launch-bound
        {"name": "cloth step", "kind": "step", "scene": "cloth", "size": 32, "solver": "jacobi", "lanes": 4},
        # the reference CPU backend's solver on the same cloth: damped system, conjugate gradients
        # to convergence, serial contact
        {"name": "cloth step, CPU backend", "kind": "step", "scene": "cloth", "size": 32, "solver": "cpu", "lanes": 4},
        # one soft body of 9261 vertices at the moment it hits the ground
        {"name": "cube step", "kind": "step", "scene": "cube", "size": 20, "solver": "jacobi", "lanes": 4},
        # a batch of uneven bodies on the ground with the reference's Jacobi step (several times the
        # work of the cube), and with the learned step run to the residual tolerance as in bench.py
        {"name": "batch step", "kind": "step", "scene": "batch", "size": 24, "solver": "jacobi", "lanes": 2},
        {"name": "batch step, learned", "kind": "step", "scene": "batch", "size": 16, "solver": "learned", "lanes": 2},
        # cloth sheets falling onto a sphere: triangle and bending rows, many edge-edge queries
        {"name": "sheets step", "kind": "step", "scene": "sheets", "size": 128, "solver": "jacobi", "lanes": 2},
        # the collision detector alone, as the application's display and tools call it
        {"name": "detect", "kind": "detect", "scene": "batch", "size": 16},
        # the global step alone, read back on the host (the linear solver's own entry point)
        {"name": "global step", "kind": "global", "scene": "cube", "size": 20, "lanes": 4},
        # the learned step's network on a new scene: what a user pays once per scene
        {"name": "network outputs", "kind": "outputs", "scene": "cube", "size": 20},
        # one iteration of training on a batch of four bodies, the family of the shipped model
        {"name": "training iteration", "kind": "train", "scene": "batch", "size": 4, "sweeps": 6, "samples": 4},
        # converged solve of one training sample
        {"name": "converged solve", "kind": "solve", "scene": "cube", "size": 20},
        # Jacobi sweeps on a caller's own device buffers, on the caller's stream
        {"name": "allocation-free Jacobi", "kind": "noalloc", "scene": "batch", "size": 4, "sweeps": 20},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 5 + ["detect", "global", "outputs", "train", "solve", "noalloc"])
    if kind == "step":
        what = rng.choice(["cloth", "cloth", "cube", "cube", "batch", "sheets"])
        size = {"cloth": (12, 64), "cube": (5, 24), "batch": (3, 24), "sheets": (32, 128)}[what]
        solvers = {"cloth": ["jacobi", "jacobi", "cpu"], "cube": ["jacobi", "learned"],
                   "batch": ["jacobi", "learned"], "sheets": ["jacobi", "learned"]}[what]
        solver = rng.choice(solvers)
        n = _log_int(rng, *((12, 40) if solver == "cpu" else size))
        return {"kind": kind, "scene": what, "size": n, "solver": solver, "lanes": rng.choice([1, 2, 4, 8])}
    if kind == "detect":
        what = rng.choice(["cube", "batch", "sheets"])
        return {"kind": kind, "scene": what,
                "size": _log_int(rng, *{"cube": (8, 28), "batch": (3, 20), "sheets": (32, 128)}[what])}
    if kind == "global":
        what = rng.choice(["cloth", "cube", "sheets"])
        return {"kind": kind, "scene": what, "lanes": rng.choice([1, 2, 4, 8]),
                "size": _log_int(rng, *{"cloth": (12, 64), "cube": (5, 28), "sheets": (32, 96)}[what])}
    if kind == "train":
        what = rng.choice(["cube", "batch"])
        return {"kind": kind, "scene": what, "size": _log_int(rng, *{"cube": (6, 22), "batch": (2, 4)}[what]),
                "sweeps": rng.randint(4, 12), "samples": rng.randint(1, 6)}
    what = rng.choice(["cube", "sheets"])
    case = {"kind": kind, "scene": what, "size": _log_int(rng, *{"cube": (6, 24), "sheets": (24, 80)}[what])}
    if kind == "noalloc":
        case["sweeps"] = _log_int(rng, 1, 40)
    return case


# ------------------------------------------------------------------------------------------------
# scenes and states
# ------------------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=3)
def _scene(what, size):
    """The scene of a family at a size (host arrays; its geometry does not depend on the seed)."""
    if what == "cloth":
        return S.cloth_on_box(nx=size)
    if what == "cube":
        return S.cube_on_ground(n=size, E=1e5)
    if what == "sheets":
        return S.sheets_on_sphere(nx=size, layers=2)
    return S.batch_bodies(n_bodies=size, seed=7)


def _state(sc, what, seed):
    """Positions and velocities at the moment that the scene's bodies meet their collider."""
    rng = np.random.default_rng(seed)
    x = sc.verts.astype(np.float64).copy()
    v = np.zeros_like(x)
    nd = sc.n_dyn
    d = x[:nd]
    if what == "cloth":
        # the sheet swung down about its pinned edge until its free edge is at the box's top
        pins = d[sc.pin_inds]
        a, e = pins[0], (pins[1] - pins[0]) / np.linalg.norm(pins[1] - pins[0])
        r = d - a
        along = (r @ e)[:, None] * e
        out = r - along
        s = np.linalg.norm(out, axis=1)
        u = out / np.maximum(s, 1e-9)[:, None]
        u[s < 1e-3] = 0.0
        ang = math.radians(29.8) + rng.uniform(-0.004, 0.002)
        wave = 2e-3 * np.sin(2 * math.pi * (rng.uniform(1, 3) * (r @ e) + rng.uniform())) * np.minimum(s / 0.2, 1.0)
        down = np.array([0.0, -1.0, 0.0])
        d[:] = a + along + s[:, None] * (math.cos(ang) * u + math.sin(ang) * down) + wave[:, None] * down
        v[:nd] = (s * rng.uniform(1.0, 3.0))[:, None] * (math.cos(ang) * down - math.sin(ang) * u)
        v[sc.pin_inds] = 0.0
    elif what == "cube":
        c = d.mean(0)
        tilt = rng.uniform(-0.05, 0.05, size=2)
        cx, sx, cz, sz = math.cos(tilt[0]), math.sin(tilt[0]), math.cos(tilt[1]), math.sin(tilt[1])
        rot = np.array([[1, 0, 0], [0, cx, -sx], [0, sx, cx]]) @ np.array([[cz, -sz, 0], [sz, cz, 0], [0, 0, 1]])
        d[:] = (d - c) @ rot.T
        d[:, 1] += -d[:, 1].min() + rng.uniform(0.002, 0.015)
        v[:nd, 1] = -rng.uniform(2.0, 4.4)
    elif what == "sheets":
        for k in range(2):
            w = slice(k * (nd // 2), (k + 1) * (nd // 2))
            q = d[w]
            f = rng.uniform(1.0, 3.0, size=2)
            q[:, 1] += 0.012 * np.sin(2 * math.pi * (f[0] * q[:, 0] + f[1] * q[:, 2]) + rng.uniform(0, 6))
            v[:nd][w] = [rng.uniform(-0.2, 0.2), rng.uniform(-1.2, -0.6), rng.uniform(-0.2, 0.2)]
        near = np.hypot(d[:, 0], d[:, 2]) < 0.05
        d[:, 1] -= d[near, 1].min() - x[nd:, 1].max() - 5e-4
    else:
        d[:, 1] -= rng.uniform(0.0, 4e-3)
        d[:] += rng.normal(scale=2e-4, size=d.shape)
        v[:nd] = rng.normal(scale=0.05, size=(nd, 3)) + [0.0, -rng.uniform(0.1, 0.5), 0.0]
    return x.astype(np.float32), v.astype(np.float32)


def _pinned(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.float32)).pin_memory().numpy()


def _options(case):
    o = {"ell_lanes": case.get("lanes", 4)}
    if case.get("solver") == "learned":
        o.update(global_solver=3, residual_tol=1e-4)
    elif case.get("solver") == "cpu":
        o.update(backend_semantics=1, contact_semantics=1, global_solver=1, pcg_iter=150)
    return o


class State:
    pass


def _system(case, st):
    """The global matrix of the scene and the network's features for it."""
    sc = _scene(case["scene"], case["size"])
    h = B.Handle(sc, ell_lanes=4, jacobi_mode=1)
    st.sysm = gnn.system(h)
    h.close()
    return sc


def _samples(st, sc, case, seed, count):
    """Right-hand sides, iterates and solutions of the global step's kind: the solution is a
    displaced shape, the received iterate is off by a rough field, the one before it by another."""
    rng = np.random.default_rng(seed)
    n = st.sysm.n
    base = sc.verts[:n].astype(np.float64)
    rows = []
    for _ in range(count):
        k = rng.uniform(2, 8, size=3)
        xs = base + 0.01 * np.sin(base @ np.diag(k) + rng.uniform(0, 6, 3))
        rough = rng.normal(scale=2e-4, size=xs.shape)
        xc = xs + rough + 1e-3 * np.cos(base[:, [1, 2, 0]] * k)
        rows.append((st.sysm.matvec(xs), xc, xc + 0.5 * rough + 3e-4 * np.sin(base * k), xs))
    return tuple(np.stack(a).astype(np.float32) for a in zip(*rows))


def _chebyshev(K):
    om, be = gnn.chebyshev_coefficients(K, 0.2, 2.0)
    return om, be


def prepare(case, seed):
    st = State()
    st.case = dict(case)
    kind = case["kind"]
    if kind in ("step", "detect", "global"):
        sc = _scene(case["scene"], case["size"])
        st.sc = sc
        st.h = B.Handle(sc, **_options(case))
        x, v = _state(sc, case["scene"], seed)
    if kind == "step":
        if case["solver"] == "learned":
            model = gnn.LearnedGlobalStep.load(os.path.join(WEIGHTS, MODELS[case["scene"]]))
            sysm = gnn.system(st.h)
            model.apply(st.h, sysm, *gnn.scene_features(sc, sysm))
            model.net.close()
        st.x, st.v = _pinned(x), _pinned(v)
        st.x_out, st.v_out = _pinned(np.zeros_like(x)), _pinned(np.zeros_like(v))
    elif kind == "detect":
        st.x = x
        st.det = B.BVHB200(st.h)
        st.slots = 16384  # the display's own arrays, zero past the contact count
        st.out = {"pairs": np.zeros((st.slots, 4), np.int32), "bary": np.zeros((st.slots, 4), np.float32),
                  "normal": np.zeros((st.slots, 3), np.float32), "point": np.zeros((st.slots, 3), np.float32),
                  "gap": np.zeros(st.slots, np.float32)}
    elif kind == "global":
        rng = np.random.default_rng(seed + 1)
        st.x0, st.v0 = x, v
        st.h.set_state(x, v)
        st.h.pre_integration()
        st.z = (_rows(sc, torch.from_numpy(x).double()).numpy()
                + rng.normal(scale=1e-2, size=(sc.n_rows, 3))).astype(np.float32)
        st.h.write(B.BUF_Z, st.z)
        st.p = v.copy()
        st.h.write(B.BUF_P, st.p)
    else:
        sc = _system(case, st)
        st.feat, st.edge = gnn.scene_features(sc, st.sysm)
        if kind in ("outputs", "train"):
            st.model = gnn.LearnedGlobalStep.load(os.path.join(WEIGHTS, MODELS[case["scene"]]))
            rng = np.random.default_rng(seed)
            st.params = (st.model.net.params() * (1 + 0.05 * rng.standard_normal(st.model.net.P))).astype(np.float32)
            st.model.net.set_params(st.params)
            st.model.net.bind(st.sysm, st.feat, st.edge)
        if kind == "train":
            st.omega, st.beta = _chebyshev(case["sweeps"])
            st.trainer = gnn.SweepTrainer(st.sysm, residual_weight=0.05)
            st.S = _samples(st, sc, case, seed, case["samples"])
        elif kind == "solve":
            st.trainer = gnn.SweepTrainer(st.sysm)
            b, xc, _, _ = _samples(st, sc, case, seed, 1)
            st.b, st.xc = b[0], xc[0]
        elif kind == "noalloc":
            b, xc, _, _ = _samples(st, sc, case, seed, 1)
            up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
            st.dev = [up(a) for a in (st.sysm.start, st.sysm.col, st.sysm.val, st.sysm.diag, b[0], xc[0])]
            st.b, st.xc = b[0], xc[0]
            st.out = torch.zeros_like(st.dev[5])
    return st


def run(st):
    case = st.case
    kind = case["kind"]
    if kind == "step":
        st.h.step_host(st.x, st.v, st.x_out, st.v_out)
        return {"x": st.x_out, "v": st.v_out}
    if kind == "detect":
        st.det.detect(st.x)
        count = ctypes.c_int32()
        p = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_int32 if a.dtype == np.int32 else ctypes.c_float))
             for a in st.out.values()]
        rc = B.lib().admm_b200_contacts(st.h.h, *p, st.slots, ctypes.byref(count))
        if rc != B.OK:
            raise RuntimeError(f"admm_b200_contacts: status {rc}")
        for a in st.out.values():
            a[count.value:] = 0
        return {"count": count.value, **st.out}
    if kind == "global":
        st.h.global_step()
        return {"x": st.h.read(B.BUF_X)}
    if kind == "outputs":
        m, th = st.model.outputs(st.sysm, st.feat, st.edge)
        return {"m": m, "theta": th}
    if kind == "train":
        m, th = st.model.outputs(st.sysm, st.feat, st.edge)
        loss, go, gb, gm, gt = st.trainer.loss_grad(st.omega, st.beta, m, th, *st.S)
        grad = st.model.net.backward(st.sysm, st.feat, st.edge, gm, gt)
        st.model.net.step(1e-6)
        return {"loss": loss, "omega": go, "beta": gb, "m": gm, "theta": gt, "params": grad}
    if kind == "solve":
        x, _ = st.trainer.solve(st.b, st.xc)
        return {"x": x}
    n = st.sysm.n
    p = [ctypes.c_void_p(t.data_ptr()) for t in st.dev]
    rc = B.lib().admm_b200_jacobi_noalloc(n, p[0], p[1], p[2], p[3], p[4], p[5], ctypes.c_void_p(st.out.data_ptr()),
                                          case["sweeps"], ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != B.OK:
        raise RuntimeError(f"admm_b200_jacobi_noalloc: status {rc}")
    return st.out


# ------------------------------------------------------------------------------------------------
# bytes and operations
# ------------------------------------------------------------------------------------------------

def _offdiag(sc):
    """Off-diagonal entries of the global matrix: vertex pairs that share an element (a lattice of
    tets has about 13 neighbours per vertex, a cloth with bending rows about 18)."""
    return 13 * sc.n_dyn if len(sc.tet_inds) else 18 * sc.n_dyn


def work(case):
    sc = _scene(case["scene"], case["size"])
    nd, nnz, rows = sc.n_dyn, _offdiag(sc), sc.n_rows
    matrix = 8 * nnz + 4 * nd
    ring = int(sc.bend_offsets[-1]) if len(sc.bend_w) else 0
    entries = 12 * len(sc.tet_inds) + 6 * len(sc.tri_inds) + ring + len(sc.pin_inds)
    records = 52 * len(sc.tet_inds) + 28 * len(sc.tri_inds) + 8 * ring + 16 * len(sc.pin_inds)
    surface = 12 * len(sc.surf_tris) + 8 * len(sc.surf_edges) + 4 * len(sc.surf_verts)
    sweep = 6 * nnz + 6 * nd
    kind = case["kind"]
    if kind == "step":
        iters = sc.params.admm_max_iter
        sweeps = {"jacobi": sc.params.jacobi_iter, "learned": 7, "cpu": 150}[case["solver"]]
        local = 400 * len(sc.tet_inds) + 300 * len(sc.tri_inds) + 6 * ring
        return {"bytes": 48 * sc.n_vert + matrix + 8 * entries + records + surface + 48 * rows,
                "flops": iters * (sweeps * sweep + local + 6 * entries)}
    if kind == "detect":
        return {"bytes": 12 * sc.n_vert + surface, "flops": 100 * (len(sc.surf_verts) + len(sc.surf_edges))}
    if kind == "global":
        return {"bytes": matrix + 8 * entries + 12 * rows + 60 * nd, "flops": sc.params.jacobi_iter * sweep + 6 * entries}
    if kind in ("outputs", "train"):
        layer = 2 * 64 * (130 * nnz + 128 * nd)
        forward = 3 * layer + 2 * 64 * 13 * nd
        if kind == "outputs":
            return {"bytes": matrix + 8 * nnz + 24 * nd + 8 * nd, "flops": forward}
        K, count = case["sweeps"], case["samples"]
        return {"bytes": matrix + 8 * nnz + 24 * nd + 48 * nd * count + 16 * nd,
                "flops": 3 * forward + count * (2 * K + 4) * sweep}
    if kind == "solve":
        return {"bytes": matrix + 36 * nd, "flops": 60 * (sweep + 24 * nd)}
    return {"bytes": matrix + 36 * nd, "flops": case["sweeps"] * sweep}


# ------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------

def _gradient_rows(sc):
    """Per element type: (vertex indices, coefficients [elements, rows, vertices], first row)."""
    out = []
    if len(sc.tri_inds):
        Bi = torch.from_numpy(sc.tri_binv).double().reshape(-1, 2, 2)
        out.append((sc.tri_inds, torch.stack([-(Bi[:, 0] + Bi[:, 1]), Bi[:, 0], Bi[:, 1]], 2), sc.tri_start_row))
    if len(sc.tet_inds):
        Bi = torch.from_numpy(sc.tet_binv).double().reshape(-1, 3, 3)
        out.append((sc.tet_inds, torch.stack([-Bi.sum(1), Bi[:, 0], Bi[:, 1], Bi[:, 2]], 2), sc.tet_start_row))
    return [(torch.from_numpy(np.asarray(i)).long(), g, r) for i, g, r in out]


def _rows(sc, x):
    """D x: the rows of every constraint, from the vertices' positions."""
    y = torch.zeros((sc.n_rows, 3), dtype=torch.float64)
    for idx, g, r in _gradient_rows(sc):
        v = torch.einsum("erv,evc->erc", g, x[idx]).reshape(-1, 3)
        y[r:r + len(v)] = v
    if len(sc.bend_w):
        row = torch.from_numpy(np.repeat(np.arange(len(sc.bend_w)), np.diff(sc.bend_offsets))).long()
        c = torch.from_numpy(sc.bend_coeffs).double()
        y[sc.bend_start_row:sc.bend_start_row + len(sc.bend_w)].index_add_(0, row, c[:, None] * x[torch.from_numpy(sc.bend_inds).long()])
    if len(sc.pin_inds):
        y[sc.pin_start_row:] = x[torch.from_numpy(sc.pin_inds).long()]
    return y


def _rows_t(sc, y, square=False):
    """D^T y (square: the sums of the squared coefficients instead, for the diagonal)."""
    f = (lambda c: c * c) if square else (lambda c: c)
    x = torch.zeros((sc.n_dyn, 3), dtype=torch.float64)
    for idx, g, r in _gradient_rows(sc):
        e, q = g.shape[0], g.shape[1]
        v = torch.einsum("erv,erc->evc", f(g), y[r:r + e * q].reshape(e, q, 3))
        x.index_add_(0, idx.reshape(-1), v.reshape(-1, 3))
    if len(sc.bend_w):
        row = torch.from_numpy(np.repeat(np.arange(len(sc.bend_w)), np.diff(sc.bend_offsets))).long()
        c = f(torch.from_numpy(sc.bend_coeffs).double())
        x.index_add_(0, torch.from_numpy(sc.bend_inds).long(), c[:, None] * y[sc.bend_start_row:][:len(sc.bend_w)][row])
    if len(sc.pin_inds):
        x.index_add_(0, torch.from_numpy(sc.pin_inds).long(), y[sc.pin_start_row:])
    return x


def _exact_global(st):
    sc, p = st.sc, st.sc.params
    nd, dt = sc.n_dyn, float(np.float32(p.dt))
    w = torch.zeros(sc.n_rows, dtype=torch.float64)
    for start, ww, per in ((sc.tri_start_row, sc.tri_w, 2), (sc.tet_start_row, sc.tet_w, 3),
                           (sc.bend_start_row, sc.bend_w, 1), (sc.pin_start_row, sc.pin_w, 1)):
        w[start:start + per * len(ww)] = torch.from_numpy(np.repeat(ww.astype(np.float64), per))
    w2 = (w * w * dt * dt)[:, None]
    mass = torch.from_numpy(sc.mass[:nd]).double()[:, None]
    wc = torch.from_numpy(np.where(sc.is_surf()[:nd] > 0, sc.contact_w[:nd].astype(np.float64) * dt * dt, 0.0))[:, None]
    x0, v0 = torch.from_numpy(st.x0[:nd]).double(), torch.from_numpy(st.v0[:nd]).double()
    free = torch.from_numpy((sc.is_fixed[:nd] == 0).astype(np.float64))[:, None]
    g = torch.tensor([0.0, -float(np.float32(p.g)) * dt, 0.0], dtype=torch.float64)
    x = x0 + free * (v0 + g) * dt
    b = mass * x + _rows_t(sc, w2 * torch.from_numpy(st.z).double())
    b = b + wc * (torch.from_numpy(st.p[:nd]).double() * dt + x0)
    diag = mass + wc + _rows_t(sc, w2.expand(-1, 3), square=True)
    full = torch.from_numpy(st.x0).double()
    for _ in range(p.jacobi_iter):
        full[:nd] = x
        x = x + (b - (mass + wc) * x - _rows_t(sc, w2 * _rows(sc, full))) / diag
    full[:nd] = x
    return full


def _matrix(sysm):
    rows = torch.from_numpy(np.repeat(np.arange(sysm.n), np.diff(sysm.start))).long()
    col, val = torch.from_numpy(sysm.col).long(), torch.from_numpy(sysm.val).double()
    diag = torch.from_numpy(sysm.diag).double()[:, None]

    def off(v):
        return torch.zeros_like(v).index_add(0, rows, val[:, None] * v[col])
    return rows, col, diag, off


def _network(st, theta):
    """The network in 64 bits on parameters `theta` (weights as the kernels see them)."""
    h, k = 64, 0

    def take(shape):
        nonlocal k
        n = int(np.prod(shape))
        v = theta[k:k + n].reshape(shape)
        k += n
        return v
    rows, col, diag, _ = _matrix(st.sysm)
    x, ef = torch.from_numpy(st.feat).double(), torch.from_numpy(st.edge).double()
    deg = torch.from_numpy(np.maximum(np.diff(st.sysm.start), 1)).double()[:, None]
    W, bias = take((h, 6)), take((h,))
    a = torch.relu(x @ W.T + bias)
    for _ in range(3):
        We, be, Wn, bn = take((h, 130)), take((h,)), take((h, 128)), take((h,))
        # the edge layer by its three parts: W [h_row, h_col, edge]
        part = a @ We[:, 64:128].T
        msg = torch.relu((a @ We[:, :64].T)[rows] + part[col] + ef @ We[:, 128:].T + be)
        agg = torch.zeros_like(a).index_add(0, rows, msg) / deg
        a = a + torch.relu(torch.cat([a, agg], 1) @ Wn.T + bn)
    W, bias = take((7, h)), take((7,))
    o = a @ W.T + bias
    d = torch.exp(o[:, :3].clamp(-8, 8))
    tr = (d * d).sum(1) + (o[:, 3:6] ** 2).sum(1)
    return tr / diag[:, 0] / 3.0, o[:, 6].clamp(-1, 1)


def _kernel_weights(st):
    """The parameters in 64 bits, the weight matrices rounded to BF16 where the model has them so."""
    t = torch.from_numpy(st.params).clone()
    if st.model.net.bf16:
        h, k = 64, 0
        shapes = [(h, 6), (h,)] + [(h, 130), (h,), (h, 128), (h,)] * 3 + [(7, h), (7,)]
        for s in shapes:
            n = int(np.prod(s))
            if len(s) == 2:
                t[k:k + n] = t[k:k + n].bfloat16().float()
            k += n
    return t.double()


def _exact_train(st):
    K = st.case["sweeps"]
    theta = _kernel_weights(st).requires_grad_()
    m, th = _network(st, theta)
    _, _, diag, off = _matrix(st.sysm)
    om = torch.from_numpy(st.omega).double().requires_grad_()
    be = torch.from_numpy(st.beta).double().requires_grad_()
    md, td = m.detach().requires_grad_(), th.detach().requires_grad_()
    total = 0.0
    count = st.S[0].shape[0]
    for s in range(count):
        b, xc, xl, xs = (torch.from_numpy(a[s]).double() for a in st.S)
        A = lambda v: diag * v + off(v)  # noqa: E731
        ec = xc - xs
        aec = A(ec)
        prev = x = xc + td[:, None] * (xc - xl)
        for k in range(K):
            nxt = x + om[k] * md[:, None] * (b - A(x))
            if k:
                nxt = nxt + be[k] * (x - prev)
            prev, x = x, nxt
        e = x - xs
        ae = A(e)
        total = total + (e * ae).sum() / (ec * aec).sum() + 0.05 * (ae * ae).sum() / (aec * aec).sum()
    loss = total / count
    go, gb, gm, gt = torch.autograd.grad(loss, (om, be, md, td))
    (grad,) = torch.autograd.grad((m * gm).sum() + (th * gt).sum(), theta)
    return {"loss": loss.detach(), "omega": go, "beta": gb, "m": gm, "theta": gt, "params": grad}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "detect"):
        return None  # a whole substep or detection: no short restatement
    st = prepare(case, seed)
    if kind == "global":
        return {"x": _exact_global(st)}
    if kind == "outputs":
        m, th = _network(st, _kernel_weights(st))
        return {"m": m, "theta": th}
    if kind == "train":
        return _exact_train(st)
    _, _, diag, off = _matrix(st.sysm)
    b, x = torch.from_numpy(st.b).double(), torch.from_numpy(st.xc).double()
    if kind == "noalloc":
        for _ in range(case["sweeps"]):
            x = (b - off(x)) / diag
        return x
    r = b - diag * x - off(x)  # conjugate gradients to 64-bit convergence
    z = r / diag
    p, rz = z, (r * z).sum()
    first = rz
    for _ in range(5000):
        if rz <= 1e-24 * first:
            break
        q = diag * p + off(p)
        a = rz / (p * q).sum()
        x, r = x + a * p, r - a * q
        z = r / diag
        new = (r * z).sum()
        p, rz = z + (new / rz) * p, new
    return {"x": x}
