"""The global step resident in shared memory (csrc/resident.cuh) against the kernels it replaces
(jacobi_mode 1: one kernel per sweep): the same bits for the Jacobi sweeps and the learned step,
the same solution for conjugate gradients, whose FP64 sums are added in another order."""
import numpy as np
import pytest

from parallel_admm_b200 import backend as B
from parallel_admm_b200 import scene as S

pytestmark = pytest.mark.gpu

SCENES = {"cloth5": lambda: S.cloth_on_box(nx=5), "cloth33": lambda: S.cloth_on_box(nx=33),
          "cloth46": lambda: S.cloth_on_box(nx=46), "cube3": lambda: S.cube_on_ground(n=3, drop=0.01),
          "cube11": lambda: S.cube_on_ground(n=11, drop=0.01, rotate=True),
          "bodies": lambda: S.batch_bodies(n_bodies=6, seed=3, vmax=3000)}


def _pair(name, lanes, **kw):
    sc = SCENES[name]()
    hs = [B.Handle(sc, ell_lanes=lanes, jacobi_mode=m, **kw) for m in (1, 0)]
    assert hs[0].global_mode()["mode"] == "sweeps"
    assert hs[1].global_mode()["mode"] == "resident"
    rng = np.random.default_rng(7)
    x = sc.verts + rng.normal(scale=1e-3, size=sc.verts.shape).astype(np.float32)
    v = rng.normal(scale=0.2, size=sc.verts.shape).astype(np.float32)
    for h in hs:
        h.set_state(x, v)
    return hs


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("name", list(SCENES))
def test_sweeps_bitwise(name, lanes):
    a, b = _pair(name, lanes)
    for h in (a, b):
        h.pre_integration()
        h.local_step()
        h.global_step()
    assert np.array_equal(a.read(B.BUF_X), b.read(B.BUF_X))
    for sweeps in (1, 2, 3, 7):
        a.jacobi(sweeps)
        b.jacobi(sweeps)
        assert np.array_equal(a.read(B.BUF_X), b.read(B.BUF_X)), sweeps


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
@pytest.mark.parametrize("name", ["cloth5", "cloth46", "cube3", "cube11", "bodies"])
def test_two_sweeps_per_launch_bitwise(name, lanes):
    """jacobi_mode 3 (a tile of rows per block; tiles of fewer rows than a slice, and with more
    slices than the block has warps, among them)."""
    sc = SCENES[name]()
    hs = [B.Handle(sc, ell_lanes=lanes, jacobi_mode=m) for m in (1, 3)]
    rng = np.random.default_rng(5)
    x = sc.verts + rng.normal(scale=1e-3, size=sc.verts.shape).astype(np.float32)
    for h in hs:
        h.set_state(x)
        h.pre_integration()
        h.local_step()
        h.global_step()
    assert hs[1].global_mode()["mode"] == "tiled"
    for sweeps in (0, 2, 3, 4, 5):
        for h in hs:
            h.jacobi(sweeps)
        assert np.array_equal(hs[0].read(B.BUF_X), hs[1].read(B.BUF_X)), sweeps


@pytest.mark.parametrize("name", ["cloth33", "cube11", "bodies"])
def test_substeps_bitwise(name):
    a, b = _pair(name, 4)
    for _ in range(4):
        sa, sb = (h.step(1, allow=(B.ERR_CONTACT_OVERFLOW,)) for h in (a, b))
        assert sa["n_contacts"] == sb["n_contacts"]
        for p, q in zip(a.get_state(), b.get_state()):
            assert np.array_equal(p, q)
    assert b.kernels_per_step() < a.kernels_per_step()


@pytest.mark.parametrize("tol", [0.0, 1e-4])
@pytest.mark.parametrize("sweeps", [1, 5, 6, 7])
def test_learned_bitwise(sweeps, tol):
    # the schedule of sweep 6 steps backwards: its solves fail and are replaced
    a, b = _pair("cloth33", 2, global_solver=3, residual_tol=tol)
    omega = np.full(sweeps, -1.0 if sweeps == 6 else 0.9, np.float32)
    beta = np.full(sweeps, 0.1, np.float32)
    theta = np.full(a.n_dyn, 0.3, np.float32)
    for h in (a, b):
        h.set_learned(omega, beta, None, theta)
    for _ in range(3):
        for h in (a, b):
            h.step(1, allow=(B.ERR_CONTACT_OVERFLOW,))
        for p, q in zip(a.get_state(), b.get_state()):
            assert np.array_equal(p, q)
    assert a.learned_stats() == b.learned_stats()


@pytest.mark.parametrize("name", ["cloth5", "cloth33", "cube11"])
@pytest.mark.parametrize("solver", [1, 2])
def test_pcg(name, solver):
    a, b = _pair(name, 4, global_solver=solver, pcg_iter=25)
    blocks = np.zeros((a.n_dyn, 9), np.float32)
    blocks[:, [0, 4, 8]] = np.random.default_rng(2).uniform(0.5, 1.5, (a.n_dyn, 1)) / 10.0
    blocks[:, [1, 3]] = 0.01
    for h in (a, b):
        if solver == 2:
            h.set_preconditioner(blocks)
        h.pre_integration()
        h.local_step()
        h.global_step()
    x, y = a.read(B.BUF_X), b.read(B.BUF_X)
    assert np.abs(x - y).max() <= 1e-5 * max(1.0, np.abs(x).max())


@pytest.mark.parametrize("lanes", [1, 2, 4, 8])
def test_non_finite_body_stays_alone(lanes):
    """A CTA of the resident kernels holds rows of several bodies: one that has diverged, wherever
    its rows lie in the plan, leaves the others' sweeps as they were."""
    from scipy.sparse import coo_matrix
    from scipy.sparse.csgraph import connected_components
    sc = S.batch_bodies(n_bodies=12, seed=3, vmax=3000)
    e = sc.tet_inds[:, [0, 0, 0]].ravel(), sc.tet_inds[:, 1:].ravel()
    body = connected_components(coo_matrix((np.ones(len(e[0])), e), (sc.n_dyn, sc.n_dyn)), directed=False)[1]
    hs = [B.Handle(sc, ell_lanes=lanes, jacobi_mode=m) for m in (1, 0)]
    assert hs[1].global_mode()["mode"] == "resident"
    for h in hs:
        h.pre_integration()
        h.local_step()
        h.global_step()
    x0 = hs[0].read(B.BUF_X)
    for k, value in zip(range(body.max() + 1), (np.inf, -np.inf, np.nan) * 4):
        x = x0.copy()
        x[:sc.n_dyn][body == k] = value
        out = []
        for h in hs:
            h.write(B.BUF_X, x)
            h.jacobi(3)
            out.append(h.read(B.BUF_X)[:sc.n_dyn][body != k])
        assert np.isfinite(out[0]).all() and np.array_equal(out[0], out[1]), k


@pytest.mark.parametrize("sweeps", [31, 32, 33, 40])
def test_learned_step_before_its_model(sweeps):
    """Without a model the learned step runs jacobi_iter plain sweeps, more than a model may have."""
    a, b = _pair("cloth33", 2, global_solver=3, jacobi_iter=sweeps)
    for _ in range(2):
        for h in (a, b):
            h.step(1, allow=(B.ERR_CONTACT_OVERFLOW,))
        for p, q in zip(a.get_state(), b.get_state()):
            assert np.array_equal(p, q)
    assert a.learned_stats() == b.learned_stats()


@pytest.mark.parametrize("tol", [0.0, 1e-4])
@pytest.mark.parametrize("lanes", [1, 4])
def test_learned_bodies_bitwise(lanes, tol):
    """Several bodies in a group: vertex-wise m and theta, and one partial sum per CTA."""
    from parallel_admm_b200 import gnn
    SCENES["small bodies"] = lambda: S.batch_bodies(n_bodies=12, seed=3, vmin=100, vmax=600)
    a, b = _pair("small bodies", lanes, global_solver=3, residual_tol=tol)
    rng = np.random.default_rng(1)
    m = (rng.uniform(0.8, 1.1, a.n_dyn) / gnn.system(a).diag).astype(np.float32)
    theta = rng.uniform(-0.5, 0.5, a.n_dyn).astype(np.float32)
    for h in (a, b):
        h.set_learned(np.full(5, 0.9, np.float32), np.full(5, 0.1, np.float32), m, theta)
    for _ in range(3):
        for h in (a, b):
            h.step(1, allow=(B.ERR_CONTACT_OVERFLOW,))
        for p, q in zip(a.get_state(), b.get_state()):
            assert np.array_equal(p, q)
    assert a.learned_stats() == b.learned_stats()
