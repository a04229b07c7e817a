"""The grid queries over the ranges their kernel treats differently, against the oracle's pair set:
ranges of a few cells, of several lists of cells, too wide for one lane group (walked by the whole
warp), elements too large for the grid, and more partners than the count pass records."""
import numpy as np
import pytest

from parallel_admm_b200 import backend as B
from parallel_admm_b200 import scene

pytestmark = pytest.mark.gpu


def _scattered(scales, spread, seed):
    """Small sheets, each stretched by one of `scales`, turned and moved at random."""
    rng = np.random.default_rng(seed)
    v, f = scene.grid_cloth(3, 0.06)
    bodies = [scene._Body(v + np.array([0.0, 0.2 * k, 0.0]), f, np.zeros((0, 4), np.int32), 0.1, 1e3, 1e-3)
              for k in range(len(scales))]
    sc = scene.assemble("scattered", bodies, [], scene.SolverParams(thickness=5e-3, max_contacts=1_000_000))
    x = sc.verts.astype(np.float64).copy()
    n = len(v)
    for k, scale in enumerate(scales):
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        p = x[k * n:(k + 1) * n]
        x[k * n:(k + 1) * n] = (p - p.mean(0)) * scale @ q + rng.uniform(-spread, spread, size=3)
    return sc, np.ascontiguousarray(x, np.float32)


CASES = {
    "few": ([1.0] * 3, 0.02),
    "lists": ([1.0] * 20 + [6.0] * 6, 0.08),
    "wide": ([1.0] * 24 + [8.0] * 4 + [16.0] * 3, 0.1),
    "big": ([1.0] * 24 + [16.0] * 2 + [60.0] * 3, 0.1),
    "many": ([0.25] * 40, 0.002),
}


@pytest.mark.parametrize("semantics", [0, 1])
@pytest.mark.parametrize("lanes", [0, 8, 16, 32])
@pytest.mark.parametrize("case", list(CASES))
def test_grid_query_ranges(case, lanes, semantics):
    from oracle import oracle as O
    sc, x = _scattered(*CASES[case], seed=len(case))
    sc.params.query_lanes = lanes
    sc.params.contact_semantics = semantics
    sc.params.broad_phase = 2
    h = B.Handle(sc)
    n = h.detect(x)
    kw = dict(semantics=1, static_begin=sc.n_dyn) if semantics else {}
    ref, _ = O.dcd(x, sc.surf_verts, sc.surf_tris, sc.surf_edges, sc.params.thickness, **kw)
    assert n == len(ref) and n > 0
    assert sorted(map(tuple, h.contacts()["pairs"].tolist())) == sorted(map(tuple, ref.tolist()))
    h.close()


@pytest.mark.parametrize("lanes", [8, 16, 32])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_vertex(value, lanes):
    """A vertex without a finite position leaves the pairs of the elements that it is no part of as
    they are when it is far away."""
    sc, x = _scattered(*CASES["lists"], seed=5)
    sc.params.query_lanes = lanes
    sc.params.broad_phase = 2
    v = 100
    out = []
    for p in ((50.0, 50.0, 50.0), (value, value, value), (float(x[v, 0]), value, float(x[v, 2]))):
        h = B.Handle(sc)
        y = x.copy()
        y[v] = p
        h.detect(y)
        pairs = h.contacts()["pairs"]
        out.append(sorted(map(tuple, pairs[(pairs != v).all(1)].tolist())))
        h.close()
    assert out[0] and out[1] == out[0] and out[2] == out[0]


@pytest.mark.parametrize("n", [8, 56])
def test_contact_arrays_one_by_one(n):
    """Contacts read all at once (records up to 4096 of them, arrays above) and array by array."""
    import ctypes
    v, f = scene.grid_cloth(n, 1.0)
    e = 1.0 / (n - 1)
    bodies = [scene._Body(v + np.array([0.0, 0.5 + 0.3 * e * k, 0.0]), f, np.zeros((0, 4), np.int32), 0.1, 1e3, 1e-3)
              for k in range(2)]
    h = B.Handle(scene.assemble("two", bodies, [], scene.SolverParams(thickness=e, max_contacts=1_000_000)))
    k = h.detect()
    assert (k > 4096) == (n == 56)
    every = h.contacts()
    names = ["pairs", "bary", "normal", "point", "gap"]
    cnt = ctypes.c_int32()
    for ask in [(name,) for name in names] + [("pairs", "point"), ("bary", "normal", "point"), ("pairs", "gap", "point")]:
        out = {a: np.zeros_like(every[a]) for a in ask}
        ptr = [out[a].ctypes.data_as(ctypes.POINTER(ctypes.c_int32 if a == "pairs" else ctypes.c_float)) if a in out
               else None for a in names]
        assert B.lib().admm_b200_contacts(h.h, *ptr, k, ctypes.byref(cnt)) == B.OK and cnt.value == k
        assert all(np.array_equal(out[a], every[a]) for a in ask), ask
    h.close()
