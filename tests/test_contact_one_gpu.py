"""The contact passes in one block against a launch per pass: identical bits.  A scene of more than
8192 surface vertices always takes the launches, so the same bodies with a large sheet far away
give the other side."""
import numpy as np
import pytest

from parallel_admm_b200 import backend as B
from parallel_admm_b200 import scene

pytestmark = pytest.mark.gpu


def _stack(layers, n, far=False):
    v, f = scene.grid_cloth(n, 0.1)
    none = np.zeros((0, 4), np.int32)
    bodies = [scene._Body(v + np.array([0.0, 0.5 + 2e-3 * k, 0.0]), f, none, 0.1, 1e3, 1e-3) for k in range(layers)]
    if far:
        w, g = scene.grid_cloth(92, 4.0)
        bodies.append(scene._Body(w + np.array([50.0, 0.0, 0.0]), g, none, 0.1, 1e3, 1e-3))
    sc = scene.assemble("stack", bodies, [], scene.SolverParams(thickness=5e-3, max_contacts=1_000_000, ell_lanes=4))
    x = sc.verts.astype(np.float64).copy()
    m = layers * len(v)
    x[:m] += np.random.default_rng(layers).normal(scale=2e-4, size=(m, 3))
    return sc, x, m


@pytest.mark.parametrize("layers,n,lo,hi", [(2, 2, 1, 31), (3, 6, 513, 768), (3, 8, 769, 1 << 20), (12, 6, 769, 1 << 20)],
                         ids=["few", "one block", "more than a block", "long lists"])
def test_contact_passes_in_one_block(layers, n, lo, hi):
    out = []
    for far in (False, True):
        sc, x, m = _stack(layers, n, far)
        uc = np.zeros((sc.n_dyn, 3))
        uc[:m] = np.random.default_rng(3).normal(scale=1e-4, size=(m, 3))
        h = B.Handle(sc)
        h.write(B.BUF_X, x)
        h.write(B.BUF_UC, uc)
        count = h.detect()
        h.contact_step()
        out.append((count, h.read(B.BUF_P)[:m].copy(), h.contacts()["pairs"]))
        h.close()
    assert lo <= out[0][0] <= hi and out[0][0] == out[1][0]
    assert np.array_equal(out[0][2], out[1][2])
    assert np.array_equal(out[0][1], out[1][1])


def test_contact_passes_follow_the_count():
    """Substeps from the same reset state, whichever way the last one's contacts made them run."""
    sc, many, m = _stack(3, 8)
    few = many.copy()
    for k in range(3):
        few[k * m // 3:(k + 1) * m // 3, 1] += 0.1 * k
    few[0] = few[m // 3:m // 3 + 11].mean(0) - np.array([0.0, 1e-3, 0.0])  # just under the second sheet
    v = np.zeros_like(many)

    def run(h, x):
        h.reset()
        h.set_state(x, v)
        st = h.step(1)
        return st["n_contacts"], h.get_state()[0]

    fresh = []
    for x in (many, few):
        h = B.Handle(sc)
        fresh.append(run(h, x))
        h.close()
    assert fresh[0][0] > 768 > fresh[1][0]
    h = B.Handle(sc)
    for k in (0, 0, 1, 1, 0, 1):
        n, x = run(h, (many, few)[k])
        assert n == fresh[k][0] and np.array_equal(x, fresh[k][1])
    h.close()


def test_contact_passes_follow_the_count_within_a_call():
    """Twelve sheets that fall onto each other: contacts grow out of the one block in a call of many
    substeps.  The launches take over in the call itself, and whichever way the substeps are queued
    and run, the bits are those of one call per substep."""
    n = 20
    sc, x, m = _stack(12, 6)
    v = np.zeros_like(x)
    for k in range(12):
        x[k * m // 12:(k + 1) * m // 12, 1] += 8e-3 * k
        v[k * m // 12:(k + 1) * m // 12, 1] = -0.1 * k

    def run(step):
        h = B.Handle(sc)
        h.set_state(x, v)
        assert h.step(1)["n_contacts"] == 0
        few = h.kernels_per_step()
        counts = step(h)
        out = h.get_state(), counts, h.kernels_per_step() > few
        h.close()
        return out

    ref, counts, _ = run(lambda h: [h.step(1)["n_contacts"] for _ in range(n)])
    assert max(counts) > 768
    state, _, launches = run(lambda h: h.step(n))
    assert launches and all(np.array_equal(p, q) for p, q in zip(state, ref))

    def queued(h):
        h.step_async(n // 2)
        for _ in range(n // 2):
            h.step_async()
        h.sync()

    state, _, _ = run(queued)
    assert all(np.array_equal(p, q) for p, q in zip(state, ref))
