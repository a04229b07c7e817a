"""The converged solve over the row shapes that its kernels treat differently: rows without, with
few and with more entries than are loaded ahead, and more rows than threads."""
import numpy as np
import pytest

from parallel_admm_b200 import gnn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [0, 3, 20])
@pytest.mark.parametrize("n", [1, 127, 129, 80_000])
def test_solve_row_shapes(n, side):
    """A banded, diagonally dominant system.  The iteration ends at a residual of 1e-6 in the norm
    of diag(A)^-1, whose entries lie within a factor of 2: 2e-6 of |b| in the 2-norm, and FP32
    rounding of x and of the recursive residual adds a few 1e-7 x cond(A) (at most 4): 1e-5."""
    rng = np.random.default_rng(n + side)
    rows = np.arange(n)
    off = np.concatenate([np.arange(-side, 0), np.arange(1, side + 1)])
    col = rows[:, None] + off[None, :]
    keep = (col >= 0) & (col < n)
    lo, hi = np.minimum(rows[:, None], col), np.maximum(rows[:, None], col)
    val = -(0.5 + ((lo * 7 + hi * 13) % 11) / 22.0)  # symmetric
    w = np.where(keep, val, 0.0)
    diag = (1.0 + rng.uniform(size=n)) * 1.7 * max(2 * side, 1)
    start = np.concatenate([[0], np.cumsum(keep.sum(1))])
    sysm = gnn.System(start, col[keep], val[keep], diag)
    b = rng.normal(size=(n, 3)).astype(np.float32)
    tr = gnn.SweepTrainer(sysm)
    x, it = tr.solve(b, np.zeros_like(b))
    tr.close()
    r = b - sysm.matvec(x.astype(np.float64))
    assert it > 0 and np.linalg.norm(r) <= 1e-5 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [16_384, 16_385, 303_105])
def test_solve_row_counts(n):
    """The largest system whose iteration takes two launches, the smallest with three, and one more
    row than the kernels have threads."""
    test_solve_row_shapes(n, 3)
