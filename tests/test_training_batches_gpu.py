"""Training losses whose samples go through the device in several batches: by the limit on a batch's
memory (uneven batches, one sample each) and because the device has no room for all of them."""
import numpy as np
import pytest

from parallel_admm_b200 import gnn

pytestmark = pytest.mark.gpu


def _problem(n, samples, K, seed=0):
    rng = np.random.default_rng(seed)
    side = 3
    rows = np.arange(n)[:, None]
    col = rows + np.concatenate([np.arange(-side, 0), np.arange(1, side + 1)])[None, :]
    keep = (col >= 0) & (col < n)
    start = np.concatenate([[0], np.cumsum(keep.sum(1))])
    diag = rng.uniform(8.0, 10.0, size=n)
    sysm = gnn.System(start, col[keep], np.full(keep.sum(), -1.0), diag)
    f = np.float32
    coef = (rng.uniform(0.7, 1.0, K).astype(f), np.where(np.arange(K) > 0, 0.1, 0.0).astype(f),
            (rng.uniform(0.9, 1.1, n) / diag).astype(f), rng.uniform(-0.3, 0.3, n).astype(f))
    xs = rng.normal(size=(samples, n, 3)).astype(f)
    b = np.stack([sysm.matvec(x.astype(np.float64)) for x in xs]).astype(f)
    xc = xs + rng.normal(scale=0.1, size=xs.shape).astype(f)
    xl = xc + rng.normal(scale=0.1, size=xs.shape).astype(f)
    return sysm, coef + (b, xc, xl, xs)


def _same(got, ref):
    """Loss, m and theta gradients are summed sample by sample on either path; the coefficients'
    FP64 sums are associated differently, then rounded to FP32 (one unit in the last place)."""
    assert got[0] == ref[0]
    for k in (1, 2):
        assert np.allclose(got[k], ref[k], rtol=2.0 ** -23, atol=0.0)
    for k in (3, 4):
        assert np.array_equal(got[k], ref[k])


@pytest.mark.parametrize("mu", [0.0, 0.5])
@pytest.mark.parametrize("batch", [1, 3, 4])
def test_batches_of_a_loss(batch, mu):
    n, samples, K = 1500, 7, 5
    sysm, args = _problem(n, samples, K)
    one = gnn.SweepTrainer(sysm, residual_weight=mu)
    ref = one.loss_grad(*args)
    per = 4 * ((2 * K + 9) * 3 * n + n)
    tr = gnn.SweepTrainer(sysm, residual_weight=mu, batch_bytes=batch * per if batch > 1 else 0)
    _same(tr.loss_grad(*args), ref)
    for t in (one, tr):
        t.close()


def test_loss_on_a_full_device():
    import torch
    n, samples, K = 200_000, 40, 6
    sysm, args = _problem(n, samples, K)
    tr = gnn.SweepTrainer(sysm)
    ref = gnn.SweepTrainer(sysm, batch_bytes=1 << 29)
    want = ref.loss_grad(*args)
    ref.close()
    need = 4 * samples * ((2 * K + 9) * 3 * n + n)
    free = torch.cuda.mem_get_info()[0]
    held = torch.empty(free - int(0.7 * need), dtype=torch.uint8, device="cuda:0")
    got = tr.loss_grad(*args)
    del held
    torch.cuda.empty_cache()
    tr.close()
    _same(got, want)
