"""Ensemble moments at the limits of values and sizes."""
import numpy as np
import pytest

from test_ensemble_stats_gpu import _close, _stepped
from test_march_gpu import WALLS, _sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5, 20, 130])
@pytest.mark.parametrize("quantity", ["state", "velocity"])
def test_members_that_are_not_finite(gpu_ctx, n, quantity):
    """One infinite member value gives an infinite mean and one NaN a NaN, in
    their cell alone; squares that overflow in a sum that does not give an
    infinite variance.  Members early and late in the sum."""
    ens, sims = _stepped(gpu_ctx, n, 21, 10, steps=1)
    spots = {(4, 5): [(1, np.inf)], (5, 9): [(n - 1, -np.inf)], (7, 3): [(3, np.nan)], (8, 18): [(1, 2e22), (2, -2e22)],
             (9, 12): [(1, np.inf), (3, np.inf)]}
    before = ens.moments(quantity=quantity)
    for (j, i), values in spots.items():
        for m, v in values:
            eta, hu, hv = (np.array(np.ma.getdata(a)) for a in sims[m].download())
            hu[j, i] = v
            sims[m].upload(eta, hu, hv)
    q = 1 if quantity == "state" else 0         # the plane of hu or u
    mean, var = ens.moments(quantity=quantity)
    at = lambda a, j, i: a[q, j - 2, i - 2]     # noqa: E731
    assert at(mean, 4, 5) == np.inf and at(mean, 5, 9) == -np.inf and at(mean, 9, 12) == np.inf
    assert np.isnan(at(mean, 7, 3)) and np.isnan(at(var, 7, 3)) and np.isnan(at(var, 4, 5))
    assert at(var, 8, 18) == np.inf and np.isfinite(at(mean, 8, 18))
    for a, b in zip((mean, var), before):
        a, b = a.copy(), b.copy()
        for j, i in spots:
            a[q, j - 2, i - 2] = b[q, j - 2, i - 2] = 0.0
        assert np.array_equal(a, b)
    ens.release()


def test_moments_of_a_tall_grid(gpu_ctx):
    """More rows than a launch has blocks in y when a block takes four."""
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    nx, ny = 3, 262149
    sims = [_sim(gpu_ctx, nx, ny, WALLS, m) for m in range(3)]
    ens = BatchedEnsemble(sims, autotune=False)
    mean, var = ens.moments()
    x = np.stack([np.stack([np.asarray(np.ma.getdata(a))[2:-2, 2:-2] for a in s.download()]) for s in sims])
    x = x.astype(np.float64)
    for q in range(3):      # the bars of the other moments tests
        assert _close(mean[q], x[:, q].mean(axis=0), 2e-6) and _close(var[q], x[:, q].var(axis=0), 1e-5)
    ens.release()
