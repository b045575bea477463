"""The marching kernel against the tile kernel, bit for bit, on states that
are not finite everywhere: a member that has blown up steps (and shows that it
has) the same way whichever kernel the autotuner picks.  A NaN or infinite
momentum in deep water reaches the rows and columns around it through the
limiters, the fluxes of "still" faces and the sources; a NaN in eta is taken
out by the scheme's final clamp."""
import numpy as np
import pytest

from test_march_gpu import CHANNEL, TORUS, WALLS, _march, _sim, _states

pytestmark = pytest.mark.gpu

SPOTS = {
    "nan_momentum": [(1, 9, 20, np.nan)],
    "infinite_momentum": [(2, 12, 7, np.inf), (1, 20, 40, -np.inf)],
    "nan_eta": [(0, 10, 30, np.nan)],
    # the value of eta that marks a dry cell, in wet ones
    "dry_flag": [(0, 15, 30, 1e-30), (0, 16, 31, 1e-30), (0, 25, 4, 1e-30)],
    "huge": [(1, 14, 33, 1e25), (2, 5, 11, -1e30)],
    # rows at which a run of the queue starts, its pipeline rows, the domain's edges
    "many": [(q, j, i, v) for j in (2, 3, 7, 9, 10, 11, 17, 25) for q, i, v in
             ((1, 2 + j, np.nan), (2, 50 - j, np.inf), (0, 25 + j, np.nan))],
}


@pytest.mark.parametrize("spots", sorted(SPOTS))
@pytest.mark.parametrize("bc,options", [(WALLS, {}), (CHANNEL, dict(beta=2e-11)), (TORUS, {}), (WALLS, dict(angle=0.4)),
                                        (WALLS, dict(r=2.4e-3, land=True))])
def test_march_equals_tiles_on_values_that_are_not_finite(gpu_ctx, spots, bc, options):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    out = []
    for march in (False, True):
        sims = [_sim(gpu_ctx, 61, 27, bc, 10 + m, **options) for m in range(2)]
        s = sims[1]
        state = [np.array(np.ma.getdata(a)) for a in s.download()]
        for q, j, i, v in SPOTS[spots]:
            state[q][j, i] = v
        s.upload(*state)
        ens = BatchedEnsemble(sims, autotune=False)
        if march:
            _march(ens)
        ens.step(3 * float(np.float32(1.3)))
        ens.synchronize()
        out.append(_states(sims, False))
        ens.release()
    assert np.isfinite(np.concatenate([x.ravel() for x in out[0][0]])).all()
    for a, b in zip(*out):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)
