"""Members with one Coriolis value and a per-cell table beside it: the value
counts, on every tile shape."""
import numpy as np
import pytest

from test_march_gpu import WALLS, _sim, _states

pytestmark = pytest.mark.gpu


def test_one_value_counts_before_a_table(gpu_ctx):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    from gpuocean_gb300.utils import Common
    nx, ny, out = 61, 27, []
    for table, shape in ((False, 0), (True, 0), (True, -1)):
        sims = [_sim(gpu_ctx, nx, ny, WALLS, 10 + m) for m in range(2)]
        if table:
            for s in sims:
                s.coriolis_cell = Common.CUDAArray2D(s.gpu_stream, nx, ny, 2, 2, np.full((ny + 4, nx + 4), 3e-3, np.float32))
        ens = BatchedEnsemble(sims, autotune=False)
        ens.set_tile_shape(shape % len(ens.tile_shapes()))
        ens.step(3 * float(np.float32(1.3)))
        ens.synchronize()
        out.append(_states(sims, False))
        ens.release()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            for x, y in zip(a, b):
                assert np.array_equal(x, y)
