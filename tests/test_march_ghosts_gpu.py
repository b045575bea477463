"""The marching kernel's periodic ghost images in domains with walls in the
other direction, against the tile kernel's: drifters, and a tile kernel that
takes over, read them."""
import numpy as np
import pytest

from test_march_gpu import CASES, CHANNEL, TURNED, _march, _sim

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,bc,options", [c for c in CASES if c[2] in (CHANNEL, TURNED)])
def test_march_images_equal_tiles(gpu_ctx, nx, ny, bc, options):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    out = []
    for march in (False, True):
        sims = [_sim(gpu_ctx, nx, ny, bc, 10 + m, **options) for m in range(2)]
        ens = BatchedEnsemble(sims, autotune=False)
        if march:
            _march(ens)
        ens.step(3 * float(np.float32(1.3)))
        ens.synchronize()
        # interior rows with the images of columns, or the other way round
        cut = (slice(2, -2), slice(None)) if bc == CHANNEL else (slice(None), slice(2, -2))
        out.append([np.asarray(np.ma.getdata(x))[cut] for s in sims for x in s.download()])
        ens.release()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    for a in out[1]:
        a = a if bc == CHANNEL else a.T
        assert np.array_equal(a[:, :2], a[:, -4:-2]) and np.array_equal(a[:, -2:], a[:, 2:4])
