"""Steps of small and large grids: the tile shapes and thread counts that grids
with few or many tiles take give the bits of the engine's tiles (32 x 16 cells,
256 threads).  The sizes sit on both sides of the limits (38 and 152 tiles, 912
tiles of 32 x 32) and at ragged edges of the 16 x 8 and 32 x 32 tiles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,bc,beta,r", [
    (1, 1, (1, 1, 1, 1), 0.0, 0.0), (5, 4, (2, 2, 2, 2), 0.0, 0.0), (16, 8, (1, 2, 1, 2), 2e-11, 0.0),
    (17, 9, (1, 1, 1, 1), 0.0, 1e-3), (64, 64, (1, 1, 1, 1), 2e-11, 0.0), (608, 32, (1, 2, 1, 2), 0.0, 0.0),
    (609, 32, (1, 2, 1, 2), 2e-11, 0.0), (255, 257, (2, 1, 2, 1), 0.0, 1e-3), (2432, 32, (1, 2, 1, 2), 2e-11, 0.0),
    (2433, 32, (1, 1, 1, 1), 0.0, 0.0), (1216, 768, (1, 1, 1, 1), 2e-11, 1e-3), (1185, 737, (2, 2, 2, 2), 0.0, 0.0),
    (1184, 768, (1, 2, 1, 2), 2e-11, 0.0), (33, 29153, (1, 1, 1, 1), 0.0, 0.0)])
def test_small_grids_step_like_tiles(gpu_ctx, nx, ny, bc, beta, r):
    from gpuocean_gb300.SWEsimulators.CDKLM16 import CDKLM16
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    from gpuocean_gb300.utils import Common
    rng = np.random.default_rng(nx + 7 * ny)
    shape = (ny + 4, nx + 4)
    H = (60.0 + 5.0 * rng.standard_normal((ny + 5, nx + 5))).astype(np.float32)
    q = [(a * rng.standard_normal(shape)).astype(np.float32) for a in (0.3, 8.0, 8.0)]
    sims = [CDKLM16(gpu_ctx, *q, H, nx, ny, 500.0, 700.0, 1.3, 9.81, 1.2e-4, r, coriolis_beta=beta,
                    boundary_conditions=Common.BoundaryConditions(*bc)) for _ in range(2)]
    ens = BatchedEnsemble(sims[:1], autotune=False)
    t = 3 * float(np.float32(1.3))
    ens.step(t)
    ens.synchronize()
    sims[1].step(t)
    for a, b in zip(sims[0].download(), sims[1].download()):
        a, b = np.asarray(a)[2:-2, 2:-2], np.asarray(b)[2:-2, 2:-2]
        assert np.isfinite(a).all() and np.array_equal(a, b)
    ens.release()
