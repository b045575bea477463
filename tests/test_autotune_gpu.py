"""The autotuner's choice belongs to the kind of ensemble that it was timed on."""
import numpy as np
import pytest

from test_march_gpu import CHANNEL, WALLS, _sim

pytestmark = pytest.mark.gpu


def _textured(ctx, nx, ny):
    from gpuocean_gb300.SWEsimulators.CDKLM16 import CDKLM16
    from gpuocean_gb300.utils import Common, WindStress
    z = np.zeros((ny + 4, nx + 4), dtype=np.float32)
    wind = [np.full((3, 4), 1e-4, dtype=np.float32)]
    return CDKLM16(ctx, z, z.copy(), z.copy(), np.full((ny + 5, nx + 5), 60.0, dtype=np.float32), nx, ny, 500.0, 700.0,
                   1.3, 9.81, 1.2e-4, 0.0, boundary_conditions=Common.BoundaryConditions(*WALLS),
                   wind=WindStress.WindStress(t=[0.0], stress_u=wind, stress_v=wind))


def test_a_choice_is_not_passed_on_to_other_kinds(gpu_ctx, monkeypatch):
    """Ensembles of one grid size: each kind is timed for itself, a second one
    of a kind is not, and the marching shape is timed only where it can run."""
    from gpuocean_gb300.ensembles import BatchedEnsemble as B
    monkeypatch.setattr(B, "_AUTOTUNE_CACHE", {})
    nx, ny = 64, 40
    kinds = {"open": lambda m: _sim(gpu_ctx, nx, ny, WALLS, m), "land": lambda m: _sim(gpu_ctx, nx, ny, WALLS, m, land=True),
             "turned": lambda m: _sim(gpu_ctx, nx, ny, WALLS, m, angle=0.4),
             "one_dimensional": lambda m: _sim(gpu_ctx, nx, ny, WALLS, m, one_dimensional=True),
             "channel": lambda m: _sim(gpu_ctx, nx, ny, CHANNEL, m), "textured": lambda m: _textured(gpu_ctx, nx, ny)}
    for name, make in kinds.items():
        for again in (False, True):
            ens = B.BatchedEnsemble([make(m) for m in range(2)])
            assert hasattr(ens, "autotune_timings") != again, name
            if name == "textured":
                assert ens.tile_shape != (56, 8)
                if not again:
                    assert len(ens.autotune_timings) == len(ens.tile_shapes()) - 1
            elif not again:
                assert set(ens.autotune_timings) == set(ens.tile_shapes())
            ens.step(2.6)
            ens.synchronize()
            ens.release()
