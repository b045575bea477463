"""Checkpointed rollouts on both sides of the limits at which the forward step
changes its tiles: the recomputed segments step in the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from test_march_gpu import CHANNEL, WALLS, _sim  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,bc,options", [(33, 40, WALLS, {}), (128, 128, WALLS, dict(r=1e-3)), (200, 61, CHANNEL, {}),
                                              (224, 224, CHANNEL, dict(beta=2e-11)), (321, 300, WALLS, {})])
def test_checkpointed_equals_stored(gpu_ctx, nx, ny, bc, options):
    from gpuocean_gb300.adjoint import CDKLM16Rollout, StepAdjoint
    sim = _sim(gpu_ctx, nx, ny, bc, 3, **options)
    grads = []
    for frac in (0.5, 0.0):
        adj = StepAdjoint(sim, memory_fraction=frac)
        x = [a.clone().requires_grad_(True) for a in adj.state(*[np.ma.getdata(a) for a in sim.download()])]
        w = torch.tensor([1.0e-4, -3.0e-5], device=adj.device, requires_grad=True)
        out = CDKLM16Rollout.apply(adj, 11, 2, *x, w)
        (out[:, 0] ** 2 + out[:, 1] * out[:, 2]).sum().backward()
        grads.append([out.detach()] + [a.grad.clone() for a in x] + [w.grad.clone()])
    assert all(torch.isfinite(g).all() for g in grads[0])
    for a, b in zip(*grads):
        assert torch.equal(a, b)
    sim.cleanUp()
