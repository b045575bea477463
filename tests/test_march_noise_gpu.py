"""SOAR model error in the batched engine, tile shape by tile shape: the tile
kernels add it to the state that a step writes, the marching shape (56, 8) in
launches of its own, and every state and drifter has to come out in the same
bits."""
import numpy as np
import pytest

from test_ensemble_gpu import _member, _with_noise

pytestmark = pytest.mark.gpu

# grids whose steps differ in length, so that blocks hold different numbers of them
SPECS = [(63, 42, (1, 2, 1, 2), 3), (84, 21, (1, 1, 1, 1), 4), (42, 63, (2, 2, 2, 2), 5), (126, 42, (2, 1, 2, 1), 6)]
COURANT = [0.8, 0.3, 0.55, 0.8]


def _engine(ctx, shape, factor, rng_seed, drifters=20, use_graph=True):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    sims = [_member(ctx, *s, drifters=drifters) for s in SPECS]
    _with_noise(sims, factor, 1)
    for s, c in zip(sims, COURANT):
        s.updateDt(courant_number=c)
    ens = BatchedEnsemble(sims, use_graph=use_graph, autotune=False)
    ens.set_tile_shape(ens.tile_shapes().index(shape))
    ens.set_noise([s.model_error for s in sims], rng_seed=rng_seed)
    return ens, sims


def _results(ens, sims):
    ens.synchronize()
    out = [np.asarray(np.ma.getdata(x))[2:-2, 2:-2] for s in sims for x in s.download()]
    if ens.has_drifters:
        out.append(ens.download_drifters())
    return out


def _same(a, b):
    return len(a) == len(b) and all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("factor", [1, 3, 7])
@pytest.mark.parametrize("rng_seed", [None, 5])
@pytest.mark.parametrize("cadence", ["block", "step"])
def test_noise_is_the_same_on_every_shape(gpu_ctx, factor, rng_seed, cadence):
    """Both cadences, injected and drawn normals, members without model error,
    blocks of unequal length, an idle member, drifters, factors on both sides
    of the row transfer's."""
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    first = None
    for shape in BatchedEnsemble.tile_shapes():
        ens, sims = _engine(gpu_ctx, shape, factor, rng_seed)
        assert ens._marches() == (shape == (56, 8))
        ens.step(300.0, True, noise_cadence=cadence)
        ens.step(300.0, [True, False, True, True], noise_cadence=cadence)
        ens.step(200.0, True, noise_cadence=cadence, members=[0, 2, 3])
        ens.step(300.0, False)
        ens.step(300.0, True, noise_cadence=cadence)
        assert len({s.num_iterations for s in sims}) > 1
        got = _results(ens, sims)
        ens.release()
        if first is None:
            first = got
        assert _same(got, first), shape


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("shape", [(32, 16), (56, 8)])
def test_blocks_without_steps_draw_nothing(gpu_ctx, shape, use_graph):
    """A block in which no member takes a step leaves states and generators
    where they were, with the same draws in the blocks that follow."""
    out = []
    for empty in (False, True):
        ens, sims = _engine(gpu_ctx, shape, 3, 5, drifters=0, use_graph=use_graph)
        ens.step(300.0, True)
        if empty:
            ens.step(0.0, True)
            ens.step(300.0, True, members=[])
        ens.step(300.0, True)
        out.append(_results(ens, sims))
        ens.release()
    assert _same(*out)


def test_unperturbed_copies_where_a_step_needs_them(gpu_ctx):
    """A marching engine allocates none of the copies that fused model error
    reads; one that is given a tile shape later does, before its next block."""
    import torch
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    out = []
    for late in (False, True):
        sims = [_member(gpu_ctx, 504, 301, (1, 2, 1, 2), 3 + m, drifters=20) for m in range(12)]
        _with_noise(sims, 7, 1)
        for s in sims:
            s.updateDt()
        ens = BatchedEnsemble(sims, autotune=False)
        ens.set_tile_shape(ens.tile_shapes().index((56, 8) if late else (32, 16)))
        free = torch.cuda.mem_get_info()[0]
        ens.set_noise([s.model_error for s in sims], rng_seed=5)
        used = free - torch.cuda.mem_get_info()[0]
        copies = 12 * 3 * 4 * 508 * 305
        assert used < copies if late else used >= copies
        ens.step(120.0, True)
        ens.set_tile_shape(0)
        ens.step(120.0, True)
        out.append(_results(ens, sims))
        ens.release()
    assert _same(*out)
