"""Benchmark members through the engine with the tile shape set, not timed:
the fused tile launches, whose interior tiles stage their input by TMA, and the
marching kernel with its model error in launches of its own."""
import numpy as np
import pytest

from test_headline_parity_gpu import _assert_identical, _member, _run_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(32, 16), (56, 8)])
def test_members_equal_on_a_set_shape(gpu_ctx, shape):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    from gpuocean_gb300.utils.BenchmarkCases import double_jet_case
    case = double_jet_case()
    a = [_member(gpu_ctx, case, m, 200) for m in range(4)]
    b = [_member(gpu_ctx, case, m, 200) for m in range(4)]
    ens = BatchedEnsemble(a, autotune=False)
    ens.set_tile_shape(ens.tile_shapes().index(shape))
    ens.set_noise([s.model_error for s in a])
    before = ens.tma_status()[1]
    _run_pairs(ens, a, b, blocks=4)
    _assert_identical(a, b)
    staged, tiles, errors = ens.tma_status()
    assert staged == 4 and errors == 0
    assert (tiles > before) == (shape != (56, 8))       # staged by the blocks' own launches
    ens.release()
    assert np.isfinite(a[0].download()[0]).all()
