"""The device buffers that moments() keeps between calls."""
import threading

import numpy as np
import pytest

from test_march_gpu import WALLS, _sim

pytestmark = pytest.mark.gpu


def _engine(ctx, n=3, nx=40, ny=30, seed=0):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    return BatchedEnsemble([_sim(ctx, nx, ny, WALLS, seed + m) for m in range(n)], autotune=False)


class _Count:
    """Allocations and frees of device buffers by the engine's module."""

    def __init__(self, monkeypatch):
        from gpuocean_gb300.ensembles import BatchedEnsemble as B
        base, self.live, self.made = B.Common.DevicePtr, 0, 0
        counts = self

        class Counted(base):
            def __init__(self, nbytes):
                super().__init__(nbytes)
                counts.live += 1
                counts.made += 1

            def free(self):
                counts.live -= bool(self.ptr)
                super().free()

        monkeypatch.setattr(B.Common, "DevicePtr", Counted)


def test_a_first_call_takes_what_other_engines_put_back(gpu_ctx, monkeypatch):
    """Nothing is allocated by the first call of an engine, or of one whose
    tables were built again, when an earlier call left buffers that are large
    enough; smaller ones are replaced; the last engine frees them."""
    import gc
    gc.collect()
    first = _engine(gpu_ctx)
    want = first.moments()
    second, large = _engine(gpu_ctx, seed=5), _engine(gpu_ctx, nx=80)
    n = _Count(monkeypatch)
    second.moments()
    assert n.made == 0
    assert all(np.array_equal(a, b) for a, b in zip(first.moments(), want)) and n.made == 0
    first._build()
    made = n.made       # what the tables take
    assert all(np.array_equal(a, b) for a, b in zip(first.moments(), want)) and n.made == made
    large.moments()
    assert n.made == made + 2
    first.moments(quantity="velocity")
    assert n.made == made + 2
    # a buffer that is handed out is the caller's
    mean, var = first.moments(download=False)
    first.moments()
    assert n.made == made + 4
    mean.free()
    var.free()
    for e in (first, second, large):
        e.release()
        e.release()
    from gpuocean_gb300.ensembles.BatchedEnsemble import _MOMENT_BUFFERS
    if not _MOMENT_BUFFERS._engines:    # engines of other tests may live on
        assert not _MOMENT_BUFFERS._free


def test_threads_share_the_buffers(gpu_ctx):
    """Engines of three threads, more calls at once than buffers are kept."""
    engines = [_engine(gpu_ctx, n=4, seed=10 * t) for t in range(3)]
    want = [e.moments() for e in engines]
    wrong = []

    def work(t):
        for _ in range(50):
            if not all(np.array_equal(a, b) for a, b in zip(engines[t].moments(), want[t])):
                wrong.append(t)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for e in engines:
        e.release()
