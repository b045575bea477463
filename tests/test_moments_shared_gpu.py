"""Moments of small ensembles, whose members are summed in slices, from several
engines, streams and threads at once: each call's sums are its own."""
import ctypes
import threading

import numpy as np
import pytest

from test_march_gpu import WALLS, _sim

pytestmark = pytest.mark.gpu


def _engine(ctx, seed, n=64, nx=40, ny=30):
    from gpuocean_gb300.ensembles.BatchedEnsemble import BatchedEnsemble
    return BatchedEnsemble([_sim(ctx, nx, ny, WALLS, seed + m) for m in range(n)], autotune=False)


def test_engines_on_their_streams(gpu_ctx):
    """Calls of three engines queued in turn, with nothing waited for."""
    engines = [_engine(gpu_ctx, 100 * i) for i in range(3)]
    want = [e.moments() for e in engines]
    held = [(e, w, e.moments(download=False)) for _ in range(20) for e, w in zip(engines, want)]
    for e, w, (mean, var) in held:
        for buf, x in ((mean, w[0]), (var, w[1])):
            assert np.array_equal(e._download(buf, x.shape), x)
            buf.free()
    for e in engines:
        e.release()


def test_one_engine_on_two_streams_and_threads(gpu_ctx):
    """Groups of the members, by two threads, each on a stream of its own."""
    from gpuocean_gb300 import _lib
    from gpuocean_gb300.utils import Common
    e = _engine(gpu_ctx, 7, n=80)
    groups = [(0, 48), (32, 48)]
    want = [e.moments(first=f, count=n) for f, n in groups]
    e.synchronize()
    wrong = []

    def work(i):
        stream, (f, n), x = Common.Stream(), groups[i], want[i]
        bufs = [Common.DevicePtr(x[0].nbytes) for _ in range(2)]
        for _ in range(50):
            _lib.call("goc_ensemble_moments", e._handle, f, n, 0, ctypes.c_float(0.0), 0, bufs[0].ptr, bufs[1].ptr,
                      stream.handle)
            for b, y in zip(bufs, x):
                got = np.empty_like(y)
                _lib.call("goc_memcpy_d2h_async", got.ctypes.data, b.ptr, ctypes.c_size_t(got.nbytes), stream.handle)
                stream.synchronize()
                if not np.array_equal(got, y):
                    wrong.append(i)
        for b in bufs:
            b.free()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    e.release()
