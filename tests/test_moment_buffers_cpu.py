"""The pool of moments() buffers without a GPU."""
import threading


class _Buffer:
    def __init__(self, nbytes):
        self.nbytes, self.freed = nbytes, False

    def free(self):
        assert not self.freed
        self.freed = True


def test_an_engine_released_inside_a_call(monkeypatch):
    """The garbage collector may release an engine on the thread that is in
    the pool: that call may not wait for itself."""
    from gpuocean_gb300.ensembles import BatchedEnsemble as B
    monkeypatch.setattr(B.Common, "DevicePtr", _Buffer)
    pool = B._MomentBuffers()
    pool.open()
    pool.open()
    bufs = [pool.take(8), pool.take(8)]
    for b in bufs:
        pool.put(b)

    def collect():
        with pool._lock:
            pool.close()

    t = threading.Thread(target=collect, daemon=True)
    t.start()
    t.join(10.0)
    assert not t.is_alive()
    assert not any(b.freed for b in bufs)
    assert pool.take(8) in bufs and not pool.take(16).freed
    pool.put(bufs[0])
    pool.close()
    assert bufs[0].freed
