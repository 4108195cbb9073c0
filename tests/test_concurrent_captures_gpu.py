"""Graphs of steps captured in several host threads at the same time, while the
others allocate and free device memory: the same results, bit for bit, as with
every step launched by itself."""
import threading

import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
NZ, NX, NT, EAL = 40, 60, 230, 5


def _cfg(stype):
    return dict(variant="coordinate_rotation", nz=NZ, nx=NX, nt=NT, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0,
                ealThick=EAL, freesurface=1, stype=stype, seistype=1)


def _model():
    return synthetic.padded(synthetic.layered_model(NZ, NX, seed=3), EAL)


def _shot(h, i):
    h.set_source([4 + 5 * i], [2], synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)[None, :])
    for k in (0, 1):
        h.set_receivers(k, np.arange(NX), 4)


# (stype 2 allocates its source tables at the start of each gradient run)
@pytest.mark.parametrize("stype", [1, 2])
def test_batch_gradient(stype, monkeypatch, gpu_lib):
    import ttifd

    out = []
    for steps in (None, "0"):
        if steps is not None:
            monkeypatch.setenv("TTIFD_GRAPH_STEPS", steps)
        with ttifd.Batch([_cfg(stype)], [0] * 10) as b:
            b.upload_model(0, *_model())
            for i, h in enumerate(b.instances):
                _shot(h, i)
                for k in (0, 1):
                    h.grad_set_observed(k, np.zeros((NX, NT), np.float32))
            res = []
            for _ in range(2):
                j = b.grad_run(2, 35)
                res.append(([h.fetch_traces(0) for h in b.instances],
                            [b.instances[0].grad_fetch(n) for n in ("vp", "eps", "delta", "theta")]))
            assert min(j) > 0
            out.append(res)
    for got, ref in zip(*out):
        for a, r in zip(got[0] + got[1], ref[0] + ref[1]):
            assert np.array_equal(a.view(np.uint32), r.view(np.uint32)) and np.any(r != 0)


def test_handles_in_threads(monkeypatch, gpu_lib):
    import ttifd

    m, got = _model(), {}

    def work(i):
        for n in range(4):  # a new handle, and with it new captures, each time
            with ttifd.Modeling(**_cfg(1)) as h:
                h.upload_model(*m)
                _shot(h, i)
                h.run()
                got[i, n] = h.fetch_traces(0), h.fetch_field(0)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(got) == 24
    monkeypatch.setenv("TTIFD_GRAPH_STEPS", "0")
    for i in range(6):
        with ttifd.Modeling(**_cfg(1)) as h:
            h.upload_model(*m)
            _shot(h, i)
            h.run()
            ref = h.fetch_traces(0), h.fetch_field(0)
        for n in range(4):
            for a, r in zip(got[i, n], ref):
                assert np.array_equal(a.view(np.uint32), r.view(np.uint32)) and np.any(r != 0)
