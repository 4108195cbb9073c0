"""A gradient whose arrays do not fit the device's memory: every call that needs
them reports TTI_ERR_NOMEM, the second as the first, and leaves nothing behind;
with memory free again the same handle and the same batch run."""
import ctypes as C

import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
NZ, NX, NT, EAL = 1200, 1200, 24, 10
CFG = dict(variant="coordinate_rotation", nz=NZ, nx=NX, nt=NT, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=EAL,
           freesurface=1, stype=1, seistype=1)


class _Full:
    """Holds all device memory but less than 64 MB: some of the gradient's 24 arrays
    of 6 MB still fit, not all of them."""

    def __enter__(self):
        self.rt = C.CDLL("libcudart.so.12")
        self.held, block = [], 8 << 30
        while block >= 64 << 20:
            p = C.c_void_p()
            if self.rt.cudaMalloc(C.byref(p), C.c_size_t(block)) == 0:
                self.held.append(p)
            else:
                self.rt.cudaGetLastError()
                block //= 2

    def __exit__(self, *exc):
        for p in self.held:
            assert self.rt.cudaFree(p) == 0


def _shot(h, sx):
    h.set_source([sx], [2], synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)[None, :])
    for k in (0, 1):
        h.set_receivers(k, np.arange(NX), 4)


def _gradient(h):
    for k in (0, 1):
        h.grad_set_observed(k, np.zeros((NX, NT), np.float32))
    h.grad_zero()
    j = h.grad_run(3)
    return j, [h.grad_fetch(n) for n in ("vp", "eps", "delta", "theta")]


def _nomem(f, *args):
    import ttifd

    with pytest.raises(ttifd.TTIError) as e:
        f(*args)
    assert e.value.code == ttifd.ERR_NOMEM


def test_single_shot(gpu_lib):
    import ttifd

    m = synthetic.padded(synthetic.layered_model(NZ, NX, seed=3), EAL)
    with ttifd.Modeling(**CFG) as h, ttifd.Modeling(**CFG) as r:
        for q in (h, r):
            q.upload_model(*m)
            _shot(q, 50)
        with _Full():
            for _ in range(2):
                _nomem(h.grad_zero)
            for _ in range(2):
                _nomem(h.grad_set_observed, 0, np.zeros((NX, NT), np.float32))
            with pytest.raises(ttifd.TTIError) as e:  # nothing is there to fetch from
                h.grad_fetch("vp")
            assert e.value.code == ttifd.ERR_STATE
        got, ref = _gradient(h), _gradient(r)
    assert got[0] == pytest.approx(ref[0], rel=1e-12) and ref[0] > 0  # (added up by atomics, in double)
    for a, b in zip(got[1], ref[1]):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)) and np.any(b != 0)


def test_batch(gpu_lib):
    import ttifd

    m = synthetic.padded(synthetic.layered_model(NZ, NX, seed=3), EAL)
    with ttifd.Batch([CFG], [0, 0]) as b:
        b.upload_model(0, *m)
        for i, h in enumerate(b.instances):  # no receivers: no observed traces come first
            h.set_source([40 + i], [2], synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)[None, :])
        with _Full():
            for _ in range(2):
                _nomem(b.grad_run, 2, 4)
        assert b.grad_run(2, 4) == [0.0, 0.0]
        for i, h in enumerate(b.instances):
            _shot(h, 40 + i)
            for k in (0, 1):
                h.grad_set_observed(k, np.zeros((NX, NT), np.float32))
        j = b.grad_run(2, 4)
        assert min(j) > 0 and all(np.isfinite(b.instances[0].grad_fetch(n)).all() for n in ("vp", "theta"))
