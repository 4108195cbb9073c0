"""Observed traces and receivers that are set again between gradient runs."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
NZ, NX, NT = 40, 60, 60


def _handle(seistype=1):
    import ttifd

    h = ttifd.Modeling(variant="coordinate_rotation", nz=NZ, nx=NX, nt=NT, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0,
                       ealThick=4, freesurface=1, stype=1, seistype=seistype)
    h.upload_model(*synthetic.padded(synthetic.layered_model(NZ, NX, seed=2), 4))
    h.set_source([NX // 2], [2], synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)[None, :])
    return h


def _receivers(h, n, kinds=(0, 1), gz=3):
    for k in kinds:
        h.set_receivers(k, np.arange(n), gz)


def _observed(h, n, kinds=(0, 1)):
    for k in kinds:
        h.grad_set_observed(k, np.zeros((n, NT), np.float32))


@pytest.mark.parametrize("n", [NX, 20])
def test_another_number_of_receivers(n, gpu_lib):
    import ttifd

    with _handle() as h:
        _receivers(h, 40)
        _observed(h, 40)
        first = h.grad_run(2)
        _receivers(h, n, kinds=(1,))
        for run in (lambda: h.grad_run(2), lambda: h.grad_run_binomial(2, 10)):
            with pytest.raises(ttifd.TTIError) as e:
                run()
            assert e.value.code == ttifd.ERR_STATE
        _receivers(h, 40, kinds=(1,))  # as many as before: the traces are still there
        assert h.grad_run(2) == pytest.approx(first, rel=1e-12)
        _receivers(h, n, kinds=(1,))
        _observed(h, n, kinds=(1,))
        assert 0 < h.grad_run(2) < np.inf


def test_component_that_is_not_recorded(gpu_lib):
    """Observed traces of a component that seistype leaves out change nothing."""
    out = []
    for kinds in ((0, 1, 2), (0, 1)):
        with _handle(seistype=1) as h:
            _receivers(h, NX, (0, 1))
            _observed(h, NX, (0, 1))
            if 2 in kinds:  # the smaller arrays fall into the freed memory of the larger
                h.set_receivers(2, np.arange(NX).repeat(8), 3)
                h.grad_set_observed(2, np.full((8 * NX, NT), 1e3, np.float32))
                _receivers(h, NX, (2,))
                h.grad_set_observed(2, np.full((NX, NT), 1e3, np.float32))
            h.grad_zero()
            h.grad_run(2)
            out.append([h.grad_fetch(n) for n in ("vp", "eps", "delta", "theta")])
    for got, ref in zip(*out):
        assert np.array_equal(got.view(np.uint32), ref.view(np.uint32)) and np.any(ref != 0)
