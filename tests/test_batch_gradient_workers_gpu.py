"""More instances than the batch gradient runs at once (8 at most): each
instance's misfit is that of the shot alone, and the sums of the model are the
shots' sums. Ten sums of FP32 fields in another order: 10 roundings of 6e-8;
bound 1e-6."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shots", [7, 10])
def test_more_instances_than_workers(shots, gpu_lib):
    import ttifd

    nz, nx, nt, eal = 50, 70, 120, 5
    cfg = dict(variant=0, nz=nz, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=eal, freesurface=1,
               stype=1, seistype=1)
    m = synthetic.padded(synthetic.layered_model(nz, nx, seed=3), eal)
    w = synthetic.ricker(nt, cfg["dt"], cfg["fpeak"], delay=0.01)[None, :]
    dobs = np.zeros((nx, nt), np.float32)
    names = ("vp", "eps", "delta", "theta")

    def shot(h, i):
        h.set_source([5 + 6 * i], [2], w)
        for k in (0, 1):
            h.set_receivers(k, np.arange(nx), 4)
            h.grad_set_observed(k, dobs)

    with ttifd.Batch([cfg], [0] * shots) as b:
        b.upload_model(0, *m)
        for i in range(shots):
            shot(b.instances[i], i)
        j = b.grad_run(3, 10)
        got = [b.instances[0].grad_fetch(n) for n in names]
    with ttifd.Modeling(**cfg) as h:
        h.upload_model(*m)
        h.grad_zero()
        jr = []
        for i in range(shots):
            shot(h, i)
            jr.append(h.grad_run_binomial(3, 10))
        ref = [h.grad_fetch(n) for n in names]
    assert j == pytest.approx(jr, rel=1e-12) and min(jr) > 0
    for a, r in zip(got, ref):
        assert np.linalg.norm(a.astype(np.float64) - r) <= 1e-6 * np.linalg.norm(r.astype(np.float64))
