"""Many sources, half of them in one column, the others where they happen to
fall, so that their windows overlap: added in the list's order, as the CPU
restatement of the reference adds them. Both round every product and sum
separately, so traces and fields agree bit for bit. Sources along the surface
are added in the tiles, sources at all depths by launches of their own; a batch
always uses launches of its own."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
NZ, NX, NT, EAL = 290, 90, 40, 4


def _shot(h, n, where):
    rng = np.random.default_rng(n)
    sx, sz = rng.integers(0, NX, n), rng.integers(0, 6 if where == "surface" else NZ, n)
    sx[n // 2:] = sx[0]  # half of them in one column
    w = synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)
    h.set_source(sx, sz, np.stack([w * np.float32(a) for a in rng.uniform(-2, 2, n)]))
    # and more than a warp of receivers in a column, which with two sources none reaches
    gx, gz = np.append(np.arange(NX), np.full(40, NX - 1)), np.append(np.full(NX, 3), np.arange(40))
    for k in (0, 1, 2):
        h.set_receivers(k, gx, gz)


def _result(h):
    return [h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(5)]


@pytest.mark.parametrize("where", ["surface", "all depths", "batch"])
@pytest.mark.parametrize("n", [2, 33, 100])
@pytest.mark.parametrize("variant,stype", [("coordinate_rotation", 1), ("tensor_rotation", 1),
                                           ("bond_transformation", 4), ("coordinate_rotation", 6),
                                           ("coordinate_rotation", 8)])
def test_order_of_sources(variant, stype, n, where, monkeypatch, gpu_lib, oracle_lib):
    import ttifd

    monkeypatch.delenv("TTIFD_EXACT", raising=False)
    cfg = dict(variant=variant, nz=NZ, nx=NX, nt=NT, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=EAL,
               freesurface=1, stype=stype, seistype=3)
    m = synthetic.padded(synthetic.layered_model(NZ, NX, seed=8), EAL)
    with oracle_lib.Oracle(**cfg) as o:
        o.upload_model(*m)
        _shot(o, n, where)
        o.run()
        ref = _result(o)
    if where == "batch":
        with ttifd.Batch([cfg], [0, 0]) as b:
            b.upload_model(0, *m)
            for h in b.instances:
                _shot(h, n, where)
            b.run()
            got = _result(b.instances[1])
    else:
        with ttifd.Modeling(**cfg) as h:
            h.upload_model(*m)
            _shot(h, n, where)
            h.run()
            got = _result(h)
    for k, (a, r) in enumerate(zip(got, ref)):
        assert np.array_equal(a.view(np.uint32), r.view(np.uint32)), (k, np.max(np.abs(a - r)))
        assert np.any(r != 0), k
