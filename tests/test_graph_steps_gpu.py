"""Steps that go out as replays of a captured graph are the steps that go out
as launches: fields, traces, snapshots and gradients agree bit for bit. Whole
replays and remainders, both time directions, runs in pieces, other sources
and receivers between runs, checkpointed gradient segments."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
NZ, NX, NT = 30, 40, 217


def _handle(variant, mode):
    import ttifd

    h = ttifd.Modeling(variant=variant, nz=NZ, nx=NX, nt=NT, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=6,
                       freesurface=1, stype=1, seistype=3, mt=2, mode=mode, wsave=3, snap_sample=33)
    h.upload_model(*synthetic.padded(synthetic.layered_model(NZ, NX, seed=5), 6))
    return h


def _geometry(h, sx, gz):
    w = synthetic.ricker(NT, 0.0008, 30.0, delay=0.01)
    h.set_source([sx, sx + 3], [2, 4], np.stack([w, 0.5 * w]))
    for k in (0, 1, 2):
        h.set_receivers(k, np.arange(NX), gz)


def _state(h):
    return [h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(5)]


def _run(how, variant, launches):
    with _handle(variant, 2 if how == "reversed" else 1) as h:
        _geometry(h, 12, 2)
        out = []
        if how == "gradient":
            rng = np.random.default_rng(3)
            for k, amp in ((0, 5e-12), (1, 5e-12), (2, 4e-5)):
                t = np.cumsum(rng.standard_normal((NX, h.nts)), axis=1)
                h.grad_set_observed(k, (amp * t / 5).astype(np.float32))
            for ncheck in (1, 3):
                h.grad_zero()
                out.append(np.float32(h.grad_run(ncheck)))
                out += [h.grad_fetch(g) for g in ("vp", "eps", "delta", "theta")]
        elif how == "snapshots":
            h.run(lambda it, kind, a: out.append(a.copy()))
        elif how == "pieces":
            h.run()
            h.reset()
            for n in (1, 10, 11, 35, 160):
                h.step(n)
        else:
            h.run()
        out += _state(h)
        _geometry(h, 20, 5)  # another shot on the same handle
        h.run()
        out += _state(h)
        launches.append(h.kernel_launches)
        return out


@pytest.mark.parametrize("how", ["run", "reversed", "pieces", "snapshots", "gradient"])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_replays(variant, how, monkeypatch, gpu_lib):
    launches = []
    got = _run(how, variant, launches)
    monkeypatch.setenv("TTIFD_GRAPH_STEPS", "0")
    ref = _run(how, variant, launches)
    assert launches[0] > launches[1]  # the replays' step counters
    assert len(got) == len(ref) and any(np.any(b != 0) for b in ref)
    for k, (a, b) in enumerate(zip(got, ref)):
        assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32)), k


# Either side of the largest grid whose launches trigger the next one at their
# start and go out as replays (296 tiles of 8 columns), against the per-cell
# kernels.
@pytest.mark.parametrize("tiles", [296, 297])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation"])
def test_two_launches_on_the_device(variant, tiles, monkeypatch, gpu_lib):
    import ttifd

    nz, eal, nt = 12, 2, 215
    nx = 8 * tiles - 2 * eal
    m = synthetic.layered_model(nz, nx, seed=4)
    out = []
    for kernel in ("tiled", "naive"):
        monkeypatch.setenv("TTIFD_KERNEL", kernel)
        with ttifd.Modeling(variant=variant, nz=nz, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0,
                            ealThick=eal, freesurface=1, stype=1, seistype=3) as h:
            h.upload_model(*synthetic.padded(m, eal))
            w = synthetic.ricker(nt, 0.0008, 30.0, delay=0.01)
            h.set_source([nx // 2, 7], [3, 5], np.stack([w, w]))
            for k in (0, 1, 2):
                h.set_receivers(k, np.arange(nx), 2)
            h.run()
            out.append([h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(5)])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, np.max(np.abs(a - b)))
        assert np.any(b != 0), k
