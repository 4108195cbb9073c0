"""Either grid setting over several waves of work items, with items of finished
instances in between: fields and traces agree bit for bit."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu
WAVE = 4 * 148  # the most CTAs that are resident together
NZ, EAL = 120, 6


def _tiles(nx):
    """Tiles of a model of NZ rows with a free surface (8 columns, up to 120 rows)."""
    E = EAL + 5
    rows = NZ + 2 * E - 5 - E // 8 * 8
    return -(-rows // 120) * -(-(nx + 2 * E - 10) // 8)


@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_several_waves(variant, monkeypatch, gpu_lib):
    import ttifd

    monkeypatch.delenv("TTIFD_EXACT", raising=False)
    nxs, nts, modes, model_of = (820, 611), (45, 32), (1, 2), [0, 1, 0, 0, 1, 0, 1, 0, 0, 1, 0, 0, 1, 0]
    assert sum(_tiles(nxs[m]) for m in model_of) > 4 * WAVE
    cfgs = [dict(variant=variant, nz=NZ, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=EAL,
                 freesurface=1, stype=1, seistype=3, mt=2, mode=mode) for nx, nt, mode in zip(nxs, nts, modes)]
    models = [synthetic.padded(synthetic.layered_model(NZ, nx, seed=nx), EAL) for nx in nxs]
    fields = 8 if variant == "tensor_rotation" else 5
    out = []
    for grid in ("per-tile", "persistent"):
        with ttifd.Batch(cfgs, model_of) as b:
            for m, model in enumerate(models):
                b.upload_model(m, *model)
            b.set_schedule(grid)
            for i, m in enumerate(model_of):
                # sources all over the model, so that hardly a tile stays at rest
                sx = np.arange(2 + i, nxs[m], 13)
                w = synthetic.ricker(nts[m], 0.0008, 30.0, delay=0.01)
                b.instances[i].set_source(sx, (sx * 29 + i) % NZ, np.stack([w * (1 + k % 5) for k in range(len(sx))]))
                for k in (0, 1, 2):
                    b.instances[i].set_receivers(k, np.arange(nxs[m]), (np.arange(nxs[m]) * 7 + i) % NZ)
            b.run()
            out.append([[h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(fields)]
                        for h in b.instances])
    for i, (got, ref) in enumerate(zip(out[1], out[0])):
        for k, (a, r) in enumerate(zip(got, ref)):
            assert np.array_equal(a.view(np.uint32), r.view(np.uint32)), (i, k)
            assert np.mean(r != 0) > 0.5, (i, k)
