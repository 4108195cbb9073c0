"""The tiled adjoint kernels at the edges of their tiles (8 columns, up to 120
rows, the first tile from five rows above a free surface), and where the
column work (receivers, source window) reaches cells outside the tiles, so that
it runs as a launch of its own. Against the per-cell kernels: both are FP32
with other roundings, about 50 operations a cell and step of 6e-8 each whose
errors add as a random walk over 50 steps, 3e-6; the bound is 2e-5."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu


def _run(kernel, monkeypatch, variant, nz, nx, eal, fs, edge):
    import ttifd

    monkeypatch.setenv("TTIFD_KERNEL", kernel)
    nt = 50
    cfg = dict(variant=variant, nz=nz, nx=nx, nt=nt, dx=10.0, dz=9.0, dt=0.0008, fpeak=30.0, ealThick=eal,
               freesurface=fs, stype=1, seistype=3, mt=2)
    m = synthetic.layered_model(nz, nx, seed=5)
    rng = np.random.default_rng(nz + nx)
    with ttifd.Modeling(**cfg) as h:
        h.upload_model(*synthetic.padded(m, eal))
        sx, sz = (0, nz) if edge else (nx // 2, nz // 2)
        h.set_source([sx], [sz], synthetic.ricker(nt, cfg["dt"], cfg["fpeak"], delay=0.01)[None, :])
        for k, amp in ((0, 5e-12), (1, 5e-12), (2, 4e-5)):
            h.set_receivers(k, np.arange(nx + 1) if edge else np.arange(nx),
                            nz - 4 if edge else max(nz // 2 - 3, 0))
            t = np.cumsum(rng.standard_normal((nx + 1 if edge else nx, h.nts)), axis=1)
            h.grad_set_observed(k, (amp * t / 5).astype(np.float32))
        h.grad_zero()
        j = h.grad_run(3)
        out = [h.grad_fetch(g) for g in ("vp", "eps", "delta", "theta")] + [h.grad_fetch_source(1)]
    return j, out


@pytest.mark.parametrize("nz,nx,eal,fs,edge", [
    (1, 1, 1, 0, False),     # 3 x 3 cells
    (119, 7, 1, 0, False),   # 121 rows, 9 columns: two tiles each way
    (112, 23, 4, 1, False),  # 121 rows from the first image row on
    (237, 16, 2, 1, False),  # two tiles and a remainder, surface row 7
    (30, 20, 0, 0, True),    # receivers and source window outside the update
    (30, 20, 0, 1, True),
])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_tile_edges(variant, nz, nx, eal, fs, edge, monkeypatch, gpu_lib):
    jr, ref = _run("naive", monkeypatch, variant, nz, nx, eal, fs, edge)
    j, got = _run("tiled", monkeypatch, variant, nz, nx, eal, fs, edge)
    assert abs(j - jr) <= 1e-12 * jr
    for k, (a, b) in enumerate(zip(got, ref)):
        assert np.any(b != 0), k
        rel = np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64))
        assert rel <= 2e-5, (k, rel)


# Column work in the tiles with more than one warp of receivers in a column and
# more than one source over it; receivers of every component share cells.
@pytest.mark.parametrize("fs", [0, 1])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_crowded_columns(variant, fs, monkeypatch, gpu_lib):
    import ttifd

    nz, nx, nt, eal = 90, 30, 50, 4
    m = synthetic.layered_model(nz, nx, seed=9)
    w = synthetic.ricker(nt, 0.0008, 30.0, delay=0.01)
    gx = np.concatenate([np.full(70, 9), np.arange(nx), np.arange(nx)])
    gz = np.concatenate([np.arange(70), np.full(nx, 1), np.full(nx, 1)])
    out = []
    for kernel in ("naive", "tiled"):
        monkeypatch.setenv("TTIFD_KERNEL", kernel)
        rng = np.random.default_rng(7)
        with ttifd.Modeling(variant=variant, nz=nz, nx=nx, nt=nt, dx=10.0, dz=9.0, dt=0.0008, fpeak=30.0,
                            ealThick=eal, freesurface=fs, stype=1, seistype=3) as h:
            h.upload_model(*synthetic.padded(m, eal))
            h.set_source([9, 12, 8, 20], [1, 0, 6, 50], np.stack([w, 0.5 * w, -w, 2 * w]))
            for k, amp in ((0, 5e-12), (1, 5e-12), (2, 4e-5)):
                h.set_receivers(k, gx, gz)
                t = np.cumsum(rng.standard_normal((len(gx), h.nts)), axis=1)
                h.grad_set_observed(k, (amp * t / 5).astype(np.float32))
            h.grad_zero()
            j = h.grad_run(2)
            out.append((j, [h.grad_fetch(g) for g in ("vp", "eps", "delta", "theta")] + [h.grad_fetch_source(4)]))
    (jr, ref), (jt, got) = out
    assert abs(jt - jr) <= 1e-12 * jr
    for k, (a, b) in enumerate(zip(got, ref)):
        assert np.any(b != 0), k
        rel = np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64))
        assert rel <= 2e-5, (k, rel)
