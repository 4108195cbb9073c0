"""The tiled half-steps at the edges of their tiles (8 columns, up to 120 rows
in four warps of diagonals): one to three rows and columns, a tile exactly full
and one row or column over, two tiles of uneven remainder, a surface row that
is not a multiple of four. The per-cell kernels perform the same operations in
the same order, so fields and traces must agree bit for bit."""
import numpy as np
import pytest

import synthetic

pytestmark = pytest.mark.gpu


def _run(kernel, monkeypatch, variant, nz, nx, eal, fs, dz):
    import ttifd

    monkeypatch.setenv("TTIFD_EXACT", "1")
    monkeypatch.setenv("TTIFD_KERNEL", kernel)
    nt = 60
    cfg = dict(variant=variant, nz=nz, nx=nx, nt=nt, dx=10.0, dz=dz, dt=0.0008, fpeak=30.0, ealThick=eal,
               freesurface=fs, stype=1, seistype=3)
    m = synthetic.layered_model(nz, nx, seed=5)
    with ttifd.Modeling(**cfg) as h:
        h.upload_model(*synthetic.padded(m, eal))
        h.set_source([nx // 2], [min(2, nz - 1)], synthetic.ricker(nt, cfg["dt"], cfg["fpeak"], delay=0.01)[None, :])
        for k in (0, 1, 2):
            h.set_receivers(k, np.arange(nx), nz // 2)
        h.run()
        out = [h.fetch_traces(k) for k in (0, 1, 2)]
        out += [h.fetch_field(f) for f in range(8 if variant == "tensor_rotation" else 5)]
    return out


# updated rows: nz + 2 (eal + 5) - 10 without a free surface, less eal + 5 with one
@pytest.mark.parametrize("nz,nx,eal,fs,dz", [
    (1, 1, 1, 0, 10.0),      # 3 x 3 cells
    (2, 7, 2, 1, 10.0),      # surface row 7
    (118, 6, 1, 0, 10.0),    # 120 rows, 8 columns: one full tile
    (119, 7, 1, 0, 8.0),     # 121 rows, 9 columns: two tiles each way
    (113, 23, 4, 1, 10.0),   # surface row 9, 121 rows from row 8
    (236, 9, 2, 0, 12.5),    # 240 rows: two full tiles
    (237, 16, 2, 1, 10.0),   # surface row 7, two tiles and a remainder
])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_tile_edges(variant, nz, nx, eal, fs, dz, monkeypatch, gpu_lib):
    ref = _run("naive", monkeypatch, variant, nz, nx, eal, fs, dz)
    got = _run("tiled", monkeypatch, variant, nz, nx, eal, fs, dz)
    for k, (a, b) in enumerate(zip(got, ref)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, np.max(np.abs(a - b)))
    assert any(np.any(b != 0) for b in ref)


# The column work (sources, free surface, receivers) runs in the tiles, in one
# or two rows of tiles, or as launches of its own where a column lies outside
# the updated ones or receivers spread over more rows.
@pytest.mark.parametrize("where", ["surface", "two tiles", "all depths", "outside"])
@pytest.mark.parametrize("stype", [1, 2, 3, 4, 5, 6, 7, 8])
def test_column_work(where, stype, monkeypatch, gpu_lib):
    import ttifd

    nz, nx, nt, eal = 300, 40, 50, 0 if where == "outside" else 3
    m = synthetic.layered_model(nz, nx, seed=8)
    w = synthetic.ricker(nt, 0.0008, 30.0, delay=0.01)
    gx = np.arange(nx)
    sx, sz, gz = {"surface": ([20, 22], [2, 3], 2), "two tiles": ([20, 22], [112 - eal - 5, 105], 112),
                  "all depths": ([20, 21], [140, 3], (gx * 7) % nz), "outside": ([0, nx], [nz, 2], 2)}[where]
    out = []
    for kernel in ("naive", "tiled"):
        monkeypatch.setenv("TTIFD_EXACT", "1")
        monkeypatch.setenv("TTIFD_KERNEL", kernel)
        with ttifd.Modeling(variant=1, nz=nz, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=eal,
                            freesurface=1, stype=stype, seistype=3, mt=2) as h:
            h.upload_model(*synthetic.padded(m, eal))
            h.set_source(sx, sz, np.stack([w, 0.5 * w]))
            for k in (0, 1, 2):
                h.set_receivers(k, gx, gz)
            h.run()
            out.append([h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(8)])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, np.max(np.abs(a - b)))
    assert np.any(out[0][3] != 0)


# Column work in the tile with more than one warp of receivers in a column and
# more than one source over it, near the surface and away from it; the per-cell
# kernels' launches of their own are the reference.
@pytest.mark.parametrize("fs", [0, 1])
@pytest.mark.parametrize("variant", ["coordinate_rotation", "tensor_rotation", "bond_transformation"])
def test_crowded_columns(variant, fs, monkeypatch, gpu_lib):
    import ttifd

    nz, nx, nt, eal = 90, 30, 60, 4
    m = synthetic.layered_model(nz, nx, seed=9)
    w = synthetic.ricker(nt, 0.0008, 30.0, delay=0.01)
    gx = np.concatenate([np.full(70, 9), np.arange(nx)])
    gz = np.concatenate([np.arange(70), np.full(nx, 1)])
    out = []
    for kernel in ("naive", "tiled"):
        monkeypatch.setenv("TTIFD_EXACT", "1")
        monkeypatch.setenv("TTIFD_KERNEL", kernel)
        with ttifd.Modeling(variant=variant, nz=nz, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0,
                            ealThick=eal, freesurface=fs, stype=1, seistype=3, mt=3) as h:
            h.upload_model(*synthetic.padded(m, eal))
            h.set_source([9, 12, 8, 20], [1, 0, 6, 50], np.stack([w, 0.5 * w, -w, 2 * w]))
            for k in (0, 1, 2):
                h.set_receivers(k, gx, gz)
            h.run()
            out.append([h.fetch_traces(k) for k in (0, 1, 2)]
                       + [h.fetch_field(f) for f in range(8 if variant == "tensor_rotation" else 5)])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, np.max(np.abs(a - b)))
    assert all(np.any(b != 0) for b in out[0])


# One velocity source per column: its window at the surface (rows that are not
# updated), over two rows of tiles, and one row and column from the edge.
@pytest.mark.parametrize("sx,sz", [(20, 1), (9, 108), (1, 60)])
@pytest.mark.parametrize("stype", [2, 3, 4, 5, 6, 7, 8])
def test_velocity_source(stype, sx, sz, monkeypatch, gpu_lib):
    import ttifd

    nz, nx, nt, eal = 150, 40, 50, 3
    m = synthetic.layered_model(nz, nx, seed=8)
    w = synthetic.ricker(nt, 0.0008, 30.0, delay=0.01)
    out = []
    for kernel in ("naive", "tiled"):
        monkeypatch.setenv("TTIFD_EXACT", "1")
        monkeypatch.setenv("TTIFD_KERNEL", kernel)
        with ttifd.Modeling(variant=0, nz=nz, nx=nx, nt=nt, dx=10.0, dz=10.0, dt=0.0008, fpeak=30.0, ealThick=eal,
                            freesurface=1, stype=stype, seistype=3) as h:
            h.upload_model(*synthetic.padded(m, eal))
            h.set_source([sx], [sz], w[None, :])
            for k in (0, 1, 2):
                h.set_receivers(k, np.arange(nx), sz)
            h.run()
            out.append([h.fetch_traces(k) for k in (0, 1, 2)] + [h.fetch_field(f) for f in range(5)])
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (k, np.max(np.abs(a - b)))
        assert np.any(b != 0), k
