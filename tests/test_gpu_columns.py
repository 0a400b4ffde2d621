"""Column-wise Siddon cone projectors (upright views) at the sizes where they
can go wrong: rows around the 16-lane and 64-row passes, z around the 32-voxel
chunks, detector windows wider than the staged one, flipped axes, and views
left to the ray-driven kernels."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# A ray or a voxel adds at most n = 1000 FP32 terms here, each rounded to 2^-24
# of the partial sum: sqrt(n) 2^-24 = 1.9e-6 for random signs, and a segment
# split at a z plane is off by up to 2^-24 of z (128 voxels) over its z rise
# (about 1% of the segments, less than 1e-4 of a voxel each).
TOL = 4e-6


SIDDON_COLUMNS = 0x800  # CTP_FLAG_SIDDON_COLUMNS: the column kernels at these sizes too


@pytest.fixture(autouse=True)
def _columns(monkeypatch):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from ctprojector_b200.projector import _device

    flags = _device._io_flags
    monkeypatch.setattr(_device, "_io_flags", lambda a, b: flags(a, b) | SIDDON_COLUMNS)


def scan(nx, ny, nz, nu, nv, nview=13, pixel=3.0, dz=2.0, cell=None, row=None, **kw):
    from cases import Proj

    cell = cell if cell is not None else 1.9 * pixel * max(nx, ny) / nu
    row = row if row is not None else 1.9 * dz * nz / nv
    return Proj(nx=nx, ny=ny, nz=nz, dx=pixel, dy=pixel, dz=dz, nu=nu, nv=nv, du=cell, dv=row, nview=nview, **kw)


def helix(p, feed=0.0):
    from ctprojector_b200 import synthetic as S

    return list(S.helical(p.nview, 1.0, p.dso, p.dsd, feed))


def check(p, geo, oracle, nbatch=1, tol=TOL):
    from ctprojector_b200.projector.cupy import cone

    rng = np.random.default_rng(p.nu + p.nv)
    img = rng.uniform(0, 1, (nbatch, p.nz, p.ny, p.nx)).astype(np.float32)
    prj = rng.uniform(-0.5, 1, (nbatch, p.nview, p.nv, p.nu)).astype(np.float32)
    dev = [torch.tensor(a, device="cuda") for a in geo]
    fp = cone.siddon_fp_arbitrary(p, torch.tensor(img, device="cuda"), *dev).cpu().numpy()
    bp = cone.siddon_bp_arbitrary(p, torch.tensor(prj, device="cuda"), *dev).cpu().numpy()
    assert rel_l2(fp, oracle.siddon_fp(p, img, *geo)) <= tol
    assert rel_l2(bp, oracle.siddon_bp(p, prj, *geo)) <= tol


@pytest.mark.parametrize("nz,nv", [(4, 8), (16, 17), (31, 16), (32, 33), (33, 48), (40, 65), (65, 130)])
def test_rows_and_slices(nz, nv, oracle):
    p = scan(37, 29, nz, 53, nv)
    check(p, helix(p, feed=0.4 * nz * p.dz), oracle, nbatch=2)


@pytest.mark.parametrize("nx,ny,nu", [(16, 16, 16), (17, 47, 33), (64, 15, 129), (48, 48, 400)])
def test_grid_and_detector_sizes(nx, ny, nu, oracle):
    """400 cells over 48 pixels: windows wider than the staged one."""
    p = scan(nx, ny, 12, nu, 12, off_u=0.3, off_v=-0.7, cx=1.5, cy=-2.0, cz=0.6)
    check(p, helix(p), oracle)


@pytest.mark.parametrize("row", [0.2, 30.0])
def test_fine_and_coarse_rows(row, oracle):
    """0.2 mm rows: many through one plane inside a pixel, and more than the staged rows per chunk."""
    p = scan(24, 24, 36, 40, 150 if row < 1 else 9, dz=1.0, row=row)
    check(p, helix(p), oracle)


@pytest.mark.parametrize("flip", ["u", "v", "uv"])
def test_flipped_detector_axes(flip, oracle):
    p = scan(33, 40, 20, 50, 24)
    geo = helix(p, feed=10.0)
    if "u" in flip:
        geo[1] = -geo[1]
    if "v" in flip:
        geo[2] = -geo[2]
    check(p, geo, oracle)


def test_tilted_views_among_upright_ones(oracle):
    """Every third view tilts its detector: the ray-driven kernels take those."""
    p = scan(33, 28, 18, 44, 21)
    geo = helix(p, feed=8.0)
    a = 0.15
    for k in range(0, p.nview, 3):
        u, v = geo[1][k].copy(), geo[2][k].copy()
        geo[1][k] = np.cos(a) * u + np.sin(a) * v
        geo[2][k] = np.cos(a) * v - np.sin(a) * u
    check(p, geo, oracle)


def test_infinite_and_nan_cells_stay_on_their_rays(oracle):
    """A view with an infinity or NaN is scattered ray by ray: the voxels that
    its ray does not cross are those of the projections without it."""
    from ctprojector_b200.projector.cupy import cone

    p = scan(24, 24, 12, 30, 14)
    geo = helix(p)
    dev = [torch.tensor(a, device="cuda") for a in geo]
    prj = np.random.default_rng(3).uniform(0, 1, (1, p.nview, p.nv, p.nu)).astype(np.float32)
    bad = prj.copy()
    bad[0, 4, 6, 15] = np.nan
    bad[0, 7, 3, 11] = np.inf
    mark = np.zeros_like(prj)
    mark[0, 4, 6, 15] = mark[0, 7, 3, 11] = 1
    chord = oracle.siddon_bp(p, mark, *geo)
    out = cone.siddon_bp_arbitrary(p, torch.tensor(bad, device="cuda"), *dev).cpu().numpy()
    ref = oracle.siddon_bp(p, np.where(mark > 0, 0, prj).astype(np.float32), *geo)
    assert not np.isfinite(out[chord > 1e-3]).any()
    clean = (chord == 0) & np.isfinite(out)
    assert (chord == 0).sum() - clean.sum() <= 2  # a ray may graze one voxel more or less
    assert rel_l2(out[clean], ref[clean]) <= TOL


def test_large_cell_leaves_the_other_rows_alone(oracle):
    """One cell of 1e6 among values of order one: voxels off its ray keep their bits."""
    from ctprojector_b200.projector.cupy import cone

    p = scan(24, 24, 24, 30, 28)
    geo = helix(p)
    dev = [torch.tensor(a, device="cuda") for a in geo]
    prj = np.random.default_rng(3).uniform(0.5, 1, (1, p.nview, p.nv, p.nu)).astype(np.float32)
    for big in (300.0, 1e4, 1e6):
        mark = np.zeros_like(prj)
        mark[0, 4, 6, 15] = mark[0, 7, 3, 11] = 1
        out = cone.siddon_bp_arbitrary(p, torch.tensor(np.where(mark > 0, np.float32(big), prj), device="cuda"), *dev)
        out = out.cpu().numpy()
        away = oracle.siddon_bp(p, mark, *geo) == 0
        ref = oracle.siddon_bp(p, np.where(mark > 0, 0, prj).astype(np.float32), *geo)
        bad = np.abs(out - ref)[away] > 4 * TOL * np.abs(ref).max()
        assert bad.sum() <= 2, big  # a ray may graze one voxel more or less


@pytest.mark.parametrize("nv", [70, 200, 512])
def test_tall_detectors(nv, oracle):
    """The rows before a voxel's do not cost it precision, however many there are."""
    from ctprojector_b200.projector.cupy import cone

    p = scan(16, 16, int(nv / 1.7), 20, nv, pixel=1.0, dz=1.0, nview=3)
    geo = helix(p, feed=0.1 * nv)
    prj = np.random.default_rng(nv).uniform(1, 2, (1, p.nview, nv, p.nu)).astype(np.float32)
    out = cone.siddon_bp_arbitrary(p, torch.tensor(prj, device="cuda"), *[torch.tensor(a, device="cuda") for a in geo])
    # a voxel adds about ten terms
    assert rel_l2(out.cpu().numpy(), oracle.siddon_bp(p, prj, *geo)) <= TOL / 4


def test_no_less_exact_than_ray_by_ray(oracle, monkeypatch):
    """The back projection's error against 64 bits, by columns and by rays on the
    same projections (97 and 180 views add up to 700 terms a voxel)."""
    from ctprojector_b200.projector import _device
    from ctprojector_b200.projector.cupy import cone

    flags = _device._io_flags
    for n, nz, nu, nv, nview in ((100, 33, 126, 37, 97), (96, 40, 138, 40, 180)):
        p = scan(n, n, nz, nu, nv, nview=nview, pixel=358.0 / n, dz=1.1, cell=946.0 / nu, row=1.6)
        geo = helix(p, feed=nz * p.dz)
        dev = [torch.tensor(a, device="cuda") for a in geo]
        prj = np.random.default_rng(n).uniform(0, 1, (1, nview, nv, nu)).astype(np.float32)
        ref = oracle.siddon_bp(p, prj, *geo)
        x = torch.tensor(prj, device="cuda")
        columns = rel_l2(cone.siddon_bp_arbitrary(p, x, *dev).cpu().numpy(), ref)
        with monkeypatch.context() as m:
            m.setattr(_device, "_io_flags", lambda a, b: flags(a, b) & ~SIDDON_COLUMNS)
            rays = rel_l2(cone.siddon_bp_arbitrary(p, x, *dev).cpu().numpy(), ref)
        assert columns <= 1.02 * rays, (nview, columns, rays)  # (both are sums of some 1e6 roundings)


@pytest.mark.parametrize("nx,nu,nv", [(150, 195, 31), (64, 65, 33), (32, 33, 64)])
def test_rays_along_grid_planes(nx, nu, nv, oracle):
    """An odd detector over an even grid, views at 0, 90, 180 and 270 degrees: the
    middle column's rays run along the plane between two pixel columns, and belong
    to the side on which each enters the grid."""
    p = scan(nx, nx, 32, nu, nv, nview=12, pixel=358.0 / nx, dz=1.1)
    check(p, helix(p, feed=35.0), oracle)
    check(p, helix(p), oracle)


@pytest.mark.parametrize("n,nu", [(64, 65), (32, 33), (150, 195), (33, 47)])
def test_rays_through_pixel_corners(n, nu, oracle):
    """The middle column at 45 degrees runs from corner to corner of square pixels."""
    p = scan(n, n, 32, nu, 32, nview=8, pixel=358.0 / n, dz=1.1)
    check(p, helix(p, feed=35.0), oracle)
    check(p, helix(p), oracle)


@pytest.mark.parametrize("cz", [-1.665, -1.664, -1.66, 0.555, 0.5551, 4.995, 4.9949999, 4.9950005, -4.995, -4.9950005])
def test_level_rays_beside_slice_planes(cz, oracle):
    """The middle row of an odd panel is level at the source's height, here at
    1.665 / 1.11 = 1.5 slices and nearly so from the middle of nine (7e-8, 9e-4 and
    more of a slice from a plane), and at the lowest and the highest plane."""
    p = scan(40, 40, 9, 52, 33, nview=10, pixel=9.0, dz=1.11, cz=cz)
    check(p, helix(p), oracle)


def test_columns_by_their_own_size_rule(oracle, monkeypatch):
    """A scan that both size rules accept by themselves: the forward projection's
    bits are those of the flagged call, not those of the rays (views that a
    rounding of the detector axis keeps from being upright)."""
    from ctprojector_b200.projector import _device
    from ctprojector_b200.projector.cupy import cone

    p = scan(128, 128, 32, 64, 48, nview=300, pixel=2.8, dz=1.2, cell=14.0, row=1.6)
    geo = helix(p, feed=20.0)
    rng = np.random.default_rng(0)
    img = rng.uniform(0, 1, (1, p.nz, p.ny, p.nx)).astype(np.float32)
    prj = rng.uniform(0, 1, (1, p.nview, p.nv, p.nu)).astype(np.float32)
    flags = _device._io_flags

    def run(geo):
        dev = [torch.tensor(a, device="cuda") for a in geo]
        return (cone.siddon_fp_arbitrary(p, torch.tensor(img, device="cuda"), *dev).cpu().numpy(),
                cone.siddon_bp_arbitrary(p, torch.tensor(prj, device="cuda"), *dev).cpu().numpy())

    flagged = run(geo)
    with monkeypatch.context() as m:
        m.setattr(_device, "_io_flags", lambda a, b: flags(a, b) & ~SIDDON_COLUMNS)
        fp, bp = run(geo)
        tilted = [a.copy() for a in geo]
        tilted[1][:, 2] = 1e-12
        rays, _ = run(tilted)
    np.testing.assert_array_equal(fp, flagged[0])
    assert not np.array_equal(fp, rays)
    assert rel_l2(fp, oracle.siddon_fp(p, img, *geo)) <= TOL
    assert rel_l2(bp, oracle.siddon_bp(p, prj, *geo)) <= TOL


@pytest.mark.parametrize("nv", [2, 25, 57])
@pytest.mark.parametrize("flip", ["axis", "pitch"])
def test_level_rows_of_a_panel_upside_down(flip, nv, oracle):
    """Rows on slice planes exactly, with rows that go down: they belong to the
    slice above, as they do with rows that go up."""
    p = scan(33, 40, 32, 50, nv, dz=1.0, off_v=0.5 if nv == 2 else 0.0)
    geo = helix(p, feed=16.0)
    if flip == "axis":
        geo[2] = -geo[2]
    else:
        p.dv = -p.dv
    check(p, geo, oracle)
    check(p, [*helix(p)[:2], geo[2], helix(p)[3]], oracle)
