"""Row-sharing tomosynthesis kernels at the sizes where they can go wrong: rows
and planes around their tiles, footprints on both sides of the 2 x 2 and 3 x 3
cells that they hold, borders and weights; against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# sums of at most 17 planes or 11 views of FP32 products of two weights, each
# rounded to 2^-24 of a value of order one after a subtraction of coordinates
# below 2^9: 2^-24 2^2 at random over the terms
TOL = 1e-6


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda")


@pytest.mark.parametrize("nx,ny,nz,nu,nv,cell", [(129, 7, 3, 130, 9, 0.3), (40, 33, 9, 257, 65, 0.25), (64, 40, 17, 31, 33, 0.4),
                                                 (64, 40, 17, 31, 33, 0.45),
                                                 (50, 37, 8, 40, 24, 1.1)])
def test_tomo_rows(nx, ny, nz, nu, nv, cell, oracle):
    """Rows and planes around the kernels' tiles; 0.45 and 1.1 mm cells take one
    rectangle per thread."""
    from cases import Proj

    from ctprojector_b200 import synthetic as S
    from ctprojector_b200.projector.cupy import tomo

    p = Proj(nx=nx, ny=ny, nz=nz, dx=0.4, dy=0.4, dz=1.0, nu=nu, nv=nv, du=cell, dv=cell, nview=11, off_u=0.3, off_v=-0.4)
    dc, sr = S.tomo_geometry(11, 40.0, 500.0, -(nz / 2 + 15.0))
    rng = np.random.default_rng(nx)
    img = rng.uniform(0, 1, (2, nz, ny, nx)).astype(np.float32)
    prj = rng.uniform(0, 1, (2, 11, nv, nu)).astype(np.float32)
    fp = tomo.distance_driven_fp(p, dev(img), dev(dc), dev(sr)).cpu().numpy()
    bp = tomo.distance_driven_bp(p, dev(prj), dev(dc), dev(sr)).cpu().numpy()
    # one rectangle per thread takes its edges in FP32 relative to the source, up to
    # 182 mm to the side: 182 / 0.4 pixels of 2^-23 between a footprint's two edges
    tol = TOL if cell <= 0.4 else 182 / 0.4 * 2.0**-23
    assert rel_l2(fp, oracle.tomo_fp(p, img, dc, sr)) <= tol
    assert rel_l2(bp, oracle.tomo_bp(p, prj, dc, sr)) <= tol


def scan(nx, ny, nz, nu, nv, cell, nview, **kw):
    from cases import Proj

    from ctprojector_b200 import synthetic as S

    p = Proj(nx=nx, ny=ny, nz=nz, dx=0.4, dy=0.4, dz=1.0, nu=nu, nv=nv, du=cell, dv=cell, nview=nview, **kw)
    dc, sr = S.tomo_geometry(nview, 40.0, 500.0, -(nz / 2 + 15.0))
    return p, dc, sr


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_tomo_values_off_the_footprint_do_not_matter(bad, oracle):
    """Cells and pixels that a footprint does not reach, though it was clamped
    to the border they lie on, leave its result alone."""
    p, dc, sr = scan(48, 40, 9, 100, 90, 0.3, 11)
    rng = np.random.default_rng(2)
    img = rng.uniform(0, 1, (1, 9, 40, 48)).astype(np.float32)
    mark = np.zeros_like(img)
    for z, y, x in ((4, 0, 20), (3, 39, 11), (6, 17, 0), (2, 25, 47), (5, 0, 0)):
        img[0, z, y, x] = bad
        mark[0, z, max(y - 1, 0):y + 2, max(x - 1, 0):x + 2] = 1
    away = oracle.tomo_fp(p, mark, dc, sr) == 0
    ref = oracle.tomo_fp(p, np.where(np.isfinite(img), img, 0).astype(np.float32), dc, sr)
    out = tomo_call("distance_driven_fp", p, img, dc, sr)
    assert away.any() and np.isfinite(out[away]).all()
    assert rel_l2(out[away], ref[away]) <= TOL

    p, dc, sr = scan(96, 80, 9, 40, 30, 0.3, 11)  # voxels past the detector's borders
    prj = rng.uniform(0, 1, (1, 11, 30, 40)).astype(np.float32)
    mark = np.zeros_like(prj)
    for view, v, u in ((0, 0, 20), (3, 29, 11), (6, 17, 0), (9, 25, 39), (10, 29, 39)):
        prj[0, view, v, u] = bad
        mark[0, view, max(v - 2, 0):v + 3, max(u - 2, 0):u + 3] = 1
    away = oracle.tomo_bp(p, mark, dc, sr) == 0
    ref = oracle.tomo_bp(p, np.where(np.isfinite(prj), prj, 0).astype(np.float32), dc, sr)
    out = tomo_call("distance_driven_bp", p, prj, dc, sr)
    assert away.any() and np.isfinite(out[away]).all()
    assert rel_l2(out[away], ref[away]) <= TOL


def tomo_call(name, p, x, dc, sr):
    from ctprojector_b200.projector.cupy import tomo

    return getattr(tomo, name)(p, dev(x), dev(dc), dev(sr)).cpu().numpy()


def test_tomo_bp_more_views_than_a_grid_dimension(oracle):
    """Views times batch items past 65535."""
    nview = 33000
    p, dc, sr = scan(5, 4, 1, 6, 5, 0.3, nview)
    prj = np.random.default_rng(0).uniform(0, 1, (2, nview, 5, 6)).astype(np.float32)
    # 33000 terms in one FP32 sum: sqrt(33000 / 3) 2^-24 = 6e-6
    assert rel_l2(tomo_call("distance_driven_bp", p, prj, dc, sr), oracle.tomo_bp(p, prj, dc, sr)) <= 1.2e-5


def test_tomo_ray_length_weight_is_rounded_once():
    """A panel in the plane of the voxels, one voxel per cell: the voxels of a
    projection of ones are the cells' weights, FP64 values rounded to FP32."""
    from cases import Proj

    n, m = 200, 150
    p = Proj(nx=n, ny=m, nz=1, dx=0.5, dy=0.5, dz=1.0, nu=n, nv=m, du=0.5, dv=0.5, nview=1, off_u=0.5, off_v=0.5)
    sr = np.array([[13.3, -7.1, 613.7]], np.float32)
    out = tomo_call("distance_driven_bp", p, np.ones((1, 1, m, n)), np.zeros((1, 3)), sr)[0, 0]
    s = sr[0].astype(np.float64)
    u = (np.arange(n) - 0.5 - (n - 1) / 2) * 0.5 - s[0]
    v = (np.arange(m) - 0.5 - (m - 1) / 2) * 0.5 - s[1]
    ref = (1 / abs(s[2]) * np.sqrt(u * u + v[:, None] ** 2 + s[2] ** 2)).astype(np.float32)
    assert (out != ref).mean() < 1e-3


@pytest.mark.parametrize("cell,det_z", [(0.24, -25.0), (0.25, -170.0), (0.4, 1.5)])
def test_tomo_footprints_past_the_rows(cell, det_z, oracle):
    """Both sides of the footprints that the rows hold, within the sizes that
    take them: 0.24 mm is 0.6 of a pixel; 0.25 mm under a panel far below, where
    voxels span 2.1 cells and more (magnification above 1.3); and a panel inside
    the volume, past which the footprints of 0.4 mm cells exceed a pixel."""
    from cases import Proj

    from ctprojector_b200 import synthetic as S

    p = Proj(nx=45, ny=37, nz=21, dx=0.4, dy=0.4, dz=1.0, nu=90, nv=70, du=cell, dv=cell, nview=7)
    dc, sr = S.tomo_geometry(7, 30.0, 500.0, det_z)
    rng = np.random.default_rng(9)
    img = rng.uniform(0, 1, (1, 21, 37, 45)).astype(np.float32)
    prj = rng.uniform(0, 1, (1, 7, 70, 90)).astype(np.float32)
    assert rel_l2(tomo_call("distance_driven_fp", p, img, dc, sr), oracle.tomo_fp(p, img, dc, sr)) <= TOL_WIDE
    assert rel_l2(tomo_call("distance_driven_bp", p, prj, dc, sr), oracle.tomo_bp(p, prj, dc, sr)) <= TOL_WIDE


# whole rectangles take their edges in FP32 from the array's corner: up to 90 cells
# of 2^-24 between a footprint's two edges
TOL_WIDE = 90 * 2.0**-24
