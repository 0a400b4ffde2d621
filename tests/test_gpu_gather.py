"""The tiled gather back projection (mean, FBP, adjoint, pixel-driven) at the
sizes where it can go wrong: ragged tiles, one to five slices per CTA group, more views than one list, wide tiles,
flipped detectors and angles that are not numbers; against the FP64 oracle."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# A pixel adds one FP32 term per view (n <= 1100 here, in sums of at most 1024),
# each the difference of two table entries of up to 60 cells: a few 2^-24 of 60
# cells over a footprint of about one, at random over the views: below
# 60 2^-23 / sqrt(40) = 1.1e-6 at 40 views and less with more.
TOL = 3e-6


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def dev(a):
    return torch.tensor(np.ascontiguousarray(a, dtype=np.float32), device="cuda")


def proj(geom, nx, ny, nu, nz=1, pixel=1.0, nview=40, **kw):
    from cases import Proj

    cell = kw.pop("cell", (1.35 if geom == "parallel" else 2.5) * np.hypot(nx, ny) * pixel / nu)
    return Proj(nx=nx, ny=ny, nz=nz, dx=pixel, dy=pixel * kw.pop("aspect", 1.0), nu=nu, nv=nz, du=cell, dv=1.0,
                nview=nview, **kw)


def angles(nview, geom, start=0.013):
    span = np.pi if geom == "parallel" else 2 * np.pi
    return (start + np.arange(nview) * span / nview).astype(np.float32)


def module(geom):
    from ctprojector_b200.projector.cupy import fan_equiangular, parallel

    return fan_equiangular if geom == "fan" else parallel


def check(p, ang, geom, oracle, nbatch, modes=("mean", "fbp", "adjoint")):
    rng = np.random.default_rng(p.nx + p.nu)
    y = rng.uniform(0, 1, (nbatch, len(ang), p.nv, p.nu)).astype(np.float32)
    for mode in modes:
        kw = dict(is_fbp=mode == "fbp", adjoint=mode == "adjoint")
        out = module(geom).distance_driven_bp(p, dev(y), dev(ang), **kw).cpu().numpy()
        assert rel_l2(out, oracle.dd_bp(p, y, ang, geom, **kw)) <= TOL, mode


@pytest.mark.parametrize("geom", ["fan", "parallel"])
@pytest.mark.parametrize("nx,ny,nbatch", [(31, 33, 1), (32, 64, 2), (65, 29, 3), (40, 97, 5)])
def test_tiles_and_slices(geom, nx, ny, nbatch, oracle):
    p = proj(geom, nx, ny, 83, off_u=0.4, cx=1.0, cy=-2.0, aspect=1.2)
    check(p, angles(40, geom), geom, oracle, nbatch)


@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_stack_with_rows(geom, oracle):
    """nz = nv slices projected one to one."""
    p = proj(geom, 34, 36, 60, nz=3)
    check(p, angles(24, geom), geom, oracle, 2)


@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_more_views_than_one_list(geom, oracle):
    p = proj(geom, 36, 20, 50, nview=1100)
    check(p, angles(1100, geom), geom, oracle, 1)


@pytest.mark.parametrize("pixel", [0.1, 6.0])
def test_fan_small_and_wide_tiles(pixel, oracle):
    """6 mm pixels: a tile spans more than the series of atan is used for (its
    12 mm cells are past those that the adjoint takes: see the widest ones)."""
    p = proj("fan", 40, 40, 70, pixel=pixel)
    check(p, angles(36, "fan"), "fan", oracle, 2)


@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_flipped_detector(geom, oracle):
    p = proj(geom, 33, 40, 64)
    p.du = -p.du
    check(p, angles(30, geom), geom, oracle, 2)


@pytest.mark.parametrize("geom", ["fan", "parallel"])
@pytest.mark.parametrize("kw", [{}, {"is_fbp": True}, {"adjoint": True}])
def test_angle_that_is_not_a_number(geom, kw):
    p = proj(geom, 40, 40, 64)
    ang = angles(40, geom)
    ang[7] = np.nan
    out = module(geom).distance_driven_bp(p, torch.ones(2, 40, 1, 64, device="cuda"), dev(ang), **kw)
    assert torch.isnan(out).all()


@pytest.mark.parametrize("nbatch", [1, 2, 4])
@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_pixel_driven(geom, nbatch, oracle):
    """Detectors narrower and wider than the grid (pixels off the detector add nothing)."""
    for width in (0.6, 1.3):
        p = proj(geom, 45, 38, 61, cell=width * (2.4 if geom == "fan" else 1.0) * 45 / 61)
        ang = angles(50, geom)
        y = np.random.default_rng(nbatch).uniform(0, 1, (nbatch, 50, 1, 61)).astype(np.float32)
        if geom == "fan":
            out, ref = module(geom).fbp_bp(p, dev(y), dev(ang)), oracle.fbp_bp(p, y, ang)
        else:
            out, ref = module(geom).pixel_driven_bp(p, dev(y), dev(ang)), oracle.pixel_bp_parallel(p, y, ang)
        # a pixel whose centre falls within rounding of the detector's end may
        # count or not: one cell of one view
        bad = np.abs(out.cpu().numpy() - ref) > 1e-4 * np.abs(ref).max()
        assert bad.sum() <= 2
        assert rel_l2(np.where(bad, ref, out.cpu().numpy()), ref) <= TOL


@pytest.mark.parametrize("nbatch", [1, 2, 4])
@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_adjoint_keeps_cells_on_their_pixels(geom, nbatch, oracle):
    """Exact adjoint: pixels outside a cell's footprint do not feel it, whether
    it is not a number, infinite or six orders above the others."""
    p = proj(geom, 70, 61, 96)
    ang = angles(40, geom)
    y = np.random.default_rng(5).uniform(0.5, 1, (nbatch, 40, 1, 96)).astype(np.float32)
    cells = [(0, 3, 40), (nbatch - 1, 11, 50), (0, 29, 44), (nbatch - 1, 34, 52)]
    mark = np.zeros_like(y)
    for b, view, k in cells:
        mark[b, view, 0, k] = 1
    reach = oracle.dd_bp(p, mark, ang, geom, adjoint=True)
    ref = oracle.dd_bp(p, np.where(mark > 0, 0, y).astype(np.float32), ang, geom, adjoint=True)
    # an edge within rounding of the cell's may reach one pixel more: skip the fringe
    fringe = np.zeros_like(reach, dtype=bool)
    on = reach > 0
    for dy in (-1, 0, 1):
        for dx in (-1, 0, 1):
            fringe |= np.roll(on, (dy, dx), (2, 3))
    for bad in (np.nan, np.inf, 1e6):
        x = np.where(mark > 0, np.float32(bad), y).astype(np.float32)
        out = module(geom).distance_driven_bp(p, dev(x), dev(ang), adjoint=True).cpu().numpy()
        away = ~fringe
        assert np.isfinite(out[away]).all(), bad
        assert np.abs(out - ref)[away].max() <= 4 * TOL * np.abs(ref).max(), bad
        deep = reach > 0.05 * reach.max()
        assert not np.isfinite(out[deep]).any() if not np.isfinite(bad) else (out[deep] > 1e3).all()
        if bad == np.inf:
            assert (out[deep] == np.inf).all()


@pytest.mark.parametrize("nbatch", [1, 3])
@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_pixel_driven_infinity(geom, nbatch, oracle):
    """An infinite cell gives infinity, not NaN, between its neighbours' centres."""
    p = proj(geom, 45, 38, 61)
    ang = angles(50, geom)
    y = np.random.default_rng(4).uniform(0, 1, (nbatch, 50, 1, 61)).astype(np.float32)
    call, ref = ("fbp_bp", "fbp_bp") if geom == "fan" else ("pixel_driven_bp", "pixel_bp_parallel")
    mark = np.zeros_like(y)
    mark[0, 7, 0, 30] = mark[nbatch - 1, 20, 0, 25] = mark[nbatch - 1, 20, 0, 26] = 1
    x = np.where(mark > 0, np.float32(np.inf), y)
    reach = getattr(oracle, ref)(p, mark, ang)
    out = getattr(module(geom), call)(p, dev(x), dev(ang)).cpu().numpy()
    assert (out[reach > 1e-3 * reach.max()] == np.inf).all()
    away = reach == 0
    clean = getattr(oracle, ref)(p, np.where(mark > 0, 0, y).astype(np.float32), ang)
    ok = away & np.isfinite(out)
    assert away.sum() - ok.sum() <= 4  # a centre within rounding of the neighbour's
    assert rel_l2(out[ok], clean[ok]) <= TOL


def test_fan_adjoint_at_its_widest_cells(oracle):
    """Cells of 0.0098 rad, where the expansion in the cell's angle ends, on
    tiles wide enough for the full arctangent."""
    p = proj("fan", 40, 40, 81, pixel=6.0, cell=10.6)
    check(p, angles(36, "fan"), "fan", oracle, 2, modes=("adjoint",))


@pytest.mark.parametrize("geom", ["fan", "parallel"])
def test_adjoint_of_fine_and_coarse_cells(geom, oracle):
    """Cells from a fifth of a pixel (several within one) to six pixels."""
    for factor, nu in ((0.2, 300), (6.0, 12)):
        p = proj(geom, 37, 45, nu, cell=factor * (1.82 if geom == "fan" else 1.0))
        check(p, angles(40, geom), geom, oracle, 3, modes=("adjoint",))
